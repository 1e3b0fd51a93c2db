"""Copying pages by numbers that travel in the launch: against indexing, for more pages than one launch takes, odd page sizes and
with and without a page table."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pages_copied", [1, 255, 256, 257, 600])
@pytest.mark.parametrize("page", [(8,), (24,), (8, 64, 64), (3, 64, 40)])
@pytest.mark.parametrize("table", [False, True])
def test_pages_and_table(pages_copied, page, table):
    from catena_models_b200 import kernels as K

    g = torch.Generator("cuda").manual_seed(pages_copied)
    total = 2 * pages_copied + 3
    pool = torch.randn(2, 3, total, *page, generator=g, device="cuda").to(torch.bfloat16)
    order = torch.randperm(total, generator=torch.Generator().manual_seed(7)).tolist()
    src, dst = order[:pages_copied], order[pages_copied:2 * pages_copied]
    want = pool.clone()
    want[:, :, dst] = pool[:, :, src]
    ptab = torch.full((2, pages_copied + 2), -5, dtype=torch.int32, device="cuda")
    K.copy_pages_ids(pool, src, dst, 2, ptab[1, 1:-1] if table else None)
    assert torch.equal(pool, want)
    assert (ptab[0] == -5).all() and (ptab[1, [0, -1]] == -5).all()
    assert ptab[1, 1:-1].tolist() == (dst if table else [-5] * pages_copied)


def test_refusals():
    from catena_models_b200 import kernels as K

    pool = torch.zeros(1, 1, 4, 8, dtype=torch.bfloat16, device="cuda")
    for src, dst in (([0], [4]), ([-1], [1]), ([0, 1], [2])):
        with pytest.raises(K.KernelError):
            K.copy_pages_ids(pool, src, dst, 2)
    K.copy_pages_ids(pool, [], [], 2)
