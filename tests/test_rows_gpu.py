"""The forms for many rows of the residual kernel (a warp per row) and of the short convolution (eight tokens a thread) against
their forms for few rows: the same bits, whatever the width, the options and the cuts between sequences."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def K():
    from catena_models_b200 import kernels

    kernels.lib()
    return kernels


@pytest.mark.parametrize("H", [8, 256, 504, 512, 520, 1000, 1024, 1032, 2040, 2048])
@pytest.mark.parametrize("post,nxt", [(True, True), (True, False), (False, True), (False, False)])
def test_add_norm_of_many_rows(K, H, post, nxt):
    rows = 1500
    g = torch.Generator(DEV).manual_seed(H)
    m = (3 * torch.randn(rows, H, generator=g, device=DEV)).to(torch.bfloat16)
    h = torch.randn(rows, H, generator=g, device=DEV).to(torch.bfloat16)
    m[7], h[9, 0], m[11, H - 1] = 0.0, float("inf"), float("nan")
    wp = 1 + 0.1 * torch.randn(H, generator=g, device=DEV) if post else None
    wn = 1 + 0.1 * torch.randn(H, generator=g, device=DEV) if nxt else None
    few_h, few_n = torch.empty_like(h), torch.empty_like(h)
    for at in range(0, rows, 500):                                     # 500 rows at a time: the form of a block per row
        s = slice(at, at + 500)
        K.add_norm(few_h[s], few_n[s] if nxt else None, m[s], h[s], wp, wn, 1e-5, 1e-6)
    stream, n = h.clone(), torch.full_like(h, 7.0)
    K.add_norm(stream, n if nxt else None, m, stream, wp, wn, 1e-5, 1e-6)      # in place, as the blocks call it
    same = lambda a, b: torch.equal(a.view(torch.int16), b.view(torch.int16)) or torch.equal(torch.nan_to_num(a.float()), torch.nan_to_num(b.float()))  # noqa: E731
    assert same(stream, few_h)
    if nxt:
        assert same(n, few_n)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("H", [8, 264, 1024])
@pytest.mark.parametrize("how", ["prompts", "append"])
def test_shortconv_of_many_tokens(K, dtype, taps, H, how):
    lens = [1, 2, 3, 700, 5, 1, 8, 331, 16, 7, 9]                      # cuts at, before and inside a thread's run of tokens
    pad = 13
    T = sum(lens) + pad
    g = torch.Generator(DEV).manual_seed(T + H + taps)
    bcx = torch.randn(T, 3 * H + 8, generator=g, device=DEV).to(dtype)[:, :3 * H]
    w = torch.randn(H, taps, generator=g, device=DEV)
    starts = torch.tensor([0] + lens).cumsum(0).to(torch.int32).to(DEV)
    seq = torch.tensor([b for b, n in enumerate(lens) for _ in range(n)] + [-1] * pad, dtype=torch.int32, device=DEV)
    slots = torch.arange(len(lens), 0, -1, dtype=torch.int32, device=DEV)
    pos0 = torch.tensor([0 if b % 3 == 0 else 40 + b for b in range(len(lens))], dtype=torch.int32, device=DEV) if how == "append" else None
    state0 = torch.randn(len(lens) + 2, taps - 1, H, generator=g, device=DEV)
    out = []
    for w_t in (None, w.t().contiguous()):                             # without the second copy of the taps: the form for few tokens
        y, state = torch.full((T, H), float("nan"), dtype=dtype, device=DEV), state0.clone()
        K.shortconv(y, bcx, w, state, seq, starts, slots, taps, from_zero=how == "prompts", one_token_each=False, w_t=w_t, seq_pos0=pos0)
        out.append((y, state))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert (out[1][0][T - pad:] == 0).all()
