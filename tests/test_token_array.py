"""Token ids become one integer array whatever sequence they come in; what the quick conversion refuses goes numpy's way."""
import numpy as np
import pytest

from catena_models_b200.engine.batch import BatchLayout, fill_host, token_array


@pytest.mark.parametrize("tokens", [[5], [0, 65535, 7], (1, 2), np.array([3, 4]), np.array([9], dtype=np.int32), [np.int64(8), 2],
                                    [True, 3], [2.0, 5.0], [2 ** 40], [-1]])
def test_same_values(tokens):
    assert token_array(tokens).tolist() == np.asarray(tokens).tolist()


def test_out_of_any_range_is_left_to_the_check():
    assert token_array([2 ** 70]).max() >= 65536


def test_filled_step():
    layout = BatchLayout(64, 2, 2, 4)
    host = np.full(layout.size, 77, dtype=np.int32)
    prompts = [[9, 8, 7], list(range(50))]
    other = host.copy()
    for buf, toks in ((host, prompts), (other, [token_array(p) for p in prompts])):
        fill_host(layout, buf, [3, 1], toks, [0, 10], [[2], [49]], [(1, 2)])
    assert (host == other).all() and layout.views(host)["tokens"][:5].tolist() == [9, 8, 7, 0, 1]
