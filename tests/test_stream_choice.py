"""Which gated product 9 to 16 rows take: the few-rows kernel where its tiles of 64 outputs make one nearly full round."""
import types

import pytest


@pytest.mark.parametrize("F,fills", [(64, False), (4608, False), (7040, False), (7104, True), (8192, True), (9472, True), (9473, False),
                                     (10752, False), (65536, False)])
def test_rule(F, fills):
    from catena_models_b200.engine.runtime import Runtime

    assert Runtime._fills_one_round(types.SimpleNamespace(_sm_count=148), F) == fills
