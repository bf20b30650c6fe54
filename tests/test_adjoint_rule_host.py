"""The rule that picks the transposed step's tile: a size for every batch, and
every tile for some batch."""
import pytest

from tests.adjoint_rule import compile_rule

TILES = {"sh": {8, 16, 32}, "psv": {8, 16, 32, 64}, "spin": {8, 16}}


@pytest.mark.parametrize("mode", ["sh", "psv", "spin"])
def test_every_batch_gets_a_tile(mode, tmp_path):
    rule = compile_rule(str(tmp_path))
    if rule is None:
        pytest.skip("no host compiler")
    seen = set()
    for nx, nz in ((1, 1), (8, 32), (9, 33), (200, 260), (512, 512), (3, 2097169), (4000, 2000)):
        for nshots in (1, 2, 3, 4, 8, 33, 500):
            seen.add(rule(mode, nx, nz, nshots))
    assert seen == TILES[mode]
    # beyond the second extent of a launch grid only the largest tile has an instance that goes by z first
    assert rule(mode, 1, 32 * 65535 + 1, 1) == max(TILES[mode])
