"""Sizes that fwi_unet_wgrad_partials is asked for without a GPU: any
arguments give a count, which fwi_unet_conv3x3_wgrad checks later."""
import subprocess
import sys

import pytest

CALL = "from seispie_b200 import _lib; print(_lib.load().fwi_unet_wgrad_partials(%d, %d, %d, %d, %d))"


def _partials(*args):
    # in a process of its own: a division by zero would end this one
    r = subprocess.run([sys.executable, "-c", CALL % args], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stderr[-300:])
    return int(r.stdout)


@pytest.mark.parametrize("args", [(0, 16, 1, 8, 8), (16, 0, 1, 8, 8), (16, 16, 0, 8, 8), (16, 16, 1, 0, 8),
                                  (16, 16, 1, 8, 0), (-16, 16, 1, 8, 8), (16, 16, -1, 8, 8), (0, 0, 0, 0, 0)])
def test_empty_sizes_need_no_scratch(args):
    assert _partials(*args) == 0


@pytest.mark.parametrize("args", [(8, 16, 1, 8, 8), (16, 8, 1, 8, 8), (16, 16, 1, 2 ** 31 - 1, 1),
                                  (16, 16, 1, 1, 2 ** 31 - 1), (16, 16, 2 ** 31 - 1, 1, 1)])
def test_unusual_sizes_give_a_count(args):
    assert _partials(*args) > 0
