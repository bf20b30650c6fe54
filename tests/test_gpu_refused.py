"""A call that the runtime refuses (a launch grid beyond its extents, nothing
is launched) reports that itself and leaves nothing for the next call."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("what", ["forward", "transposed"])
def test_a_refused_launch_is_reported_once(what):
    from seispie_b200._lib import FWI_PSV, FwiError
    from seispie_b200.engine import DeviceModel, Grid, ShotBatch
    nx, nz = 32 * 65535 + 1, 3  # one tile too many along x for the second extent
    if what == "transposed":
        nx = 32 * 65535 * 2  # P-SV on 32 x 64 tiles go by z first

    m = DeviceModel(Grid(nx, nz, 10.0, 10.0), FWI_PSV, 1e-3, "cuda")
    for k, v in dict(rho=2600.0, lam=8.1e9, mu=8.1e9, bound=1.0).items():
        getattr(m, k).fill_(v)
    m.prepare()
    b = ShotBatch(m, 1, 2, np.array([5], np.int32), displacement=True)
    with pytest.raises(FwiError, match="_kernel"):
        if what == "forward":
            b.run(b.desc(), False, 0, 1)
        else:
            z = torch.zeros(1, 1, nx, m.grid.pitch, device="cuda")
            ks = [torch.zeros((nx, m.grid.pitch), dtype=torch.float64, device="cuda") for _ in range(2)]
            d = b.desc(record=False, kernels=ks)
            b.set_segment(d, [z] * 3, [None] * 3, 0, 1)
            b.run_transposed(d, 1, 1)
    m.prepare()  # the next call of the library
    torch.cuda.synchronize()
