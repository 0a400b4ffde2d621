"""Row-sharing tomosynthesis kernels at the sizes where they can go wrong: rows
and planes around their tiles, and footprints on both sides of the 2 x 2 and
3 x 3 cells that they hold; against the FP64 oracle."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# sums of at most 17 planes or 11 views of FP32 products of two weights, each
# rounded to 2^-24 of a value of order one after a subtraction of coordinates
# below 2^9: 2^-24 2^2 at random over the terms
TOL = 1e-6


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def dev(a):
    return torch.tensor(np.ascontiguousarray(a, dtype=np.float32), device="cuda")


@pytest.mark.parametrize("nx,ny,nz,nu,nv,cell", [(129, 7, 3, 130, 9, 0.3), (40, 33, 9, 257, 65, 0.25), (64, 40, 17, 31, 33, 0.4),
                                                 (64, 40, 17, 31, 33, 0.45),
                                                 (50, 37, 8, 40, 24, 1.1)])
def test_tomo_rows(nx, ny, nz, nu, nv, cell, oracle):
    """Rows and planes around the kernels' tiles; 0.45 and 1.1 mm cells take one rectangle per thread."""
    from cases import Proj

    from ctprojector_b200 import synthetic as S
    from ctprojector_b200.projector.cupy import tomo

    p = Proj(nx=nx, ny=ny, nz=nz, dx=0.4, dy=0.4, dz=1.0, nu=nu, nv=nv, du=cell, dv=cell, nview=11, off_u=0.3, off_v=-0.4)
    dc, sr = S.tomo_geometry(11, 40.0, 500.0, -(nz / 2 + 15.0))
    rng = np.random.default_rng(nx)
    img = rng.uniform(0, 1, (2, nz, ny, nx)).astype(np.float32)
    prj = rng.uniform(0, 1, (2, 11, nv, nu)).astype(np.float32)
    fp = tomo.distance_driven_fp(p, dev(img), dev(dc), dev(sr)).cpu().numpy()
    bp = tomo.distance_driven_bp(p, dev(prj), dev(dc), dev(sr)).cpu().numpy()
    # one rectangle per thread takes its edges in FP32 relative to the source, up to
    # 182 mm to the side: 182 / 0.4 pixels of 2^-23 between a footprint's two edges
    tol = TOL if cell <= 0.4 else 182 / 0.4 * 2.0**-23
    assert rel_l2(fp, oracle.tomo_fp(p, img, dc, sr)) <= tol
    assert rel_l2(bp, oracle.tomo_bp(p, prj, dc, sr)) <= tol
