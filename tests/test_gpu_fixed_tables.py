"""Parallel forward projection at the sizes where its line tables can go wrong:
lines around sixteen (the FP32 parts' renormalisation), cells much finer and
coarser than the pixels, slices of every kind of value in one call, and faint
regions beside bright ones."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# Per line the lookup position is rounded to 2^-25 of the line, n 2^-25 pixels:
# over n lines of values of the image's size, relative to a ray sum of n times
# the cell's width w in pixels, n 2^-25 sqrt(2 n) / (n w) = 2^-25 sqrt(2 n) / w:
# 9e-7 at n = 300 and w = 1.  Narrow cells (w = 0.2) lose the same five times.
TOL = 1.5e-6


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def fp(p, x, ang, dtype=torch.float32):
    from ctprojector_b200.projector.cupy import parallel

    out = parallel.distance_driven_fp(p, torch.tensor(x, device="cuda").to(dtype),
                                      torch.tensor(ang, device="cuda"))
    return out.float().cpu().numpy()


def scan(nx, ny, nu, width, nview=30, **kw):
    from cases import Proj

    p = Proj(nx=nx, ny=ny, nz=1, dx=1.0, dy=1.0, dz=1.0, nu=nu, nv=1, du=width, dv=1.0, nview=nview, **kw)
    return p, (0.011 + np.arange(nview) * np.pi / nview).astype(np.float32)


@pytest.mark.parametrize("nx,ny,nu,width", [(15, 17, 31, 0.8), (16, 16, 32, 1.0), (33, 31, 63, 0.9),
                                            (300, 129, 400, 1.0), (64, 257, 700, 0.2), (130, 96, 40, 4.7)])
@pytest.mark.parametrize("nbatch", [1, 3])
def test_lines_and_cells(nx, ny, nu, width, nbatch, oracle):
    p, ang = scan(nx, ny, nu, width, off_u=0.3, cx=0.7, cy=-1.2)
    rng = np.random.default_rng(nx + nu)
    x = rng.uniform(-0.2, 1, (nbatch, 1, ny, nx)).astype(np.float32)
    assert rel_l2(fp(p, x, ang), oracle.dd_fp(p, x, ang, "parallel")) <= TOL / min(1.0, width)


def test_slices_of_every_kind(oracle):
    """Scales, signs, a dominant pixel and zeros, each slice by itself."""
    p, ang = scan(97, 83, 140, 1.0)
    rng = np.random.default_rng(7)
    x = rng.uniform(0, 1, (9, 1, 83, 97)).astype(np.float32)
    x[1] = 0
    x[2] *= 1e-18
    x[3] *= 1e18
    x[4] *= -1
    x[5, 0, 40, 40] = 3e4       # one pixel far above the mean
    x[6, 0, :40] = 0
    out = fp(p, x, ang)
    ref = oracle.dd_fp(p, x, ang, "parallel")
    assert not out[1].any()
    for i in (0, 2, 3, 4, 6, 7, 8):
        assert rel_l2(out[i], ref[i]) <= TOL, i
    # one pixel makes up the ray sums of slice 5: a single line's position, off by
    # 2^-25 of 97 pixels at each edge: 97 2^-25 sqrt(2) = 4.1e-6
    assert rel_l2(out[5], ref[5]) <= 4.1e-6
    bad = x.copy()
    bad[7, 0, 20, 30] = np.inf
    bad[8, 0, 50, 10] = np.nan
    got = fp(p, bad, ang)
    np.testing.assert_array_equal(got[:7], out[:7])
    assert not np.isfinite(got[7]).all() and np.isnan(got[8]).any()


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
def test_storage(dtype, oracle):
    p, ang = scan(65, 70, 100, 1.0)
    dt = getattr(torch, dtype)
    x = torch.rand(2, 1, 70, 65, generator=torch.Generator().manual_seed(1)).to(dt).float().numpy()
    ref = oracle.dd_fp(p, x, ang, "parallel")
    # the stored result rounds to 2^-9 (bfloat16) or 2^-12 (float16) at most
    assert rel_l2(fp(p, x, ang, dt), ref) <= (2.0**-9 if dtype == "bfloat16" else 2.0**-12) + TOL


def test_faint_half_keeps_its_own_precision(oracle):
    """Rays that meet only the faint half of a slice (1e-4 of the bright one)
    are as exact, ray by ray, as those of a slice without a bright half."""
    n = 300
    p, ang = scan(n, n, 300, 1.0, nview=3)
    ang = np.array([0.011, 0.02, 3.13], np.float32)
    rng = np.random.default_rng(11)
    x = (1e-4 * rng.uniform(0, 1, (1, 1, n, n))).astype(np.float32)
    bright = np.zeros_like(x)
    bright[..., : n // 2] = rng.uniform(0.5, 1, (1, 1, n, n // 2))
    x += bright
    faint = oracle.dd_fp(p, bright, ang, "parallel") == 0
    ref = oracle.dd_fp(p, x, ang, "parallel")
    faint &= ref > 0.1 * n * 0.5e-4
    assert faint.sum() > 200
    out = fp(p, x, ang)
    # TOL is the root mean square over rays: four times that for the worst of some hundred
    assert (np.abs(out - ref)[faint] / ref[faint]).max() <= 4 * TOL
