"""The fused smoother's roots where they are hard: a nearly empty box with a few very dense cells, so that the first sweeps
leave the FP32 Newton region (cells whose value falls by orders of magnitude, negative starts after a correction) and the
closed form takes over, against the serial FP64-arithmetic oracle.  128^3 is the smallest mesh with the fused sweep, 64^3
the one whose levels take the tile sweep on the finest level.

Bounds: those of the other solves, 1e-5 of the field's maximum on the plain path and 1e-4 in the precision form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("model,n,cycle", [(1, 0, "V"), (1, 1, "V"), (1, 1, "W"), (1, 2, "V"), (3, 1, "V")])
def test_dense_cells_in_a_void(orc, model, n, cycle, precision, N):
    import mgglam_b200 as m

    cfg = m.make_config(N, 16, float(N), mg_model=model, fr_n=n, fr0=-1e-6, cycle=cycle, iter_count_max=2,
                        precision=precision)
    rng = np.random.default_rng(n)
    rho = np.full(N ** 3, 0.05)
    rho[rng.integers(0, N ** 3, N ** 3 // 2000)] += 1900.0   # 95 % of the mass
    d = (rho / rho.mean() - 1).astype(np.float32)
    box = m.Box(cfg)
    try:
        box.set_time(0.7, 0.01)
        box.upload_grid(m.GRID_FI, d)
        box.scalar_field(1)
        u = box.download_grid(m.GRID_FI2).astype(np.float64)
    finally:
        box.close()
    ref, _ = orc.scalar_field(d, np.zeros_like(d), cfg, 0.7, 1)
    assert np.all(np.isfinite(u))
    assert np.max(np.abs(u - ref)) < (1e-4 if precision else 1e-5) * np.max(np.abs(ref))
