"""The 3-D transform at every line length (each has its own radices and threads per line) in both forms, against numpy
(from 512 on torch, on the GPU) in FP64: the potential through the fused z pass, P(k) through the binning z pass.  At
1024 a block's P(k) sums hold 8192 modes, the most that their carry-free words allow.

Bounds: the grid is rounded to FP32 between the five passes (6e-8 each), and FP32 lines add their butterflies' rounding
(log2 N stages of 6e-8); the bounds are those of the 512^3 test of the whole solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OM, A = 0.3089, 0.5


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [16, 32, 64, 128, 256])
def test_transform_at_every_size(n, precision):
    import mgglam_b200 as m

    rng = np.random.default_rng(n)
    d = rng.standard_normal((n, n, n)).astype(np.float32)
    box = m.Box(m.make_config(n, 16, float(n), mg_flag=0, precision=precision))
    try:
        box.set_time(A, 0.01)
        box.upload_grid(m.GRID_FI, d)
        box.potential()
        got = box.download_grid(m.GRID_FI).reshape(n, n, n).astype(np.float64)
        box.upload_grid(m.GRID_FI, d)
        pk = box.power(recompute_density=False)
    finally:
        box.close()
    f = np.fft.rfftn(d.astype(np.float64))
    g = 2 * np.cos(2 * np.pi * np.arange(n) / n)
    lam = g[:, None, None] + g[None, :, None] + g[None, None, : n // 2 + 1] - 6
    lam[0, 0, 0] = 1.0
    ref = np.fft.irfftn(f / lam, s=(n, n, n)) * (1.5 * OM / A)
    assert np.max(np.abs(got - ref)) < (1e-5 if precision else 1e-6) * np.max(np.abs(ref))
    k = np.fft.fftfreq(n, 1.0 / n)
    kx = np.arange(n // 2 + 1)
    r = np.sqrt(k[:, None, None] ** 2 + k[None, :, None] ** 2 + kx ** 2)
    w = np.where((kx == 0) | (kx == n // 2), 1.0, 2.0) * np.ones_like(r)
    w[0, 0, 0] = 0
    b = np.maximum((r + 0.5).astype(int), 1)
    cnt = np.bincount(b.ravel(), w.ravel())[1 : n // 2 + 1]
    p = np.bincount(b.ravel(), (w * np.abs(f / n ** 3) ** 2).ravel())[1 : n // 2 + 1] / cnt * float(n) ** 3
    assert np.array_equal(pk["nmodes"], cnt)
    assert np.max(np.abs(pk["pk"] / p - 1)) < 2e-5


def reference(d, n):
    """Potential and P(k) of d in FP64 on the GPU."""
    import torch
    torch.cuda.empty_cache()
    f = torch.fft.rfftn(torch.from_numpy(d).cuda().double().reshape(n, n, n))
    k = torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=torch.float64)
    kx = torch.arange(n // 2 + 1, device="cuda", dtype=torch.float64)
    w = (2.0 - ((kx == 0) | (kx == n // 2)).double()).expand(n, -1).contiguous()
    cnt, p = (torch.zeros(n + 1, device="cuda", dtype=torch.float64) for _ in range(2))
    for i in range(n):   # one z plane of the spectrum at a time
        r = torch.sqrt(k[i] ** 2 + k[:, None] ** 2 + kx ** 2)
        b = (r + 0.5).long().clamp(min=1).reshape(-1)
        wi = w.clone()
        if i == 0:
            wi[0, 0] = 0
        cnt.index_add_(0, b, wi.reshape(-1))
        p.index_add_(0, b, (wi * (f[i].abs() / n ** 3) ** 2).reshape(-1))
    g = 2 * torch.cos(2 * np.pi * torch.arange(n, dtype=torch.float64, device="cuda") / n)
    for i in range(n):
        lam = g[i] + g[:, None] + g[None, : n // 2 + 1] - 6
        if i == 0:
            lam[0, 0] = 1.0
        f[i] /= lam
    phi = (torch.fft.irfftn(f, s=(n, n, n)) * (1.5 * OM / A)).reshape(-1)
    nb = slice(1, n // 2 + 1)
    return phi, cnt[nb].cpu().numpy(), (p[nb] / cnt[nb]).cpu().numpy() * float(n) ** 3


@pytest.mark.parametrize("n", [512, 1024])
def test_long_lines(n):
    import torch
    import mgglam_b200 as m

    d = np.random.default_rng(n).standard_normal(n ** 3, dtype=np.float32)
    phi, cnt, p = reference(d, n)
    try:
        for precision in (0, 1):
            box = m.Box(m.make_config(n, 16, float(n), mg_flag=0, precision=precision))
            try:
                box.set_time(A, 0.01)
                box.upload_grid(m.GRID_FI, d)
                box.potential()
                got = torch.from_numpy(box.download_grid(m.GRID_FI)).cuda().double()
                box.upload_grid(m.GRID_FI, d)
                pk = box.power(recompute_density=False)
            finally:
                box.close()
            err = float((got - phi).abs().max() / phi.abs().max())
            assert err < (1e-5 if precision else 1e-6), (precision, err)
            assert np.array_equal(pk["nmodes"], cnt), precision
            assert np.max(np.abs(pk["pk"] / p - 1)) < 2e-5, precision
            del got
    finally:
        del phi
        torch.cuda.empty_cache()
