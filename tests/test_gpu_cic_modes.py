"""The deposit's fixed-point sums, bit for bit: numpy forms the same FP64 weights, rounds each to 2^-32 and adds them as
integers.  The cases reach each way the kernel adds a value (short lists, long lists, weights from 2^17 on), both row
tiles (below and from 512^3), rows that wrap around the box, and the counts' scan in one launch and in two."""
import numpy as np
import pytest

from conftest import random_particles

pytestmark = pytest.mark.gpu


def expected(x, y, z, n):
    w = float(np.float32(n ** 3 / float(np.float32(x.size))))
    i = [a.astype(np.int64) for a in (x, y, z)]
    d = [a.astype(np.float64) - k for a, k in zip((x, y, z), i)]
    t = [1.0 - a for a in d]
    out = {}
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                v = np.rint((d[2] if dz else t[2]) * (d[0] if dx else t[0]) * ((d[1] if dy else t[1]) * w) * 2.0 ** 32)
                cell = (((i[2] - 1 + dz) % n) * n + (i[1] - 1 + dy) % n) * n + (i[0] - 1 + dx) % n
                for c, q in zip(cell.tolist(), v.tolist()):
                    out[c] = out.get(c, 0) + int(q)
    return out


@pytest.mark.parametrize("n,nrow,kind", [
    (256, 1, "uniform"),      # one particle of weight 2^24
    (128, 3, "uniform"),      # weights of 77672
    (16, 24, "one cell"),     # 13824 particles in one cell: long lists
    (16, 24, "uniform"),
    (64, 16, "faces"),        # every particle beside a face of the box
    (512, 20, "faces"),       # the wider row tile
    (512, 24, "one cell"),
])
def test_deposit_is_the_integer_sum(n, nrow, kind):
    import mgglam_b200 as m

    parts = random_particles(nrow, n, seed=n + nrow)
    if kind == "one cell":
        parts[:3] = [(a / np.float32(n + 1) + np.float32(n - 1)).astype(np.float32) for a in parts[:3]]
    elif kind == "faces":
        top = np.nextafter(np.float32(n + 1), np.float32(0))
        parts[:3] = [np.where(a > n / 2, top - (a - np.floor(a)) / 8, 1 + (a - np.floor(a)) / 8).astype(np.float32)
                     for a in parts[:3]]
    box = m.Box(m.make_config(n, nrow, float(n), mg_flag=0))
    try:
        box.upload_particles(*parts)
        box.set_time(0.5, 0.01)
        box.density()
        got = box.download_grid(m.GRID_FI)
    finally:
        box.close()
    ref = np.full(n ** 3, -1.0, np.float32)
    for c, q in expected(*parts[:3], n).items():
        ref[c] = np.float32(q / 2.0 ** 32 - 1.0)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))


# T3, T1, T2 in units of 2^-23 whose product lies within 2^-22 of a half in units of 2^-32, on the other side of it than
# the product rounded to FP64: rounded once (a product and a sum contracted into one operation) it is another integer.
TIES = [(7158006, 6728658, 6458770), (7057203, 6570542, 6373546), (7000868, 7953007, 6098447),
        (7925127, 7701376, 6431604), (6732247, 5993096, 7800782), (6210210, 7201439, 6547712)]


@pytest.mark.parametrize("crowd", ["elsewhere", "same row"])   # short and long lists
@pytest.mark.parametrize("t", TIES)
def test_weights_are_rounded_as_products(t, crowd):
    """One particle with such a weight, another that fills its cell up to 1 within 2^-23 (so that FP32 holds the sum's last
    bit), the rest on nodes."""
    import mgglam_b200 as m

    n = 32
    t3, t1, t2 = (a / 2.0 ** 23 for a in t)
    far = 1.0 if crowd == "same row" else 10.0
    x, y, z = (np.full(n ** 3, v, np.float32) for v in (10.0, far, far))
    x[0], y[0], z[0] = 2 - t1, 2 - t2, 2 - t3
    x[1], y[1], z[1] = 1 + np.rint(t3 * t1 * t2 * 2 ** 23) / 2 ** 23, 1, 1
    assert x[0] == 2 - t1 and y[0] == 2 - t2 and z[0] == 2 - t3
    product = t3 * t1 * (t2 * 2.0 ** 32)
    assert int(np.rint(product)) != (t[0] * t[1] * t[2] + 2 ** 36) // 2 ** 37
    box = m.Box(m.make_config(n, n, float(n), mg_flag=0))
    try:
        box.upload_particles(x, y, z, *[np.zeros_like(x)] * 3)
        box.set_time(0.5, 0.01)
        box.density()
        got = box.download_grid(m.GRID_FI)
    finally:
        box.close()
    ref = np.full(n ** 3, -1.0, np.float32)
    for c, q in expected(x, y, z, n).items():
        ref[c] = np.float32(q / 2.0 ** 32 - 1.0)
    assert abs(ref[0]) < 2 ** -23
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
