"""What the exact L2 search leaves out of its tensor-core scores, against the bound that
its selection rests on: every rounding of the split of an FP32 value into two BF16
parts, emulated, and the inner product that leaves most out."""
import os
import re

import numpy as np

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _constants():
    with open(os.path.join(REPO, "pynear_gb300", "csrc", "tc_scan.cu")) as f:
        text = f.read()
    lo = float.fromhex(re.search(r"constexpr float SPLIT_LO = (0x1p-\d+)f;", text).group(1))
    left = re.search(r"constexpr float SPLIT_LEFT = ([\d.]+)f \* SPLIT_LO \* SPLIT_LO;", text).group(1)
    assert re.search(r"slack\.cross = 2\.f \* \(SPLIT_LEFT \+ 0x1p-14f \* \(float\)ceil_div\(K, 512\)\);", text)
    return lo, float(left) * lo * lo


def _bf16(x):
    """Round to nearest even to BF16 (finite values)."""
    u = np.asarray(x, np.float32).view(np.uint32)
    return ((u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32)


def _split(x):
    hi = _bf16(x)
    lo = _bf16((x - hi).astype(np.float32))
    return hi, lo, x.astype(np.float64) - hi - lo


def test_parts_stay_within_their_bounds():
    lo_max, _ = _constants()
    v = (np.arange(1 << 23, dtype=np.uint32) | np.uint32(0x3F800000)).view(np.float32)  # every mantissa
    hi, lo, r = _split(v)
    assert 0.99 * lo_max < (np.abs(v.astype(np.float64) - hi) / v).max() <= lo_max
    assert (np.abs(r) / v).max() <= lo_max * lo_max


def test_products_left_out_stay_within_their_bound():
    _, left = _constants()
    v = (np.arange(1 << 23, dtype=np.uint32) | np.uint32(0x3F800000)).view(np.float32)
    hi, lo, r = _split(v)
    for sign in (1.0, -1.0):  # the value whose parts point the same way most
        i = int(np.argmax(sign * (lo.astype(np.float64) / v) + 256 * r * sign / v))
        x = v[i : i + 1]
        h, l, _ = _split(x)
        h, l, w = np.float64(h[0]), np.float64(l[0]), np.float64(x[0])
        lost = abs(w * w - (h * h + 2 * h * l)) / (w * w)
        assert lost <= left
    rng = np.random.default_rng(0)
    worst = 0.0
    for scale in (1e-3, 1e-2, 1.0):  # near the value that rounds worst
        a = np.float32(1 + 2.0**-8) + rng.random((400, 64), dtype=np.float32) * np.float32(scale * 2.0**-8)
        h, l, _ = _split(a)
        a, h, l = a.astype(np.float64), h.astype(np.float64), l.astype(np.float64)
        lost = np.abs(a @ a.T - (h @ h.T + h @ l.T + l @ h.T))
        worst = max(worst, (lost / (np.linalg.norm(a, axis=1)[:, None] * np.linalg.norm(a, axis=1))).max())
    assert 0.3 * left < worst <= left
