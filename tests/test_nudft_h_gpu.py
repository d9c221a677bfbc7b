"""The FP16 head / tail tensor-core NUDFT kernel (nudft_h.cu; the kernel behind
IMP_NUDFT_TC=1 in test_nudft_tc_gpu.py): its per-(tile, coil) power-of-two data scales."""
import numpy as np
import pytest

import oracle
from test_nudft_gpu import case_nd
from test_nudft_tc_gpu import TOL_OP, built, ctx  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def forced(monkeypatch):
    monkeypatch.setenv("IMP_NUDFT_TC", "1")


@pytest.mark.parametrize("C", [1, 4, 8, 16, 32])
@pytest.mark.parametrize("k", [-96, -20, 37, 90])
def test_power_of_two_scale_is_exact(pkg, ctx, synth, C, k):
    """Data times 2^k gives the result times 2^k, bit for bit (far outside FP16's range)."""
    from gpu_util import gpu_ift
    c = case_nd(synth, 24, 24, 1, C, 700, seed=C)
    rng = np.random.default_rng(C + 1)
    d = (rng.standard_normal((C, 700)) + 1j * rng.standard_normal((C, 700))).astype(np.complex64)
    a = gpu_ift(pkg, ctx, c, d)
    b = gpu_ift(pkg, ctx, c, d * np.float32(2.0) ** k)
    assert np.array_equal(b, a * 2.0 ** k)


@pytest.mark.parametrize("C", [4, 32])
def test_tiles_of_unlike_scale(pkg, ctx, synth, C):
    """All-zero tiles, tiles 2^60 apart and one sample 1e6 above its tile: each output keeps the
    operator bar relative to the sum of its terms' magnitudes."""
    from gpu_util import gpu_ft, gpu_ift
    c = case_nd(synth, 24, 24, 1, C, 1024, seed=C + 50)
    rng = np.random.default_rng(C + 2)
    d = rng.standard_normal((C, 1024)) + 1j * rng.standard_normal((C, 1024))
    d[:, :64] = 0.0
    d[:, 64:128] *= 2.0 ** -60
    d[:, 700] *= 1e6
    d = d.astype(np.complex64)
    assert oracle.rel_l2(gpu_ift(pkg, ctx, c, d), oracle.ift(d, c, use_z=0)) < TOL_OP
    x = rng.standard_normal(576) + 1j * rng.standard_normal(576)
    x[:128] *= 2.0 ** -50
    x[300] *= 1e6
    assert oracle.rel_l2(gpu_ft(pkg, ctx, c, x), oracle.ft(x, c, use_z=0)) < TOL_OP
