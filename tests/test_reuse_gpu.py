"""State kept between calls of one context (operator scratch, batched solver): every call gives
what a fresh context gives, whatever ran before it."""
import numpy as np
import pytest

from test_nudft_gpu import case_nd

pytestmark = pytest.mark.gpu


def test_operator_scratch_is_shared_safely(pkg, synth):
    """Forward and adjoint calls of unlike sizes and coil counts in turn on one context."""
    from gpu_util import gpu_ft, gpu_ift
    calls = []
    for C, n, M, z in ((1, 16, 300, 1), (12, 40, 1500, 1), (3, 12, 900, 4), (32, 24, 2000, 1),
                       (1, 64, 5000, 1), (5, 9, 100, 1)):
        c = case_nd(synth, n, n, z, C, M, seed=C * 10 + n)
        rng = np.random.default_rng(C)
        N, M = c["ix"].size, c["kx"].size
        x = rng.standard_normal(N) + 1j * rng.standard_normal(N)
        d = rng.standard_normal((C, M)) + 1j * rng.standard_normal((C, M))
        u = int(z > 1)
        calls.append(lambda ctx, c=c, x=x, u=u: gpu_ft(pkg, ctx, c, x, use_z=u))
        calls.append(lambda ctx, c=c, d=d, u=u: gpu_ift(pkg, ctx, c, d, use_z=u))
    with pkg.Context(0) as one:
        for _ in range(2):
            for f in calls:
                with pkg.Context(0) as fresh:
                    assert np.array_equal(f(one), f(fresh))


def test_batch_solver_reuse(pkg, synth):
    """Batched calls of the same sizes with other trajectories, maps and data, then of another
    penalty, another coil count and other slices."""
    rng = np.random.default_rng(3)
    f32 = lambda a: np.ascontiguousarray(a, np.float32)

    def call(ctx, n, C, counts, lam, seed):
        r = np.random.default_rng(seed)
        off = np.concatenate([[0], np.cumsum(counts)])
        M, N, S = int(off[-1]), n * n, len(counts)
        ix, iy, iz = synth.grid_positions(n, n, 1)
        xr, xi = np.zeros(S * N, np.float32), np.zeros(S * N, np.float32)
        k = [f32(r.uniform(-n / 2, n / 2, M)) for _ in range(2)]
        o = pkg.bf_options(cg_num=3, fd_penalizer=lam, dims=(n, n, 1))
        pkg.bruteForceBatch(ctx, o, xr, xi, f32(r.standard_normal(C * M)),
                            f32(r.standard_normal(C * M)), k[0], k[1], f32(np.zeros(M)),
                            f32(r.uniform(0, 0.01, M)), off, ix, iy, iz,
                            f32(r.uniform(-300, 300, S * N)), f32(r.standard_normal(C * N)),
                            f32(r.standard_normal(C * N)), N, C)
        return xr + 1j * xi

    runs = [(16, 4, (300, 200), 1e-2, 1), (16, 4, (300, 200), 1e-2, 2), (16, 4, (300, 200), 5e-2, 3),
            (16, 4, (200, 300), 5e-2, 4), (16, 12, (200, 300), 5e-2, 5), (16, 4, (300, 200), 1e-2, 1),
            (16, 4, (300, 200), None, 6)]
    with pkg.Context(0) as one:
        for a in runs:
            with pkg.Context(0) as fresh:
                assert np.array_equal(call(one, *a), call(fresh, *a))


def test_new_context_takes_no_work_memory(pkg):
    """A context's work memory comes with the calls that need it."""
    import torch
    pkg.Context(0).close()
    before = torch.cuda.mem_get_info()[0]
    with pkg.Context(0):
        assert before - torch.cuda.mem_get_info()[0] < 4 << 20


def test_launch_counts(pkg, synth):
    """Above 8 coils every apply of the operator is two launches (operand image and NUDFT): three
    launches of an operator call become four; a reconstruction of n updates has one more for the
    start and two per update."""
    from gpu_util import gpu_ft, gpu_ift, gpu_recon
    counts = {}
    for C in (8, 12):
        c = case_nd(synth, 16, 16, 1, C, 300, seed=C)
        rng = np.random.default_rng(C)
        c["kdata"] = (rng.standard_normal((C, 300)) + 1j * rng.standard_normal((C, 300))).astype(
            np.complex64)
        with pkg.Context(0) as ctx:
            counts[C] = []
            for f in (lambda: gpu_ft(pkg, ctx, c, np.ones(256)),
                      lambda: gpu_ift(pkg, ctx, c, c["kdata"]),
                      lambda: gpu_recon(pkg, ctx, c, cg_num=6, lam=None, tv=False)):
                f()
                counts[C].append(ctx.launch_count())
    assert counts[8][:2] == [3, 3] and counts[12][:2] == [4, 4]
    assert counts[12][2] - counts[8][2] == 1 + 2 * 5


def test_small_operator_call_maps_no_memory(pkg, synth, monkeypatch):
    """The work memory of F and F^H at 64x64, one coil, fits the allocator's 2 MB blocks: a first
    call on a new context pays for no mapping of its own (default shapes: a shape that an earlier
    reconstruction of this size was tuned to may have more parts)."""
    import torch
    from gpu_util import gpu_ft, gpu_ift
    monkeypatch.setenv("IMP_AUTOTUNE", "0")
    c = case_nd(synth, 64, 64, 1, 1, 4096, seed=3)
    x, d = np.ones(4096), np.ones((1, 4096))
    for f in (lambda ctx: gpu_ft(pkg, ctx, c, x), lambda ctx: gpu_ift(pkg, ctx, c, d)):
        with pkg.Context(0) as first:
            f(first)  # kernels loaded, the arrays' memory cached
        with pkg.Context(0) as ctx:
            before = torch.cuda.mem_get_info()[0]
            f(ctx)
            assert before - torch.cuda.mem_get_info()[0] <= 2 << 20
