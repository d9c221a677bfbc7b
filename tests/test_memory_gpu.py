"""Calls that do not fit the device memory: a set-up that failed part-way is not taken for a
finished one, and the context serves the same call once there is room."""
import contextlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def leave(nbytes):
    """The device with all but `nbytes` of its free memory taken."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - nbytes, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del fill
        torch.cuda.empty_cache()


def brute_force(pkg, C, M, slices, seed=0, n=16):
    """call(ctx) -> image: 2 CG iterations, all arrays on the device."""
    r = np.random.default_rng(seed)
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a, np.float32)).cuda()
    N, S = n * n, slices
    g = (np.arange(n) - n / 2) / n
    ix, iy, iz = dev(np.repeat(g, n)), dev(np.tile(g, n)), torch.zeros(N, device="cuda")
    T = M * max(S, 1)
    k = [dev(r.uniform(-n / 2, n / 2, T)) for _ in range(2)] + [torch.zeros(T, device="cuda")]
    t, fm = dev(r.uniform(0, 0.01, T)), dev(r.uniform(-300, 300, max(S, 1) * N))
    d = [dev(r.standard_normal(C * T)) for _ in range(2)]
    s = [dev(r.standard_normal(C * N)) for _ in range(2)]
    o = pkg.bf_options(cg_num=2, dims=(n, n, 1))

    def call(ctx):
        x = [torch.zeros(max(S, 1) * N, device="cuda") for _ in range(2)]
        if S:
            pkg.bruteForceBatch(ctx, o, *x, *d, *k, t, np.arange(S + 1) * M, ix, iy, iz, fm, *s, N,
                                C)
        else:
            pkg.bruteForceGpu(ctx, o, *x, *d, *k, ix, iy, iz, fm, t, *s, M, N, C, 1)
        return (x[0] + 1j * x[1]).cpu().numpy()
    return call


def toeplitz(pkg, dims, C, L, what="recon", seed=0):
    """call(ctx) -> image: 2 CG iterations from a given Q, one application of it, or F^H d."""
    r = np.random.default_rng(seed)
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a, np.float32)).cuda()
    nx, ny, nz = dims
    N = nx * ny * nz
    G = N * (8 if nz > 1 else 4) * (L + 1)
    t, fm = dev(np.linspace(0, 0.01, 64)), dev(r.uniform(-300, 300, N))
    q = [dev(r.standard_normal(G)) for _ in range(2)]
    b = [dev(r.standard_normal(N)) for _ in range(2)]
    s = [dev(r.standard_normal(C * N)) for _ in range(2)]
    o = pkg.toeplitz_options(cg_num=2, ntime_segs=L)
    x = [torch.zeros(N, device="cuda") for _ in range(2)]
    k = [dev(r.uniform(-v / 2, v / 2 - 1, 64)) for v in dims]
    d = [dev(r.standard_normal(C * 64)) for _ in range(2)]

    def call(ctx):
        if what == "fhd":
            pkg.toeplitz_fhd(ctx, o, *x, *d, *k, t, fm, *s, 64, C, *dims)
        elif what == "apply":
            pkg.toeplitz_apply(ctx, o, *x, *b, *q, t, 64, fm, *s, C, *dims)
        else:
            pkg.toeplitz_recon(ctx, o, *x, *b, *q, t, 64, fm, *s, C, *dims)
        return x[0].cpu().numpy() + 1j * x[1].cpu().numpy()
    return call


@pytest.mark.parametrize("C", [4, 12])
@pytest.mark.parametrize("what", ["one", "batch", "toeplitz"])
def test_failed_setup_is_done_again(pkg, what, C):
    """Two calls without room, then one with it, on one context."""
    call = {"one": lambda: brute_force(pkg, C, 1 << 18, 0),
            "batch": lambda: brute_force(pkg, C, 1 << 17, 2),
            "toeplitz": lambda: toeplitz(pkg, (512, 512, 1), C, 3)}[what]()
    with pkg.Context(0) as fresh:
        want = call(fresh)
    with pkg.Context(0) as one:
        for room in (4, 10, 20):
            with leave(room << 20):
                for _ in range(2):
                    with pytest.raises(pkg.ImpError, match="(?i)memory"):
                        call(one)
        assert np.array_equal(call(one), want)


@pytest.mark.parametrize("slices", [0, 2])
def test_optional_image_gives_way(pkg, monkeypatch, slices):
    """12 coils (the FP16 kernel and its image of the k-space data) with room for everything but
    half of that image: the call is served, by the TF32 kernel."""
    monkeypatch.setenv("IMP_AUTOTUNE", "0")
    M = 1 << 19
    image = M * 16 * 16  # bytes: 16 per sample and coil of the group
    call = brute_force(pkg, 12, M // max(slices, 1), slices)
    with pkg.Context(0) as ctx:
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        before = torch.cuda.mem_get_info()[0]
        want = call(ctx)
        torch.cuda.empty_cache()
        used = before - torch.cuda.mem_get_info()[0]
    assert used > 2 * image
    with pkg.Context(0) as ctx, leave(used - image // 2):
        got = call(ctx)
    # one CG update of FP16- and TF32-split sums, both 22 bits
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < 1e-5


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# what is left: enough for the spectra of one transform at a time (power-of-two side: its Q
# and one Qf_l of scratch), or for the zero-padded chain only (520 runs on 576 otherwise)
@pytest.mark.parametrize("n,C,segs,extra", [(512, 16, 42, 8 * 512 * 1024), (520, 1, 42, 0)])
def test_toeplitz_runs_leaner(pkg, n, C, segs, extra):
    """A^H A in the memory of one transform at a time, or of the zero-padded chain."""
    L, N = 40, n * n
    call, grids = (toeplitz(pkg, (n, n, 1), C, L, what) for what in ("apply", "fhd"))
    with pkg.Context(0) as ctx:
        want = call(ctx)
    need = 8 * 4 * N * segs + extra + 8 * N * (C + L + 1 + 6) + 4 * N
    for first in ("apply", "fhd"):
        with pkg.Context(0) as ctx, leave(need + (40 << 20)):
            if first == "fhd":  # its grids give way too
                grids(ctx)
            assert rel(call(ctx), want) < 1e-5


def test_fhd_needs_no_engine(pkg):
    """F^H d in the memory of its inputs and a single gridding grid (a batch takes 64 MB), also
    on a context that holds the engine."""
    n, C, L = 512, 4, 40
    call, other = (toeplitz(pkg, (n, n, 1), C, L, what) for what in ("fhd", "apply"))
    with pkg.Context(0) as ctx:
        want, image = call(ctx), other(ctx)
    with pkg.Context(0) as ctx, leave(8 * n * n * (C + L + 2) + 8 * 768 * 768 + (16 << 20)):
        assert rel(call(ctx), want) < 1e-5
    with pkg.Context(0) as ctx:
        other(ctx)
        with leave(8 << 20):
            assert rel(call(ctx), want) < 1e-5
        assert rel(other(ctx), image) < 1e-5


def adjoint(pkg, C, M, n=8, seed=0):
    """call(ctx) -> F^H d, all arrays on the device."""
    r = np.random.default_rng(seed)
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a, np.float32)).cuda()
    N = n * n
    g = (np.arange(n) - n / 2) / n
    args = [dev(r.standard_normal(C * M)) for _ in range(2)]
    args += [dev(r.uniform(-n / 2, n / 2, M)) for _ in range(2)] + [torch.zeros(M, device="cuda")]
    args += [dev(np.repeat(g, n)), dev(np.tile(g, n)), torch.zeros(N, device="cuda"), None,
             dev(r.uniform(0, 0.01, M))]
    sens = [dev(r.standard_normal(C * N)) for _ in range(2)]
    x = [torch.zeros(N, device="cuda") for _ in range(2)]

    def call(ctx):
        pkg.parallelIftGpu(ctx, *x, *args, M, N, *sens, C, 0)
        return x[0].cpu().numpy() + 1j * x[1].cpu().numpy()
    return call


def test_kept_memory_is_given_back(pkg, monkeypatch):
    """What earlier calls keep (operator scratch, images, engines) does not refuse a larger one."""
    monkeypatch.setenv("IMP_AUTOTUNE", "0")
    C = 12
    before = [adjoint(pkg, C, 1 << 19), toeplitz(pkg, (512, 512, 1), 4, 20, "apply"),
              brute_force(pkg, C, 1 << 18, 0), brute_force(pkg, C, 1 << 17, 2)]
    for larger in (toeplitz(pkg, (512, 512, 1), 4, 40, "apply"), brute_force(pkg, C, 3 << 17, 0),
                   brute_force(pkg, C, 3 << 16, 2), adjoint(pkg, C, 3 << 18)):
        with pkg.Context(0) as fresh:
            want = larger(fresh)
        with pkg.Context(0) as ctx:
            for f in before:
                f(ctx)
            with leave(24 << 20):
                assert rel(larger(ctx), want) < 1e-5


def test_operator_without_room_is_refused(pkg):
    """An operator call that has nothing left to give back ends with the status, and is served
    once there is room."""
    call = adjoint(pkg, 12, 1 << 19)
    with pkg.Context(0) as fresh:
        want = call(fresh)
    with pkg.Context(0) as ctx:
        for room in (4, 20, 40):
            with leave(room << 20):
                with pytest.raises(pkg.ImpError, match="NOMEM"):
                    call(ctx)
        assert np.array_equal(call(ctx), want)
