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


def toeplitz(pkg, dims, C, L, seed=0):
    """call(ctx) -> image: 2 CG iterations from a given Q."""
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

    def call(ctx):
        x = [torch.zeros(N, device="cuda") for _ in range(2)]
        pkg.toeplitz_recon(ctx, o, *x, *b, *q, t, 64, fm, *s, C, *dims)
        return (x[0] + 1j * x[1]).cpu().numpy()
    return call


@pytest.mark.parametrize("C", [4, 12])
@pytest.mark.parametrize("what", ["one", "batch", "toeplitz"])
def test_failed_setup_is_done_again(pkg, what, C):
    """Two calls without room, then one with it, on one context."""
    call = {"one": lambda: brute_force(pkg, C, 1 << 18, 0),
            "batch": lambda: brute_force(pkg, C, 1 << 17, 2),
            "toeplitz": lambda: toeplitz(pkg, (256, 256, 1), C, 3)}[what]()
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
