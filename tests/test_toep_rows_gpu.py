"""The mixed-radix F^H F engine (toep_rows.cu): one A^H A (+ lambda D^H D) application
against the FP64 oracle over the lengths of its table, the sides between them (which run on the
next length), uneven coil counts and several segments; refused sizes stay refused."""
import numpy as np
import pytest

from test_toeplitz_gpu import (TOL_OP, gpu_apply, gpu_fhd, gpu_q, gpu_recon, grid_elems, opts_of,
                               oracle_apply, rel)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(pkg):
    c = pkg.Context(0)
    yield c
    c.close()


def make(dims, C, L, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = dims
    N, M, G = nx * ny * nz, 64, grid_elems(dims)
    c = dict(dims=dims, L=L, cg=1, fdp=1e-2, tv_num=0, os_q=2.0, os_fh=1.5,
             t=np.sort(rng.uniform(0.0, 0.01, M)).astype(np.float32), kx=np.zeros(M, np.float32),
             fm=rng.uniform(-300.0, 300.0, N).astype(np.float32),
             sens=(rng.standard_normal((C, N)) + 1j * rng.standard_normal((C, N))).astype(
                 np.complex64))
    if C == 1:
        c["sens"] = np.ones((1, N), np.complex64)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
    return c, cplx(L + 1, G), cplx(N)


# (x, y): x is the strided (column) axis, y the contiguous (row) axis
SIZES = [(2, 2), (16, 16), (14, 18), (32, 48), (46, 34), (64, 80), (82, 96), (112, 98), (128, 144),
         (146, 160), (192, 162), (194, 200), (240, 202), (242, 256), (288, 258), (290, 320),
         (336, 322), (338, 384), (400, 386), (402, 448), (480, 450), (482, 512), (576, 10),
         (10, 576), (578, 12), (12, 578), (642, 8), (8, 642), (770, 6), (6, 770), (900, 4), (4, 900),
         (1024, 2), (2, 1024)]


@pytest.mark.parametrize("nx,ny", SIZES)
def test_lengths_match_oracle(pkg, ctx, nx, ny):
    c, Q, p = make((nx, ny, 1), 2, 1, nx * 7 + ny)
    got = gpu_apply(pkg, ctx, opts_of(pkg, c), c, Q, p)
    assert rel(got, oracle_apply(c, Q, p, c["fdp"])) < TOL_OP


@pytest.mark.parametrize("C,L", [(1, 0), (1, 12), (7, 1), (11, 0), (13, 2)])
def test_coils_and_segments_match_oracle(pkg, ctx, C, L):
    """Clusters of one rank, of a prime count, and ranks with unequal numbers of transforms."""
    c, Q, p = make((36, 50, 1), C, L, 100 * C + L)
    got = gpu_apply(pkg, ctx, opts_of(pkg, c), c, Q, p)
    assert rel(got, oracle_apply(c, Q, p, c["fdp"])) < TOL_OP


@pytest.mark.parametrize("dims", [(512, 512, 1), (256, 256, 1), (1024, 2, 1), (2, 1024, 1),
                                  (128, 64, 32), (240, 480, 1)])
def test_amplitude_matches_oracle(pkg, ctx, dims):
    """The share of the result that all outputs lose or gain together is below one FP32 ulp over
    the twelve or eighteen register transforms of an application."""
    c, Q, p = make(dims, 2, 0, 9)
    want = oracle_apply(c, Q, p, None)
    o = opts_of(pkg, c)
    o.enable_fd = 0
    err = gpu_apply(pkg, ctx, o, c, Q, p) - want
    gain = np.vdot(want, err).real / np.vdot(want, want).real
    print(f"{dims}: gain {gain:.1e}, error {rel(err + want, want):.2e}")
    assert abs(gain) < 2.0 ** -23


def test_sizes_past_the_table(pkg, ctx):
    """A side longer than the table runs the zero-padded chain; a doubled side with a prime
    factor above 255 is refused as before."""
    c, Q, p = make((1040, 4, 1), 2, 0, 5)
    got = gpu_apply(pkg, ctx, opts_of(pkg, c), c, Q, p)
    assert rel(got, oracle_apply(c, Q, p, c["fdp"])) < TOL_OP
    c, Q, p = make((2 * 257, 4, 1), 1, 0, 6)
    with pytest.raises(pkg.ImpError):
        gpu_apply(pkg, ctx, opts_of(pkg, c), c, Q, p)


@pytest.mark.parametrize("dims", [(514, 4, 1), (4, 2 * 257, 2), (2, 4, 514)])
@pytest.mark.parametrize("padded", ["0", "1"])
def test_refused_size_is_refused_again(pkg, monkeypatch, dims, padded):
    """A second call of a refused size on the same context is refused like the first, by every
    entry point, and the context then serves another size."""
    monkeypatch.setenv("IMP_TOEP_PADDED", padded)
    c, Q, p = make(dims, 1, 1, 6)
    c["ky"] = c["kz"] = c["kx"]
    c["kdata"] = np.ones((1, c["kx"].size), np.complex64)
    ok, Qok, pok = make((16, 18, 1), 2, 1, 7)
    with pkg.Context(0) as one:
        o = opts_of(pkg, c)
        for call in (lambda: gpu_apply(pkg, one, o, c, Q, p), lambda: gpu_fhd(pkg, one, o, c),
                     lambda: gpu_q(pkg, one, o, c), lambda: gpu_recon(pkg, one, o, c, Q, p)):
            for _ in range(2):
                with pytest.raises(pkg.ImpError):
                    call()
        got = gpu_apply(pkg, one, opts_of(pkg, ok), ok, Qok, pok)
        assert rel(got, oracle_apply(ok, Qok, pok, ok["fdp"])) < TOL_OP


# (x, y, z): y is the slow (column) axis, x the middle one, z the contiguous one
SIZES_3D = [(2, 2, 2), (4, 6, 2), (10, 12, 4), (14, 18, 10), (40, 24, 12), (16, 34, 6), (34, 16, 18),
            (20, 48, 24), (66, 10, 8), (10, 66, 8), (8, 12, 66), (24, 20, 30), (130, 6, 4),
            (6, 130, 36), (4, 258, 2), (258, 4, 2), (4, 4, 258), (4, 1040, 2)]


@pytest.mark.parametrize("nx,ny,nz", SIZES_3D)
def test_3d_lengths_match_oracle(pkg, ctx, nx, ny, nz):
    """3-D images over the table's lengths and between them (the last side is past the table:
    the zero-padded chain)."""
    c, Q, p = make((nx, ny, nz), 2, 1, nx * 7 + ny + 3 * nz)
    got = gpu_apply(pkg, ctx, opts_of(pkg, c), c, Q, p)
    assert rel(got, oracle_apply(c, Q, p, c["fdp"])) < TOL_OP


@pytest.mark.parametrize("C,L", [(1, 0), (1, 3), (5, 2), (9, 1)])
def test_3d_coils_and_segments_match_oracle(pkg, ctx, C, L):
    c, Q, p = make((20, 14, 6), C, L, 10 * C + L)
    got = gpu_apply(pkg, ctx, opts_of(pkg, c), c, Q, p)
    assert rel(got, oracle_apply(c, Q, p, c["fdp"])) < TOL_OP
