"""GPU parity of the Fourier solves at production grid sizes.

The kernels that the 512^3 cycle runs are specialised per N: the transforms'
radices, rows and columns per block and twiddle tables, and the z pass, which
loads its pencils by bulk tensor boxes for some solves (one box up to
N = 256; N = 384: three boxes of 128; N = 512: two of 256; N = 768: three of
256) and through registers for the others, and the y pass, which is staged in
FP64 at N = 512 alone.  These
tests compare each solve with an independent FP64 reference at those sizes:
pocketfft (scipy.fft, the same transform numpy uses, pinned to the oracle's
FFT in test_oracle_pin.py) for the transforms and the oracle's C restatements
for the pointwise physics (prepareFTsource, solveModifiedPoissonFT,
projectFTscalar, projectFTtensor, evolveFTtensor, projectFTvector), which are
themselves pinned to the reference's own code.

Inputs are seeded white noise, which puts weight on every mode and so on every
twiddle factor and box offset.  Tolerances: FP64 1e-10 and mixed precision
(FP32 fields and transforms, FP64 solver arithmetic) 1e-4, relative to the
largest magnitude of the compared array, as for the small-N solver tests.
Complex spectra are compared by the modulus of the complex difference.

Each test computes its reference once and checks both precisions against it."""
import numpy as np
import pytest

from _fixtures import irfft3, rel_err, rfft3
from _libs import oracle, ptr

gev = pytest.importorskip("gevb200")

pytestmark = pytest.mark.gpu

TOL = {gev.FP64: 1e-10, gev.MIXED: 1e-4}
PRECS = (gev.FP64, gev.MIXED)
FOURPIG = 1.5 * 2560.0 ** 2 / 2997.92458 ** 2
SIZES = [128, 256, 384, 512]


def noise(N, seed, amp=1.0, ncomp=1):
    rng = np.random.default_rng(seed)
    return amp * rng.standard_normal(ncomp * N ** 3)


def ctx(N, prec, **kw):
    c = gev.Context(N, precision=prec, capacity=8, **kw)
    c.set_particles(np.zeros((1, 3)), np.zeros((1, 3)))
    return c


@pytest.mark.parametrize("N", SIZES)
def test_solve_phi_sizes(N):
    """prepareFTsource (T00 form) + R2C + solveModifiedPoissonFT + C2R
    (main.cu:719-809) and the k = 0 mode, at N = 128 ... 512."""
    o = oracle()
    dx = 1.0 / N
    source = 0.32 * (1.0 + 0.5 * noise(N, 101))
    phi = noise(N, 102, 1e-5)
    chi = noise(N, 103, 1e-6)
    H, dtau_old, a = 0.8, 0.01, 0.3
    args = (0.32, 3 * H * dx * dx / dtau_old, FOURPIG * dx * dx / a, 3 * H * H * dx * dx)
    res = np.zeros(N ** 3)
    s_ref = o.prepare_T00(N, ptr(phi), ptr(chi), ptr(source), *args, ptr(res))
    FT = rfft3(res, N)
    del res
    o.solve_poisson(N, ptr(FT), ptr(FT), 1 / (dx * dx), 3 * H / dtau_old)
    phom_ref = FT[0, 0, 0].real
    scale_ft = np.abs(FT).max()
    ph_ref = irfft3(FT, N)
    del FT
    for prec in PRECS:
        with ctx(N, prec) as c:
            c.set_field(gev.FIELD_SOURCE, source)
            c.set_field(gev.FIELD_PHI, phi)
            c.set_field(gev.FIELD_CHI, chi)
            s, phom = c.solve_phi(True, *args, 1 / (dx * dx), 3 * H / dtau_old)
            assert abs(s / s_ref - 1) < (1e-12 if prec == gev.FP64 else 1e-6), prec
            assert abs(phom - phom_ref) <= TOL[prec] * scale_ft, prec
            assert rel_err(c.get_field(gev.FIELD_PHI), ph_ref) < TOL[prec], prec


def test_solve_phi_768_mixed():
    """The 768^3 passes (z: three bulk tensor boxes of 256 per pencil) in
    mixed precision, without prepareFTsource: R2C, solveModifiedPoissonFT with
    a screening term, C2R."""
    N = 768
    o = oracle()
    dx = 1.0 / N
    source = noise(N, 111)
    FT = rfft3(source, N)
    o.solve_poisson(N, ptr(FT), ptr(FT), 1 / (dx * dx), 40.0)
    ph_ref = irfft3(FT, N)
    del FT
    with ctx(N, gev.MIXED) as c:
        c.set_field(gev.FIELD_SOURCE, source)
        c.solve_phi(False, 0.0, 0.0, 0.0, 0.0, 1 / (dx * dx), 40.0)
        assert rel_err(c.get_field(gev.FIELD_PHI), ph_ref) < TOL[gev.MIXED]


@pytest.mark.parametrize("N", SIZES)
def test_solve_chi_tensor_sizes(N):
    """prepareFTsource (Tij form) + 6 R2C + projectFTscalar + C2R (main.cu:811-903)
    with the tensor state on: projectFTtensor on the first cycle, then one
    evolveFTtensor step (main.cu:961-965); h_ij and h_ij' compared as complex
    spectra, chi in real space."""
    o = oracle()
    dx = 1.0 / N
    n3 = N ** 3
    Tij = noise(N, 120, 1e-3, 6)
    phi = noise(N, 121, 1e-5)
    coeff = 2 * FOURPIG * dx * dx / 0.4
    S = np.zeros(6 * n3)
    o.prepare_Tij(N, ptr(phi), ptr(Tij), coeff, ptr(S))
    SFT = np.empty((6, N, N, N // 2 + 1), dtype=np.complex128)
    for k in range(6):
        SFT[k] = rfft3(S[k * n3:(k + 1) * n3], N)
    del S
    chiFT = np.zeros((N, N, N // 2 + 1), dtype=np.complex128)
    o.project_scalar(N, ptr(SFT), ptr(chiFT), 0)
    chi_ref = irfft3(chiFT, N)
    del chiFT
    hFT = np.zeros_like(SFT)
    o.project_tensor(N, ptr(SFT), ptr(hFT))
    hubble, dtau, dtau_old = 0.9, 0.01, 0.012
    h1, hp1 = hFT.copy(), np.zeros_like(hFT)
    o.evolve_tensor(N, ptr(SFT), ptr(h1), ptr(hp1), hubble, dtau, dtau_old)   # modifies SFT's trace at k = 0
    del SFT
    for prec in PRECS:
        with ctx(N, prec, tensor=True) as c:
            c.set_field(gev.FIELD_SIJ, Tij)
            c.set_field(gev.FIELD_PHI, phi)
            c.solve_chi(coeff, cycle0=True)
            assert rel_err(c.get_field(gev.FIELD_CHI), chi_ref) < TOL[prec], prec
            assert rel_err(c.get_field(gev.FIELD_HIJ_FT), hFT) < TOL[prec], prec
            c.solve_chi(coeff, cycle0=False, hubble=hubble, dtau=dtau, dtau_old=dtau_old)
            assert rel_err(c.get_field(gev.FIELD_CHI), chi_ref) < TOL[prec], prec
            assert rel_err(c.get_field(gev.FIELD_HIJ_FT), h1) < TOL[prec], prec
            assert rel_err(c.get_field(gev.FIELD_HIJP_FT), hp1) < TOL[prec], prec


@pytest.mark.parametrize("N", SIZES)
def test_solve_B_sizes(N):
    """3 R2C + projectFTvector + 3 C2R (main.cu:905-955)."""
    o = oracle()
    dx = 1.0 / N
    n3 = N ** 3
    T0i = noise(N, 130, 1e-4, 3)
    FT = np.empty((3, N, N, N // 2 + 1), dtype=np.complex128)
    for k in range(3):
        FT[k] = rfft3(T0i[k * n3:(k + 1) * n3], N)
    coeff = FOURPIG * dx * dx
    o.project_vector(N, ptr(FT), ptr(FT), coeff, 0.0)
    B_ref = np.concatenate([irfft3(FT[k], N) for k in range(3)])
    del FT
    for prec in PRECS:
        with ctx(N, prec) as c:
            c.set_field(gev.FIELD_BI, T0i)
            c.solve_B(coeff)
            assert rel_err(c.get_field(gev.FIELD_BI).ravel(), B_ref) < TOL[prec], prec


@pytest.mark.parametrize("tensor,parabolic", [(True, False), (False, True)])
def test_solve_chi_extras_768_mixed(tensor, parabolic):
    """h_ij and parabolic B_i on the largest grid.  The sources are a 256^3
    white-noise box repeated three times along each axis: its modes are the
    multiples of three of the 768^3 grid, where every k of the lattice is three
    times that of the small grid.  With the time step a third, the Hubble rate
    three times and a^2 dtau a ninth, chi, B_i and h_ij are those of the small
    box, and h_ij vanishes at all other modes; the small box is the oracle's.
    h_ij goes through both cycles: projectFTtensor, then evolveFTtensor."""
    n, N = 256, 768
    o = oracle()
    n3 = n ** 3
    Tij = noise(n, 150, 1e-3, 6)
    phi = noise(n, 151, 1e-5)
    coeff, hubble, dtau, dtau_old, a2dtau = 1e-3, 0.9, 0.01, 0.012, 0.3
    S = np.zeros(6 * n3)
    o.prepare_Tij(n, ptr(phi), ptr(Tij), coeff, ptr(S))
    SFT = np.stack([rfft3(S[k * n3:(k + 1) * n3], n) for k in range(6)])
    G = np.zeros((n, n, n // 2 + 1), dtype=np.complex128)
    o.project_scalar(n, ptr(SFT), ptr(G), 0)
    chi_ref = irfft3(G, n)
    B = np.zeros((3, n, n, n // 2 + 1), dtype=np.complex128)
    o.evolve_vector(n, ptr(SFT), ptr(B), a2dtau)
    B_ref = [irfft3(B[k], n) for k in range(3)]
    h = np.zeros_like(SFT)
    hp = np.zeros_like(SFT)
    o.project_tensor(n, ptr(SFT), ptr(h))
    o.evolve_tensor(n, ptr(SFT), ptr(h), ptr(hp), hubble, dtau, dtau_old)
    tile = lambda f: np.tile(f.reshape(-1, n, n, n), (1, 3, 3, 3)).ravel()  # noqa: E731
    kw = dict(tensor=tensor, vector_method=gev.VECTOR_PARABOLIC if parabolic else gev.VECTOR_ELLIPTIC)
    with ctx(N, gev.MIXED, **kw) as c:
        c.set_field(gev.FIELD_PHI, tile(phi))
        tiled = tile(Tij)
        for cycle0 in (True, False):
            c.set_field(gev.FIELD_SIJ, tiled)
            c.solve_chi(coeff, cycle0=cycle0, hubble=3 * hubble, dtau=dtau / 3, dtau_old=dtau_old / 3,
                        a2dtau=0.0 if cycle0 else a2dtau / 9)
        del tiled
        assert rel_err(c.get_field(gev.FIELD_CHI), tile(chi_ref)) < TOL[gev.MIXED]
        if parabolic:
            got = c.get_field(gev.FIELD_BI)
            for k in range(3):
                assert rel_err(got[k], tile(B_ref[k])) < TOL[gev.MIXED], k
            del got
        if tensor:
            got = c.get_field(gev.FIELD_HIJ_FT)
            sub = got[:, ::3, ::3, ::3]
            assert rel_err(sub, h) < TOL[gev.MIXED]
            sub[...] = 0.0
            assert max(np.abs(g).max() for g in got) < TOL[gev.MIXED] * np.abs(h).max()


@pytest.mark.parametrize("N,bound", [(128, 2.487e-7), (256, 2.715e-7), (384, 3.054e-7), (512, 2.860e-7), (768, 3.138e-7)])
def test_transform_rounding_fp32(N, bound):
    """Rounding error of the FP32 transforms alone: a screening far above every
    k^2 makes the solve a multiplication by -1, so that forward and back of
    white noise return its negative.  The bound is what radix-8 Stockham
    transforms of the same lines show for these inputs (it scatters by 0.1 %
    between seeds): the transforms must not be less exact than those."""
    f = np.random.default_rng(140).standard_normal(N ** 3, dtype=np.float32).astype(np.float64)
    with ctx(N, gev.MIXED) as c:
        c.set_field(gev.FIELD_SOURCE, f)
        c.solve_phi(False, 0.0, 0.0, 0.0, 0.0, 1e18, 1e18)
        d = c.get_field(gev.FIELD_PHI).ravel()
    d += f
    assert np.linalg.norm(d) / np.linalg.norm(f) < 1.002 * bound


@pytest.mark.parametrize("N", [256, 384, 512, 768])
def test_transforms_fp64(N):
    """The same round trip in FP64, on each side of the sizes from which the z
    pass (384) and the y pass (512 only) are staged by bulk copies.  A chain of
    60 butterfly levels rounds by about 60^(1/2) x 1.1e-16; the bound is ten
    times that."""
    f = np.random.default_rng(141).standard_normal(N ** 3)
    with ctx(N, gev.FP64) as c:
        c.set_field(gev.FIELD_SOURCE, f)
        c.solve_phi(False, 0.0, 0.0, 0.0, 0.0, 1e22, 1e22)
        d = c.get_field(gev.FIELD_PHI).ravel()
    d += f
    assert np.linalg.norm(d) / np.linalg.norm(f) < 1e-14
