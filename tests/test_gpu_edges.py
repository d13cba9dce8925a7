"""The kernels' own edges: every grid whose x and y transforms run as one plane
kernel and the first that does not, spectra with few and many bins, particle
arrays that the cell-ordered fast paths must not rely on, unaligned caller
arrays and recorded graphs of the allocation-free solve, and positions far
outside the box in the differentiable run.

Tolerances: as in test_gpu_parity (FP64 1e-10, mixed 2e-5 for deposits and
1e-4 for solves, relative to the largest magnitude); where two runs of the
library do the same arithmetic, equality."""
import numpy as np
import pytest

from _fixtures import irfft3, particles, rel_err, rfft3, smooth_field, trough_phi
from _libs import kshape, oracle, ptr

gev = pytest.importorskip("gevb200")
torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

TOL = {gev.FP64: 1e-10, gev.MIXED: 1e-4}
PRECS = [gev.FP64, gev.MIXED]


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("N", [16, 32, 64, 128, 256])
def test_solves_with_their_preparations(prec, N):
    """Phi (T00 preparation and its sum), chi (Tij preparation) and B_i (plain
    rows) on each side of the plane kernels' size limit."""
    o = oracle()
    n3 = N ** 3
    src = 0.32 * (1.0 + smooth_field(N, 1, 0.1))
    phi, chi = smooth_field(N, 2, 1e-5), smooth_field(N, 3, 1e-7)
    Tij = np.concatenate([smooth_field(N, 4 + c, 1e-5) for c in range(6)])
    T0i = np.concatenate([smooth_field(N, 14 + c, 1e-4) for c in range(3)])
    with gev.Context(N, precision=prec, capacity=1) as c:
        c.set_field(gev.FIELD_SOURCE, src); c.set_field(gev.FIELD_PHI, phi); c.set_field(gev.FIELD_CHI, chi)
        c.set_field(gev.FIELD_SIJ, Tij); c.set_field(gev.FIELD_BI, T0i)
        c.solve_chi(1e-3)
        chi_g = c.get_field(gev.FIELD_CHI)
        c.set_field(gev.FIELD_CHI, chi)
        c.solve_B(1e-3)
        B_g = c.get_field(gev.FIELD_BI)
        total, hom = c.solve_phi(True, 0.32, 1e-4, 2e-4, 3e-4, float(N * N), 1.5)
        phi_g = c.get_field(gev.FIELD_PHI)
    out = np.zeros(n3)
    s = o.prepare_T00(N, ptr(phi), ptr(chi), ptr(src), 0.32, 1e-4, 2e-4, 3e-4, ptr(out))
    assert abs(total / s - 1.0) < (1e-12 if prec == gev.FP64 else 1e-6)
    F = np.ascontiguousarray(rfft3(out, N)); G = np.zeros(kshape(N), dtype=np.complex128)
    o.solve_poisson(N, ptr(F), ptr(G), float(N * N), 1.5)
    assert rel_err(phi_g, irfft3(G, N)) < TOL[prec]
    assert abs(hom - G[0, 0, 0].real) < TOL[prec] * np.abs(G).max()
    S = np.zeros(6 * n3)
    o.prepare_Tij(N, ptr(phi), ptr(Tij), 1e-3, ptr(S))
    F = np.ascontiguousarray(np.stack([rfft3(S[k * n3:(k + 1) * n3], N) for k in range(6)]))
    o.project_scalar(N, ptr(F), ptr(G), 0)
    assert rel_err(chi_g, irfft3(G, N)) < TOL[prec]
    F = np.ascontiguousarray(np.stack([rfft3(T0i[k * n3:(k + 1) * n3], N) for k in range(3)]))
    G3 = np.zeros((3,) + kshape(N), dtype=np.complex128)
    o.project_vector(N, ptr(F), ptr(G3), 1e-3, 0.0)
    for k in range(3):
        assert rel_err(B_g[k], irfft3(G3[k], N)) < TOL[prec], k


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("N,bins", [(16, 1), (16, 300), (32, 33), (64, 1024)])
def test_power_spectrum_bins(prec, N, bins):
    """P(k) of particles in no cell order that the density kernel can use (a
    cell with more particles than a sorted bucket holds, a row of neighbouring
    cells across the box edge) against the oracle."""
    rng = np.random.default_rng(5)
    clump = (np.array([N - 0.5, 3.5, 7.5]) + 0.4 * (rng.random((1500, 3)) - 0.5)) / N
    row = np.stack([np.arange(N) / N + 0.3 / N, np.full(N, 0.5), np.full(N, 0.25)], axis=1)
    pos = np.remainder(np.concatenate([rng.random((3000, 3)), clump, row, row]), 1.0)
    mass = 0.32 / len(pos)
    rho = np.zeros(N ** 3)
    o = oracle()
    o.project_cic(N, len(pos), ptr(np.ascontiguousarray(pos)), mass, ptr(rho))
    F = np.ascontiguousarray(rfft3(rho, N))
    ref = [np.zeros(bins) for _ in range(4)]
    occ = np.zeros(bins, dtype=np.int32)
    o.lib.orc_power_spectrum(N, ptr(F), bins, *[ptr(r) for r in ref], ptr(occ), 0.0)
    with gev.Context(N, precision=prec, capacity=len(pos)) as c:
        c.set_particles(pos, np.zeros_like(pos), None, mass)
        for _ in range(2):   # the bins start from zero on every call
            kb, pw, ks, ps, oc = c.power_spectrum(bins)
        assert rel_err(c.get_field(gev.FIELD_SOURCE), rho) < (1e-10 if prec == gev.FP64 else 2e-7)
    # both precisions measure in FP64 (sums in another order: 1e-10)
    assert np.array_equal(oc, occ)
    assert rel_err(kb, ref[0]) < 1e-10 and rel_err(pw, ref[1]) < 1e-10
    assert rel_err(np.hypot(pw, ps), np.hypot(ref[1], ref[3])) < 1e-9


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025])
def test_rebin_ranks_one_dense_cell(n):
    """A single cell of n particles with shuffled IDs: in ID order up to the
    sorted-bucket limit (1024), complete beyond it."""
    N = 16
    rng = np.random.default_rng(n)
    pos = (np.array([3.0, 4.0, 5.0]) + rng.random((n, 3))) / N
    ids = rng.permutation(n).astype(np.int64) * 5 + 1
    with gev.Context(N, precision=gev.MIXED, capacity=n) as c:
        c.set_particles(pos, np.zeros_like(pos), ids, 1.0)
        _, _, got = c.get_particles()
    assert np.array_equal(np.sort(got), np.sort(ids))
    if n <= 1024:
        assert np.all(np.diff(got) > 0)


@pytest.mark.parametrize("prec", PRECS)
def test_dense_tile_list_is_left_empty(prec):
    """Deposits with dense tiles in a row, then one without any: each equal to
    the same deposit on a context of its own (the tile list starts empty)."""
    N = 32
    dense = particles(N, n=90000, seed=6)
    phi = trough_phi(N)

    def deposit(c, p):
        c.set_particles(*p, 1e-5)
        c.set_field(gev.FIELD_PHI, phi)
        c.project(gev.PROJ_T00 | gev.PROJ_TIJ, 0.5, 1.0, True)
        return c.get_field(gev.FIELD_SOURCE), c.get_field(gev.FIELD_SIJ)

    sparse = tuple(x[:20000] for x in dense)
    with gev.Context(N, precision=prec, capacity=90000) as c:
        runs = [deposit(c, p) for p in (dense, dense, sparse)]
    for p, got in ((dense, runs[1]), (sparse, runs[2])):
        with gev.Context(N, precision=prec, capacity=90000) as c:
            for x, y in zip(deposit(c, p), got):
                assert np.array_equal(x, y)


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("N", [16, 32, 64, 128])
def test_noalloc_unaligned_and_recorded(prec, N):
    """Arrays aligned to single values only give what aligned ones give, and a
    recorded graph of the solve replays it."""
    dt = torch.float64 if prec == gev.FP64 else torch.float32
    g = torch.Generator(device="cuda").manual_seed(N)
    src = torch.randn(N ** 3, generator=g, device="cuda", dtype=dt)
    ref, out = torch.empty_like(src), torch.empty_like(src)
    s1 = torch.empty(N ** 3 + 1, device="cuda", dtype=dt)[1:]
    o1 = torch.empty(N ** 3 + 1, device="cuda", dtype=dt)[1:]
    s1.copy_(src)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    solve = lambda a, b: gev.poisson_noalloc(N, prec, a.data_ptr(), b.data_ptr(), 0.7, 1e-2, stream.cuda_stream)
    with torch.cuda.stream(stream):
        assert solve(src, ref) == gev.GEV_OK
        assert solve(s1, o1) == gev.GEV_OK
    stream.synchronize()
    assert torch.isfinite(ref).all() and torch.equal(ref, o1)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        assert solve(src, out) == gev.GEV_OK
    for _ in range(2):
        out.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, ref)


@pytest.mark.parametrize("N,n", [(16, 1), (32, 777), (128, 5000)])
def test_pm_positions_far_outside_the_box(N, n):
    """Positions are unwrapped: shifting every particle by whole boxes (the
    quotient that reduces a cell is then large and negative as well) changes
    neither the density nor the gradients beyond the rounding of x."""
    from gevb200 import pm as gpm
    rng = np.random.default_rng(N)
    x = torch.from_numpy(rng.random((n, 3))).cuda()
    q = torch.from_numpy(1e-3 * rng.standard_normal((n, 3))).cuda()
    shift = torch.from_numpy(rng.integers(-40, 40, (n, 3)).astype(np.float64)).cuda()
    coef, _ = gpm.schedule(N, 0.01, 0.32, 0.68, 0.1, 1.0, 3)
    res = []
    for y in (x, x + shift):
        pm = gpm.PM(N, n, 0.32 / n, gev.FP64, checkpoint_every=2)
        d = torch.empty(N ** 3, dtype=torch.float64, device="cuda")
        xo, qo, gx, gq = (torch.empty_like(x) for _ in range(4))
        pm.forward(coef, y, q, d, xo, qo)
        w = torch.from_numpy(np.random.default_rng(1).standard_normal(N ** 3)).cuda()
        torch.cuda.synchronize()
        pm.adjoint(w, gx, gq)
        res.append((d, xo - y, qo, gx, gq))
        pm.close()
    # x + 40 keeps x to 2^-53 x 40 = 4.4e-15 boxes, 6e-13 cells at N = 128: that
    # times the run's own amplification, which is what makes the gradients
    # (up to 6e5 here) larger than those of a single deposit (N x |w|, about 5e2)
    for k, (a, b) in enumerate(zip(*res)):
        assert rel_err(a.cpu().numpy(), b.cpu().numpy()) < (1e-10 if k < 3 else 6e-13 * 1.2e3 * 4), k


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("N", [64, 128])
def test_failed_cycle_leaves_the_particles(N, prec):
    """An error that arises before the kick (here the lightcone's ID log, sized
    for the one particle that was there at first, overflows) leaves particles
    and state as they were, on both sides of the size from which the kick can
    be launched early; the next call finds the error cleared and the particles
    in order."""
    n = 100000
    rng = np.random.default_rng(9)
    r = np.abs(rng.standard_normal((n, 3))) + 0.05
    pos = np.ascontiguousarray(0.971 * r / np.linalg.norm(r, axis=1)[:, None])
    q = 1e-4 * rng.standard_normal((n, 3))
    ids = np.arange(n, dtype=np.int64)
    fpg = 1.5 * (5.0 * N) ** 2 / 2997.92458 ** 2
    cosmo = gev.Cosmo(0.32, 0.68, 0.0, fpg, 48.0, 0.04, 200.0, 5.0 * N)
    shell = gev.LightconeArgs((0.0, 0.0, 0.0), (1.0 / np.sqrt(3.0),) * 3, -1.0, (1.0, 0.3), 1.98, 1, 0)
    with gev.Context(N, precision=prec, capacity=n, boxsize=5.0 * N) as c:
        c.set_particles(np.full((1, 3), 0.5), np.zeros((1, 3)))
        c.lightcone(shell, 1.0, 0.02, 0.02, 0.5, 0.1, 16)
        c.set_particles(pos, q, ids, 0.32 / n)
        before = [x[np.argsort(c.get_particles()[2])] for x in c.get_particles()]
        st = gev.State(0.5, 1.0, 0.02, 0.02, 7, 0.0, 0.0, 0.0)
        with pytest.raises(gev.GevError) as e:
            c.step_lightcone(cosmo, st, shell, n)
        assert e.value.code == 4 and "0x2 " in str(e.value), str(e.value)
        assert (st.a, st.tau, st.dtau, st.cycle, st.maxvel) == (0.5, 1.0, 0.02, 7, 0.0)
        after = [x[np.argsort(c.get_particles()[2])] for x in c.get_particles()]
        assert all(np.array_equal(x, y) for x, y in zip(before, after))
        c.step(cosmo, st)
        assert st.cycle == 8
        moved = [x[np.argsort(c.get_particles()[2])] for x in c.get_particles()]
        assert np.array_equal(moved[2], ids) and not np.array_equal(moved[0], before[0])


@pytest.mark.parametrize("prec", PRECS)
def test_pm_arrays_off_the_double_boundary(prec):
    """Caller's particle arrays at any byte address, as the copies of the run
    have always taken them: the results are those of aligned arrays, bit for
    bit where no atomics are summed in between (one step, few particles far
    apart)."""
    from gevb200 import pm as gevpm

    N, n = 16, 5
    x = (torch.arange(3 * n, device="cuda", dtype=torch.float64).reshape(n, 3) * 3.0 % 15.0 + 0.25) / N
    q = 1e-3 * torch.ones((n, 3), device="cuda", dtype=torch.float64)
    run = gevpm.PM(N, n, 0.32 / n, prec, checkpoint_every=1)
    coef = np.array([0.1, 0.2, 1.0])

    class At:
        """3 n doubles whose first byte lies `off` bytes into a buffer."""

        def __init__(self, values, off):
            self.raw = torch.zeros(24 * n + 16, dtype=torch.uint8, device="cuda")
            self.off = off
            if values is not None:
                self.raw[off:off + 24 * n] = values.reshape(-1).view(torch.uint8)

        def data_ptr(self):
            return self.raw.data_ptr() + self.off

        def values(self):
            return self.raw[self.off:self.off + 24 * n].clone().view(torch.float64)

    out = []
    for off in (0, 4):
        a = [At(v, off) for v in (x, q, None, None, None, None)]
        delta = torch.empty(N ** 3, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        run.forward(coef, a[0], a[1], delta, a[2], a[3])
        run.adjoint(torch.ones_like(delta), a[4], a[5])
        out.append([delta] + [v.values() for v in a[2:]])
    for u, v in zip(*out):
        assert torch.isfinite(u).all() and torch.equal(u, v)


def test_pm_host_array_is_no_gpu_fault():
    """A pageable host array, which the run does not take, is an error of the
    call (or, where the driver can copy it, taken), and the context goes on."""
    from gevb200 import pm as gevpm

    N, n = 16, 5
    run = gevpm.PM(N, n, 0.32 / n, gev.FP64, checkpoint_every=1)
    delta = torch.empty(N ** 3, dtype=torch.float64, device="cuda")
    host = torch.full((n, 3), 0.5, dtype=torch.float64)
    torch.cuda.synchronize()
    try:
        run.forward(np.array([0.1, 0.2, 1.0]), host, host, delta)
    except gev.GevError as e:
        assert e.code == 2, str(e)
    run.forward(np.array([0.1, 0.2, 1.0]), host.cuda(), host.cuda(), delta)
    assert torch.isfinite(delta).all()


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("bins", [4096, 4097, 200001])
def test_power_spectrum_many_bins(prec, bins):
    """On each side of the number of bins from which they are kept once."""
    test_power_spectrum_bins(prec, 16, bins)


def test_power_spectrum_workspace():
    """The device memory of a spectrum with very many bins is that of the five
    sums per bin (160 MB here), with some room for the allocator."""
    with gev.Context(16, precision=gev.FP64, capacity=8) as c:
        c.set_particles(np.full((1, 3), 0.5), np.zeros((1, 3)))
        c.power_spectrum(16)
        free = torch.cuda.mem_get_info()[0]
        c.power_spectrum(4000000)
        assert free - torch.cuda.mem_get_info()[0] < 2 * 160e6
