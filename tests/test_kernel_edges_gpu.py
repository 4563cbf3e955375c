"""The kernels' edges: the sizes and routes at which a dispatch rule or a
kernel's remainder handling can go wrong, against the oracle.

Tolerances: FP64 paths 1e-11 and FP32 paths 1e-5 relative L2, the bounds of the
other parity tests (measured 1e-13 and 1e-7); element-wise kernels to a few
roundings of their own type."""
import numpy as np
import pytest
import torch

from oracle import collision as oc
from oracle import fno as ofno
from oracle import mesh as om
from oracle.collision import vhs_gll_fs
from tests._cases import op_kwargs, vhs_case, vhs_tables
from tests.test_fno_oracle import _maxwellians

pytestmark = pytest.mark.gpu
TOL = {'fp64': 1e-11, 'fp32': 1e-5}


def _rel(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / np.linalg.norm(np.ravel(b)))


@pytest.fixture(scope='module', autouse=True)
def built():
    from dgfs1d_gpu_b200 import build
    build.build()


# one radial point (no pair), an odd number of them (the last pair is half),
# every direction in a slice of its own, and a batch that fills the slices
# unevenly; the smallest and the largest grid of each terms kernel
@pytest.mark.parametrize('precision', ['fp64', 'fp32'])
@pytest.mark.parametrize('N,M,full,Nrho,points', [
    (8, 6, False, 1, 1), (8, 12, True, 5, 3), (16, 6, False, 3, 1),
    (16, 6, True, 8, 7), (24, 6, False, 1, 1), (24, 6, True, 3, 2),
    (32, 6, True, 1, 1), (32, 6, False, 3, 2), (48, 6, True, 1, 1)])
def test_direction_slices_and_radial_remainders(precision, N, M, full, Nrho, points):
    from dgfs1d_gpu_b200.collision import VHSOperator
    vm, prefac, gamma, f = vhs_case(N, M, Nrho, 6.0, full, nslots=points)
    tab = vhs_tables(vm, gamma)
    op = VHSOperator(**op_kwargs(vm, prefac, gamma), precision=precision,
                     max_evals=points)
    fd = torch.tensor(f, device='cuda')
    Q = torch.full_like(fd, 0.5)
    op.eval(fd, Q)
    got = Q.cpu().numpy() - 0.5
    for s in range(points):
        ref = vhs_gll_fs(tab, prefac, f[s])
        # += onto 0.5 rounds at 1e-16 of 0.5; the bound covers it
        floor = 1e-16 * np.sqrt(ref.size) / np.linalg.norm(ref)
        assert _rel(got[s], ref) < TOL[precision] + floor, (N, Nrho, s)


@pytest.mark.parametrize('points', [1, 3, 6, 8, 10, 12, 16])
def test_default_terms_kernel_by_batch_size(points):
    """N=32, FP32: the default kernel and its direction slices follow the batch
    size; at each the values of every variant, and (10% allowed for the timing)
    no more time than the kernel of clusters of four, which a default fixed for
    24 points once exceeded by 14% at 8 points."""
    from dgfs1d_gpu_b200.collision import VHSOperator
    vm, prefac, gamma, f = vhs_case(32, 12, 8, 6.0, True, nslots=points)
    op = VHSOperator(**op_kwargs(vm, prefac, gamma), precision='fp32', max_evals=points)
    fd = torch.tensor(f, device='cuda')
    st = torch.cuda.Stream()

    def run(code):
        op.set_variant(code)
        Q, T = torch.zeros_like(fd), torch.zeros_like(fd)
        with torch.cuda.stream(st):
            op.eval(fd, Q, stream=st)
        st.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            for _ in range(5):
                op.eval(fd, T, stream=st)
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        ms = []
        for _ in range(8):
            a.record()
            g.replay()
            b.record()
            b.synchronize()
            ms.append(a.elapsed_time(b))
        del g
        return Q.cpu().numpy(), min(ms)
    ref, t504 = run(504)
    for code in (0, 608, 616):
        Q, t = run(code)
        assert _rel(Q, ref) < 1e-6, code
        if code == 0:
            assert t < 1.1 * t504, (t, t504)


@pytest.mark.parametrize('N', [16, 24])
def test_radial_points_of_very_different_weight(N):
    """Two radial points share a forward transform: the sum of the small radius
    is large and its weight small, and its rounding must not enter with the
    other's weight.  Bound: twice the error with a transform for each (1.2e-13
    and 2.2e-12, from the cancellation of the far radius' sums); 6.9e-13 and
    1.3e-11 unscaled.  N=16: one-CTA kernel, N=24: cluster kernel."""
    from dgfs1d_gpu_b200.collision import VHSOperator
    vm, prefac, gamma, f = vhs_case(N, 6, 2, 6.0, False)
    vm.qz, vm.qw = np.array([0.05, 4.0]), np.array([1.0, 1.0])
    op = VHSOperator(**op_kwargs(vm, prefac, gamma), precision='fp64', max_evals=1)
    fd = torch.tensor(f, device='cuda')
    Q = torch.zeros_like(fd)
    op.eval(fd, Q)
    ref = vhs_gll_fs(vhs_tables(vm, gamma), prefac, f[0])
    assert _rel(Q[0].cpu().numpy(), ref) < {16: 2.5e-13, 24: 4.4e-12}[N]


def test_sliced_and_unsliced_batches_agree():
    """A point evaluated alone (sliced directions) and within a batch."""
    from dgfs1d_gpu_b200.collision import VHSOperator
    for N, precision in ((16, 'fp32'), (24, 'fp32'), (16, 'fp64'), (24, 'fp64')):
        vm, prefac, gamma, f = vhs_case(N, 6, 6, 5.0, True, nslots=40)
        op = VHSOperator(**op_kwargs(vm, prefac, gamma), precision=precision,
                         max_evals=40)
        fd = torch.tensor(f, device='cuda')
        Qb, Q1 = torch.zeros_like(fd), torch.zeros_like(fd[:1])
        op.eval(fd, Qb)
        op.eval(fd[:1].contiguous(), Q1)
        assert _rel(Q1[0].cpu().numpy(), Qb[0].cpu().numpy()) < \
            (1e-6 if precision == 'fp32' else 1e-12)


@pytest.mark.parametrize('precision', ['fp64', 'fp32'])
@pytest.mark.parametrize('N', [8, 16, 24, 32])
def test_vss_merged_antipodes_and_radial_slices(N, precision):
    """A species with itself: the same array twice (antipodal directions share
    a transform) and two equal arrays (every direction on its own); few and
    many points (one radial point and several per slice); the oracle."""
    from dgfs1d_gpu_b200.collision import VSSOperator
    masses = [1.0, 1.7]
    vm = om.VelocityMeshBi(Nv=N, M=6, masses=masses, Nrho=3, dev=5.0)
    szpre = om.sphere_design(12)
    rng = np.random.default_rng(3)
    m = 0.5 * np.exp(-np.sum(vm.cv ** 2, axis=0)) / np.pi ** 1.5
    f = np.stack([m * (1 + 0.02 * rng.uniform(-1, 1, m.shape)) for _ in range(3)])
    one = np.ones((2, 2))
    op = VSSOperator(N, vm.L, vm.qz, vm.qw, vm.sz, vm.sw, szpre, masses,
                     0.38 * one, 0.4 * one, 0.1 * one, max_evals=200 if N < 32 else 3,
                     precision=precision)
    fd = torch.tensor(f, device='cuda')
    Q1, Q2 = torch.zeros_like(fd), torch.zeros_like(fd)
    op.eval(1, 1, fd, fd, Q1)
    op.eval(1, 1, fd, fd.clone(), Q2)
    tol = TOL[precision]
    assert _rel(Q1.cpu().numpy(), Q2.cpu().numpy()) < tol
    tab = oc.VSSTables(N, vm.L, vm.qz, vm.qw, vm.sz, vm.sw, szpre, 0.38, 0.4, 0.5)
    ref = oc.vss_fs(tab, 0.1, masses[1], masses[1], f[0], f[0])
    assert _rel(Q1.cpu().numpy()[0], ref) < tol
    if N < 32:      # 200 points: fewer radial slices than radial points in FP64
        fb = fd[:1].expand(200, -1).contiguous()
        Qb = torch.zeros_like(fb)
        op.eval(1, 1, fb, fb, Qb)
        assert _rel(Qb[199].cpu().numpy(), ref) < tol


def test_scratch_is_bounded():
    """Handles for thousands of points of a large grid fit beside a solver's
    state, and a call longer than a pass gives every point its value."""
    from dgfs1d_gpu_b200.collision import VHSOperator, VSSOperator
    masses = [1.0, 2.0]
    vm = om.VelocityMeshBi(Nv=32, M=12, masses=masses, Nrho=16, dev=5.0)
    one = np.ones((2, 2))
    f = np.stack([np.exp(-np.sum(vm.cv ** 2, axis=0) / T) for T in (1.0, 1.2)])
    fd = torch.tensor(f, device='cuda')
    torch.cuda.synchronize()
    for precision in ('fp64', 'fp32'):
        free = torch.cuda.mem_get_info()[0]
        op = VSSOperator(32, vm.L, vm.qz, vm.qw, vm.sz, vm.sw, om.sphere_design(32),
                         masses, 0.38 * one, 0.4 * one, 0.1 * one, max_evals=6000,
                         precision=precision)
        assert free - torch.cuda.mem_get_info()[0] < 6 << 30, precision
        many = 230 if precision == 'fp64' else 330
        fp, fq = (x.expand(many, -1).contiguous() for x in (fd[:1], fd[1:]))
        Q, Q1 = torch.zeros_like(fp), torch.zeros_like(fp[:1])
        op.eval(0, 1, fp, fq, Q)
        op.eval(0, 1, fp[:1], fq[:1], Q1)
        for i in (0, many // 2, many - 1):
            assert _rel(Q[i].cpu().numpy(), Q1[0].cpu().numpy()) < TOL[precision], i
        op.close()
    vm, prefac, gamma, f = vhs_case(48, 32, 24, 6.0, True)
    free = torch.cuda.mem_get_info()[0]
    op = VHSOperator(**op_kwargs(vm, prefac, gamma), precision='fp64', max_evals=3000)
    assert free - torch.cuda.mem_get_info()[0] < 6 << 30
    fb = torch.tensor(f, device='cuda').expand(70, -1).contiguous()
    Q, Q1 = torch.zeros_like(fb), torch.zeros_like(fb[:1])
    op.eval(fb, Q)
    op.eval(fb[:1].contiguous(), Q1)
    for i in (0, 69):
        assert _rel(Q[i].cpu().numpy(), Q1[0].cpu().numpy()) < 1e-11, i


@pytest.mark.parametrize('points', [1, 2, 3, 4, 7])
def test_vss_gain_by_batch_size(points):
    """FP32 mixture gain with one, two and three points per thread, the last group
    part-filled, one launch for the pairs (up to three points at N=24) and one
    each: the FP64 mode's values."""
    from dgfs1d_gpu_b200.collision import VSSOperator
    masses = [1.0, 1.7]
    vm = om.VelocityMeshBi(Nv=24, M=6, masses=masses, Nrho=3, dev=5.0)
    one = np.ones((2, 2))
    rng = np.random.default_rng(9)
    fs = []
    for T in (1.0, 1.2):
        m = 0.5 * np.exp(-np.sum(vm.cv ** 2, axis=0) / T) / (np.pi * T) ** 1.5
        fs.append(torch.tensor(np.stack([
            m * (1 + 0.02 * rng.uniform(-1, 1, m.shape)) for _ in range(points)]),
            device='cuda'))
    Q = {}
    for precision in ('fp64', 'fp32'):
        op = VSSOperator(24, vm.L, vm.qz, vm.qw, vm.sz, vm.sw, om.sphere_design(12),
                         masses, 0.38 * one, 0.4 * one, 0.1 * one, max_evals=points,
                         precision=precision)
        Q[precision] = [torch.zeros_like(x) for x in fs]
        for p in range(2):
            op.eval_species(p, fs, Q[precision][p])
    for p in range(2):
        for i in range(points):
            assert _rel(Q['fp32'][p][i].cpu().numpy(),
                        Q['fp64'][p][i].cpu().numpy()) < TOL['fp32'], (p, i)


@pytest.mark.parametrize('dtype', [torch.float64, torch.float32])
def test_axnpby_vector_and_scalar_routes(dtype):
    """Sizes around the vector kernel's groups, operands off 16-byte alignment
    (scalar route), 1 to 4 terms and the three cases of a0."""
    from dgfs1d_gpu_b200.dg import axnpby
    eps = torch.finfo(dtype).eps
    for n in (1, 2, 3, 4, 1023, 1024, 1026, 4096 + 8):
        for shift in (0, 1):
            for nt in (1, 2, 3, 4):
                for a0 in (0.0, 1.0, 0.25):
                    bufs = [torch.randn(n + 4, dtype=dtype, device='cuda')[shift:shift + n]
                            for _ in range(nt + 1)]
                    x0 = bufs[0].clone() if shift == 0 else bufs[0]
                    co = [0.5, -1.25, 2.0, 0.75][:nt]
                    ref = a0 * x0.double() if a0 else torch.zeros_like(x0, dtype=torch.float64)
                    mag = ref.abs()
                    for c, x in zip(co, bufs[1:]):
                        ref = ref + c * x.double()
                        mag = mag + abs(c) * x.double().abs()
                    if a0 == 0.0:
                        x0.fill_(float('nan'))      # not read
                    axnpby(x0, a0, *[v for p in zip(co, bufs[1:]) for v in p])
                    assert ((x0.double() - ref).abs() <= 4 * eps * mag + 1e-300).all(), \
                        (n, shift, nt, a0)


@pytest.mark.parametrize('Ne,K', [(1, 3), (2, 2), (3, 3), (5, 5), (17, 3)])
@pytest.mark.parametrize('bc', ['dgfs-wall-diffuse', 'dgfs-inlet'])
def test_advection_split_over_elements(Ne, K, bc):
    """The walk split into pieces of every length (a small velocity grid
    splits it into single elements, N=32 into a few) against the oracle."""
    from dgfs1d_gpu_b200.basis import get_basis
    from dgfs1d_gpu_b200.config import Config
    from dgfs1d_gpu_b200.dg import DGOperator
    from oracle import dg as od
    for N in (8, 32):
        L = 5.0
        c0 = np.linspace(-L + L / N, L - L / N, N)
        cv = np.stack([x.ravel() for x in np.meshgrid(c0, c0, c0, indexing='ij')])
        cw = (2 * L / N) ** 3
        ini = f'[basis]\nkind = nodal-sem-gll\nK = {K}\nNqr = {K}\n'
        basis = get_basis(Config(ini))
        rng = np.random.default_rng(Ne)
        u = np.exp(-np.sum(cv ** 2, axis=0)) * (1 + 0.1 * rng.uniform(-1, 1, (K, Ne, N ** 3)))
        invjac = 2.0 / rng.uniform(0.5, 1.5, (Ne, 1))
        bcs, obc = [], []
        for side, (T, uy) in enumerate(((1.0, -0.1), (1.1, 0.2))):
            nl = -1.0 if side == 0 else 1.0
            if bc == 'dgfs-inlet':
                o = od.InletBC(cv, 1.0, T, (0.0, uy, 0.0), nl)
            else:
                o = od.WallDiffuseBC(cv, cw, T, (0.0, uy, 0.0), nl)
            obc.append(o)
            bcs.append((bc, o.f0, 0.0))
        dg = DGOperator(basis, invjac, c0, cw, bcs)
        ud = torch.tensor(u, device='cuda')
        ux = torch.empty_like(ud)
        for _ in range(2):           # the wall kernel's counter resets itself
            dg.advect(ud, ux)
        ref = _advect(basis, invjac, cv[0], obc[0], obc[1], u)
        assert _rel(ux.cpu().numpy(), ref) < 1e-13, (N, Ne, K, bc)


def _wall_case(N, Ne, K, seed=0):
    from dgfs1d_gpu_b200.basis import get_basis
    from dgfs1d_gpu_b200.config import Config
    from dgfs1d_gpu_b200.dg import DGOperator
    L = 5.0
    c0 = np.linspace(-L + L / N, L - L / N, N)
    c2 = sum(x ** 2 for x in np.meshgrid(c0, c0, c0, indexing='ij')).ravel()
    basis = get_basis(Config(f'[basis]\nkind = nodal-sem-gll\nK = {K}\nNqr = {K}\n'))
    rng = np.random.default_rng(seed)
    u = np.exp(-c2) * (1 + 0.1 * rng.uniform(-1, 1, (K, Ne, N ** 3)))
    bc = ('dgfs-wall-diffuse', np.exp(-c2) / np.pi ** 1.5, 0.0)
    dg = DGOperator(basis, np.full(Ne, 2.0 * Ne), c0, (2 * L / N) ** 3, [bc, bc])
    return dg, torch.tensor(u, device='cuda')


def test_wall_density_after_overlapping_calls():
    """Calls that overlap on one handle (two streams, beside a kernel that makes
    their CTAs trickle in) have undefined wall densities; the ordered calls after
    them have their own."""
    dg, u = _wall_case(32, 2, 3)
    u3, ux, ref = 3.0 * u, torch.empty_like(u), torch.empty_like(u)
    dg.advect(u3, ref)
    nden = dg.wall_density()
    load, first, second = [torch.cuda.Stream() for _ in range(3)]
    junk = [torch.empty_like(u) for _ in range(2)]
    big = torch.ones(1 << 27, device='cuda')
    torch.cuda.synchronize()

    def busy():
        with torch.cuda.stream(load):
            for _ in range(3):
                big.sin_()
    for i in range(100):
        busy()
        for _ in range(3):
            dg.advect(u, junk[0], stream=first)
            dg.advect(u, junk[1], stream=second)
        torch.cuda.synchronize()
        busy()
        dg.advect(u3, ux)
        torch.cuda.synchronize()
        assert np.array_equal(dg.wall_density(), nden), i
        assert torch.equal(ux, ref), i


def _advect(basis, invjac, cx, bcl, bcr, u):
    """Strong-form nodal DG advection with upwind faces, straight from the
    operators."""
    K, Ne, Nv = u.shape
    tr = np.einsum('qk,kev->qev', basis.faceOp, u)
    uL = np.concatenate([tr[0, :1], tr[-1]])
    uR = np.concatenate([tr[0], tr[-1, -1:]])
    bcl.update(uL[0])
    uL[0] = bcl.apply(uL[0])
    bcr.update(uR[-1])
    uR[-1] = bcr.apply(uR[-1])
    ac = 0.5 * np.abs(cx)
    jL = ac * (uL - uR) + 0.5 * cx * (uR - uL)
    jR = ac * (uL - uR) + 0.5 * cx * (uL - uR)
    ux = -cx * np.einsum('km,mev->kev', basis.derivOp, u)
    ux += -jL[1:][None] * basis.gRD[:, None, None] + jR[:-1][None] * basis.gLD[:, None, None]
    return ux * np.reshape(invjac, (1, Ne, 1))


def test_surrogate_gradients_over_sample_chunks():
    """Nine samples at N=16: the spectral backward passes them in chunks of
    eight; both forward routes (fused, per-axis passes)."""
    from dgfs1d_gpu_b200.surrogate import FNOSurrogate, layout
    N, K, L, B = 16, 8, 5.0, 9
    f = _maxwellians(N, L, B, 5)
    Qt = np.random.default_rng(6).standard_normal((B, N ** 3)) * 1e-3
    net = FNOSurrogate(N, L, q_scale=0.05, max_batch=B, seed=4)
    ref = ofno.FNO(N, K, L, 0.05, net.params(), emulate_bf16=True)
    out, cache = ref.forward(f)
    _, dout = ref.loss(out, Qt, cache['qs'])
    gr = ref.backward(dout, cache)
    fd, qd = torch.tensor(f, device='cuda'), torch.tensor(Qt, device='cuda')
    for fused in (True, False):
        net.set_fused(fused)
        net.train_step(fd, qd, update=False)
        g = net.grads()
        assert net.device_error() == 0
        for name, sl in layout(K).items():
            if name != 'total':
                e = _rel(g[sl[0]:sl[0] + sl[1]], gr[sl[0]:sl[0] + sl[1]])
                assert e < 2e-2, (fused, name, e)   # BF16 activations
