"""The forms a kernel takes by size, at the sizes where one can go wrong: tile
remainders, the smallest and largest lattice of each form.  FP64 kernels with
another order of accumulation than the oracle's: 1e-13 of the largest entry."""
import numpy as np
import pytest

from oracle import oracle as O
from qex_b200 import fields as F
from qex_b200 import md as MD
from qex_b200 import smear as SM
from qex_b200 import stag as S

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


# half sweeps: 4^4 (128 sites a parity), 720 = 22 1/2 sets of 32 sites, 19208 (fat
# +Naik: still spread over warps) and 23520 (no longer; 91 7/8 sets of 256), 40960
# (more of them than SMs), 65536 and 69632
@pytest.mark.parametrize("dims,naik", [((4, 4, 4, 4), 0), ((4, 6, 6, 10), 0), ((4, 6, 6, 10), 1),
                                       ((14, 14, 14, 14), 1), ((12, 14, 14, 20), 1), ((16, 16, 16, 20), 1),
                                       ((16, 16, 16, 32), 0), ((16, 16, 16, 34), 0)])
def test_half_sweep_forms(cuda, dims, naik):
    g = F.fat_naik_links(dims, 3) if naik else F.naive_links(dims, 0.3, 3)
    V = F.volume(dims)
    o, s = O.Oracle(dims, g), S.Staggered(S.Layout(dims), S.to_device_links(g))
    x, r0 = F.gaussian_vector(V, 4), F.gaussian_vector(V, 5)
    for par in (0, 1):
        r, ro = S.to_device_vector(r0), r0.copy()
        s.stagD2(par, r, S.to_device_vector(x), 0.3, 0.7)
        o.stagD2(par, ro, x, 0.3, 0.7)
        assert rel(S.to_host_vector(r), ro) < 1e-13
    r, ro = S.to_device_vector(np.zeros_like(x)), o.vec()
    s.stagD2ee(r, S.to_device_vector(x), 0.01)
    o.stagD2ee(ro, x, 0.01)
    assert rel(S.to_host_vector(r), ro) < 1e-13


# smearing sweeps: blocks of 64 half sites of both parities; 720 half sites
# are 11 1/4 of them and 22 1/2 warps (tolerances as for the other shapes)
@pytest.mark.parametrize("coef", [[0.3, 0.2, -0.1, 0.05, 0.07], [0.4, 0.2, 0.0, 0.0, 0.0], [0.3, 0.2, -0.1, 0.0, 0.0],
                                  [0.3, 0.0, 0.0, 0.05, 0.0], [0.3, 0.2, 0.0, 0.0, 0.07], [0.5, 0.0, 0.0, 0.0, 0.0]])
def test_smearing_sweep_remainders(cuda, coef):
    dims = (4, 6, 6, 10)
    V = F.volume(dims)
    g = O.apply_phases(dims, F.gauge_warm(dims, 0.5, 6))
    rng = np.random.default_rng(7)
    ch, d0 = (rng.standard_normal((4, V, 3, 3)) + 1j * rng.standard_normal((4, V, 3, 3)) for _ in range(2))
    sm, c = SM.Smear(S.Layout(dims)), SM.Fat7lCoefs(*coef)
    fl = np.empty_like(g)
    sm.makeImpLinks(fl, g, c)
    assert rel(fl, O.fat7(dims, coef, g)) < 1e-12
    d = d0.copy()
    sm.fat7Deriv(d, g, ch, c)
    assert rel(d, d0 + O.fat7_deriv(dims, coef, g, ch)[0]) < 1e-12


# multi-shift solves: 1 (one vector), 2 and 3 (one and two pairs, an odd one
# with a zero partner), 5 and 8 right-hand sides, on 720 = 22 1/2 sets of sites
@pytest.mark.parametrize("nrhs,naik", [(1, 1), (2, 1), (3, 1), (3, 0), (5, 1), (8, 0)])
def test_shifted_systems_by_right_hand_sides(cuda, nrhs, naik):
    dims, m, sigmas = (4, 6, 6, 10), 0.2, [0.3, 0.0, 1.0]
    g = F.fat_naik_links(dims, 3) if naik else F.naive_links(dims, 0.3, 3)
    V = F.volume(dims)
    o, s = O.Oracle(dims, g), S.Staggered(S.Layout(dims), S.to_device_links(g))
    bs = [F.even_source(dims, 40 + j) for j in range(nrhs)]
    ys = [[S.to_device_vector(np.zeros_like(b)) for _ in sigmas] for b in bs]
    sp = S.SolverParams(r2req=1e-20, sloppySolve=S.L.SLOPPY_SINGLE)
    r2 = s.cgm_ee(m, sigmas, [S.to_device_vector(b) for b in bs], ys, sp)
    assert sp.status == S.L.OK and (r2 <= 1e-20).all()
    for b, row in zip(bs, ys):
        for sg, y in zip(sigmas, row):
            y, ay = S.to_host_vector(y), o.vec()
            o.stagD2ee(ay, y, m * m + 0.25 * sg)
            assert np.linalg.norm((ay - b)[: V // 2]) <= 1.01e-10 * np.linalg.norm(b)
            assert not np.any(y[V // 2:])


# a solve ends where it is told to, whatever was queued behind it: after 1, 2,
# 7 (one more than are queued at a time) and 40 iterations
@pytest.mark.parametrize("sloppy", [0, 1, 2])
@pytest.mark.parametrize("maxits", [1, 2, 7, 40])
def test_solve_stops_at_maxits(cuda, sloppy, maxits):
    dims = (4, 6, 6, 10)
    s = S.Staggered(S.Layout(dims), S.to_device_links(F.fat_naik_links(dims, 3)))
    b = S.to_device_vector(F.even_source(dims, 4))
    for _ in range(2):
        sp = S.SolverParams(r2req=1e-24, maxits=maxits, sloppySolve=sloppy)
        s.solveEE(cuda.zeros_like(b), b, 0.01, sp)
        assert sp.iterations == maxits and sp.status == S.L.NOT_CONVERGED
    sp = S.SolverParams(r2req=1e-20, sloppySolve=sloppy)
    x = cuda.zeros_like(b)
    s.solveEE(x, b, 0.3, sp)
    assert sp.status == S.L.OK and sp.r2 <= 1e-20
    s.solveEE(x, cuda.zeros_like(b), 0.3, sp)  # no source: no iterations
    assert sp.iterations == 0 and not bool(x.any())


# the force with rectangles in two sweeps: 720 half sites are 11 1/4 blocks
def test_rectangle_force_remainders(cuda):
    dims = (4, 6, 6, 10)
    lay, u = S.Layout(dims), F.gauge_warm(dims, 0.5, 6)
    ud = S.to_device_links(u)
    f = cuda.empty_like(ud)
    act = MD.GaugeAction(lay, 5.6, -1.0 / 12.0)
    act.force(ud, f)
    assert rel(S.to_host_links(f), O.gauge_force(dims, u, act.c.plaq, act.c.rect)) < 1e-12


# and through more than one slab of time slices: 48 slices of 32^3 take two,
# the first of them with its lower neighbours beyond the periodic boundary.
# The links repeat after 24 slices, which are one slab by themselves, so the
# force must repeat too, bit for bit.
def test_rectangle_force_slabs(cuda):
    torch = cuda
    half, full = (32, 32, 32, 24), (32, 32, 32, 48)
    gen = torch.Generator(device="cuda").manual_seed(3)
    u = torch.view_as_complex(torch.randn((4, 3, 3, F.volume(half), 2), dtype=torch.float64, device="cuda",
                                          generator=gen))
    x = F.coords(full)
    x[:, 3] %= 24
    place = torch.from_numpy(F.index_of(half, x)).to("cuda")
    one, two = MD.GaugeAction(S.Layout(half), 5.6, -0.331), MD.GaugeAction(S.Layout(full), 5.6, -0.331)
    f1 = torch.empty_like(u)
    one.force(u, f1)
    u2 = u.index_select(3, place)
    f2 = torch.empty_like(u2)
    two.force(u2, f2)
    assert torch.equal(f2, f1.index_select(3, place))


# batches: one problem, an odd set count (720 even sites are 22 1/2 sets of 32),
# and 70 problems (more than the norms read back at a time)
@pytest.mark.parametrize("shapes", [[(4, 4, 4, 4)], [(4, 6, 6, 10), (4, 4, 4, 4), (6, 4, 4, 6)], [(4, 4, 4, 4)] * 70])
def test_batch_partitions(cuda, shapes):
    ops, bs, ms, gs = [], [], [], []
    for j, dims in enumerate(shapes):
        gs.append(F.naive_links(dims, 0.3, 3 + j % 5))
        ops.append(S.Staggered(S.Layout(dims), S.to_device_links(gs[-1])))
        bs.append(F.even_source(dims, 40 + j))
        ms.append(0.1 + 0.02 * (j % 7))
    xs = [S.to_device_vector(np.zeros_like(b)) for b in bs]
    out = S.solve_batched(ops, xs, [S.to_device_vector(b) for b in bs], ms, S.SolverParams(r2req=1e-20))
    assert (out["r2"] <= 1e-20).all()
    for dims, g, m, b, x in zip(shapes, gs, ms, bs, xs):
        o = O.Oracle(dims, g)
        x, ax = S.to_host_vector(x), o.vec()
        o.stagD2ee(ax, x, m * m)
        assert np.linalg.norm((ax - b)[: F.volume(dims) // 2]) <= 1.01e-10 * np.linalg.norm(b)


# both parities in one launch, spread over warps (up to 8192 even sites) and not:
# the same bits as one parity after the other
@pytest.mark.parametrize("dims,naik", [((4, 6, 6, 10), 0), ((4, 6, 6, 10), 1), ((8, 8, 8, 32), 1), ((8, 8, 8, 34), 1),
                                       ((16, 16, 16, 34), 0), ((24, 24, 24, 24), 1)])
def test_both_parities_in_one_launch(cuda, dims, naik):
    torch, V = cuda, F.volume(dims)
    gen = torch.Generator(device="cuda").manual_seed(3)

    def field(*shape):
        return torch.view_as_complex(torch.randn(shape + (2,), dtype=torch.float64, device="cuda", generator=gen))

    s = S.Staggered(S.Layout(dims), field(8 if naik else 4, 3, 3, V))
    x, r0 = field(3, V), field(3, V)
    for m, sc, a in ((0.1, 1.0, 0.0), (0.0, -1.0, 0.0), (0.2, 0.5, 0.7)):
        one, two = r0.clone(), r0.clone()
        s.stagD(S.L.ALL, one, x, m, sc, a)
        s.stagD(S.L.EVEN, two, x, m, sc, a)
        s.stagD(S.L.ODD, two, x, m, sc, a)
        assert torch.equal(one, two)
    one, two = x.clone(), x.clone()  # in place: odd sites see the new even ones
    s.D(one, one, 0.1)
    s.stagD(S.L.EVEN, two, two, 0.1)
    s.stagD(S.L.ODD, two, two, 0.1)
    assert torch.equal(one, two)


# several vectors at once: links through registers and, from 262144 sites times
# vectors on, through a ring in shared memory.  69120 sites a parity are 540
# sets of 128; 93600 are 731 1/4 of them and 1462 1/2 of 64.  One vector at a
# time sums the hops in another order: 1e-13 of the largest entry.
@pytest.mark.parametrize("dims,n", [((16, 16, 18, 30), 3), ((16, 16, 18, 30), 4), ((18, 20, 20, 26), 3),
                                    ((18, 20, 20, 26), 4), ((18, 20, 20, 26), 5), ((18, 20, 20, 26), 8)])
@pytest.mark.parametrize("naik", [0, 1])
def test_several_vectors_forms(cuda, dims, n, naik):
    torch, V = cuda, F.volume(dims)
    gen = torch.Generator(device="cuda").manual_seed(3)

    def field(*shape):
        return torch.view_as_complex(torch.randn(shape + (2,), dtype=torch.float64, device="cuda", generator=gen))

    s = S.Staggered(S.Layout(dims), field(8 if naik else 4, 3, 3, V))
    xs, r0 = [field(3, V) for _ in range(n)], field(3, V)
    for par in (0, 1):
        rs = [r0.clone() for _ in xs]
        s.stagDN(par, rs, xs, 0.3)
        for r, x in zip(rs, xs):
            one = r0.clone()
            s.stagD2(par, one, x, 0.0, 0.3)
            assert float((r - one).abs().max() / one.abs().max()) < 1e-13


# FP64 solves with the fused iteration (19208 even sites; 81648, 319 sets of 256)
# and without it (32768 and 40960)
@pytest.mark.parametrize("dims", [(14, 14, 14, 14), (16, 16, 16, 16), (16, 16, 16, 20), (18, 18, 18, 28)])
@pytest.mark.parametrize("naik", [0, 1])
def test_solve_forms(cuda, dims, naik):
    g = F.fat_naik_links(dims, 3) if naik else F.naive_links(dims, 0.3, 3)
    o, s = O.Oracle(dims, g), S.Staggered(S.Layout(dims), S.to_device_links(g))
    b = F.even_source(dims, 4)
    x, sp = S.to_device_vector(np.zeros_like(b)), S.SolverParams(r2req=1e-20)
    s.solveEE(x, S.to_device_vector(b), 0.5, sp)
    assert sp.status == S.L.OK and sp.r2 <= 1e-20
    x, ax = S.to_host_vector(x), o.vec()
    o.stagD2ee(ax, x, 0.25)
    assert np.linalg.norm((ax - b)[: F.volume(dims) // 2]) <= 1.01e-10 * np.linalg.norm(b)


# reduced-precision half sweeps by blocks on an SM: 36864 even sites are 144 sets
# of 256 (one block an SM), 40960 are 160 (two), 81648 are 318 15/16 (four)
@pytest.mark.parametrize("dims", [(16, 16, 16, 18), (16, 16, 16, 20), (18, 18, 18, 28)])
@pytest.mark.parametrize("sloppy", [1, 2])
@pytest.mark.parametrize("naik", [0, 1])
def test_reduced_precision_forms(cuda, dims, sloppy, naik):
    g = F.fat_naik_links(dims, 3) if naik else F.naive_links(dims, 0.3, 3)
    o, s = O.Oracle(dims, g), S.Staggered(S.Layout(dims), S.to_device_links(g))
    b = F.even_source(dims, 4)
    x, sp = S.to_device_vector(np.zeros_like(b)), S.SolverParams(r2req=1e-20, sloppySolve=sloppy)
    s.solveEE(x, S.to_device_vector(b), 0.5, sp)
    assert sp.status == S.L.OK and sp.r2 <= 1e-20
    x, ax = S.to_host_vector(x), o.vec()
    o.stagD2ee(ax, x, 0.25)
    assert np.linalg.norm((ax - b)[: F.volume(dims) // 2]) <= 1.01e-10 * np.linalg.norm(b)


# a batch whose large lattices make a block's chunk take in all 68 small ones:
# each problem ends as it does by itself, without a correction
@pytest.mark.parametrize("naik", [0, 1])
def test_batch_of_large_and_small_lattices(cuda, naik):
    links = F.fat_naik_links if naik else (lambda dims, seed: F.naive_links(dims, 0.3, seed))
    kinds = []
    for dims, n in (((16, 16, 16, 16), 60), ((4, 4, 4, 4), 68)):
        lay, g = S.Layout(dims), S.to_device_links(links(dims, 3))
        b = S.to_device_vector(F.even_source(dims, 4))
        kinds += [(lay, g, b)] * n
    ops = [S.Staggered(lay, g) for lay, g, _ in kinds]
    xs, sp = [cuda.zeros_like(b) for _, _, b in kinds], S.SolverParams(r2req=1e-20)
    out = S.solve_batched(ops, xs, [b for _, _, b in kinds], [0.3] * len(ops), sp)
    assert sp.status == S.L.OK and (out["r2"] <= 1e-20).all() and sp.outer_iterations == 0
    for j in (0, len(ops) - 1):
        one = S.SolverParams(r2req=1e-20)
        ops[j].solveEE(cuda.zeros_like(xs[j]), kinds[j][2], 0.3, one)
        same = range(60) if j == 0 else range(60, 128)
        assert all(abs(out["iterations"][i] - one.iterations) <= 1 for i in same)
        # two solutions to |r| <= 1e-10 |b|, and 4 m^2 = 0.36 below every eigenvalue
        far = 2e-10 * float(kinds[j][2].norm()) / 0.36
        assert all(float((xs[i] - xs[j]).norm()) <= far for i in same)


# separate handles from separate threads, on the default stream and on streams
# of their own: every solve ends as it does alone, bit for bit
@pytest.mark.parametrize("streams", [0, 1])
def test_solves_from_several_threads(cuda, streams):
    import threading
    dims = (4, 6, 6, 10)
    b = S.to_device_vector(F.even_source(dims, 4))
    lay, g = S.Layout(dims), S.to_device_links(F.fat_naik_links(dims, 3))

    def work(s, scale):
        out = []
        s.update_links(g * scale)
        for sloppy in (S.L.SLOPPY_NONE, S.L.SLOPPY_SINGLE, S.L.SLOPPY_HALF):
            x, sp = cuda.zeros_like(b), S.SolverParams(r2req=1e-20, sloppySolve=sloppy)
            s.solveEE(x, b, 0.1, sp)
            out += [x, sp.iterations]
        ys = [[cuda.zeros_like(b) for _ in range(2)] for _ in range(3)]
        sp = S.SolverParams(r2req=1e-20, sloppySolve=S.L.SLOPPY_SINGLE)
        out.append(s.cgm_ee(0.1, [0.0, 0.5], [b, 2.0 * b, b], ys, sp).tolist())
        return out + [y for row in ys for y in row] + [sp.iterations]

    scales = [1.0, 0.9, 1.1, 0.8]
    ops = [S.Staggered(lay, g) for _ in scales]
    alone = [work(s, c) for s, c in zip(ops, scales)]
    got, start = [[] for _ in scales], threading.Barrier(len(scales))

    def thread(i):
        with cuda.cuda.stream(cuda.cuda.Stream() if streams else cuda.cuda.default_stream()):
            S.L.load().qexstag_set_stream(cuda.cuda.current_stream().cuda_stream)
            start.wait()
            for _ in range(5):
                got[i].append(work(ops[i], scales[i]))
            cuda.cuda.current_stream().synchronize()

    cuda.cuda.synchronize()
    threads = [threading.Thread(target=thread, args=(i,)) for i in range(len(scales))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for one, runs in zip(alone, got):
        assert len(runs) == 5
        for run in runs:
            for u, v in zip(one, run):
                assert cuda.equal(u, v) if cuda.is_tensor(u) else u == v


# slabs keep within their 4 GiB on the shortest lattices too: on 72^3 x 4, whose
# four slices of half staples would take 5.2 GB, the force goes path by path, and
# agrees with the slabs of the same field with the short side third
def test_rectangle_force_scratch_of_few_slices(cuda):
    torch = cuda
    dims, turned = (72, 72, 72, 4), (72, 72, 4, 72)
    gen = torch.Generator(device="cuda").manual_seed(3)
    u = torch.view_as_complex(torch.randn((4, 3, 3, F.volume(dims), 2), dtype=torch.float64, device="cuda",
                                          generator=gen))
    lay, f = S.Layout(dims), torch.empty_like(u)
    act = MD.GaugeAction(lay, 5.6, -0.331)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    act.force(u, f)
    assert free - torch.cuda.mem_get_info()[0] <= (4 << 30) + (64 << 20)
    place = torch.from_numpy(F.index_of(dims, F.coords(turned)[:, [0, 1, 3, 2]])).to("cuda")
    u, f = (t[[0, 1, 3, 2]].index_select(3, place) for t in (u, f))
    ft = torch.empty_like(u)
    MD.GaugeAction(S.Layout(turned), 5.6, -0.331).force(u, ft)
    assert float((f - ft).abs().max() / ft.abs().max()) < 1e-12


# with the device nearly full: links are allocated in the place of the scratch
# (1.15 GB at 24^4) that a layout keeps from its last force, and a force that
# finds no room for its scratch goes path by path
def test_force_scratch_makes_way(cuda):
    torch, dims = cuda, (24, 24, 24, 24)
    gen = torch.Generator(device="cuda").manual_seed(3)
    u = torch.view_as_complex(torch.randn((8, 3, 3, F.volume(dims), 2), dtype=torch.float64, device="cuda",
                                          generator=gen))
    lay, f1, f2 = S.Layout(dims), torch.empty_like(u[:4]), torch.empty_like(u[:4])
    MD.GaugeAction(lay, 5.6, -0.331).force(u[:4], f1)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (300 << 20), dtype=torch.uint8, device="cuda")
    assert torch.cuda.mem_get_info()[0] < (320 << 20)
    ops = S.Staggered(lay, u)  # 382 MB of links and their copies in less precision
    MD.GaugeAction(S.Layout(dims), 5.6, -0.331).force(u[:4], f2)
    del fill, ops
    assert float((f1 - f2).abs().max() / f1.abs().max()) < 1e-12


# links that cannot be copied to less precision (all zero): the update says so,
# and nothing goes on with the copies of the links before them
def test_no_reduced_precision_after_a_failed_update(cuda):
    dims = (4, 6, 6, 10)
    g = S.to_device_links(F.fat_naik_links(dims, 3))
    s, b = S.Staggered(S.Layout(dims), g), S.to_device_vector(F.even_source(dims, 4))

    def shifted():
        ys = [[cuda.zeros_like(b)] for _ in range(2)]
        sp = S.SolverParams(r2req=1e-20, sloppySolve=S.L.SLOPPY_SINGLE)
        s.cgm_ee(0.3, [0.0], [b, 2.0 * b], ys, sp)
        return sp.status

    def half():
        s.solveEE(cuda.zeros_like(b), b, 0.3, S.SolverParams(r2req=1e-20, sloppySolve=S.L.SLOPPY_HALF))

    with pytest.raises(S.L.QexStagError):
        s.update_links(cuda.zeros_like(g))
    for call in (shifted, half, lambda: s.bench_schur(1, 1), lambda: s.bench_schur(2, 1)):
        with pytest.raises(S.L.QexStagError):
            call()
    s.update_links(g)
    assert shifted() == S.L.OK
    half()


# the same from 490000 sites times vectors on, where the ring takes any number of
# vectors above two: 171072 sites a parity are 1336 1/2 sets of 128 and 2673 of 64
@pytest.mark.parametrize("n", [3, 4, 5, 7])
@pytest.mark.parametrize("naik", [0, 1])
def test_several_vectors_on_large_lattices(cuda, n, naik):
    test_several_vectors_forms(cuda, (18, 22, 24, 36), n, naik)


# a chain rule without terms beyond the 3-staple takes no scratch for them: at
# most the 28 link fields that it has always held
@pytest.mark.parametrize("coef", [[0.5, 0.0, 0.0, 0.0, 0.0], [0.4, 0.2, 0.0, 0.0, 0.0]])
def test_chain_rule_scratch_of_simple_levels(cuda, coef):
    dims = (16, 16, 16, 16)
    u = cuda.zeros((4, 3, 3, F.volume(dims)), dtype=cuda.complex128, device="cuda")
    d, sm = cuda.zeros_like(u), SM.Smear(S.Layout(dims))
    cuda.cuda.synchronize()
    free = cuda.cuda.mem_get_info()[0]
    sm.fat7Deriv(d, u, u, SM.Fat7lCoefs(*coef))
    assert free - cuda.cuda.mem_get_info()[0] <= 28 * 144 * F.volume(dims) + (8 << 20)


# three right-hand sides of twelve shifts on 24^4 take 448 MB and, in two pairs,
# 552: with 500 MB left the odd one is solved by itself
def test_odd_right_hand_side_with_little_memory(cuda):
    torch, dims, sigmas = cuda, (24, 24, 24, 24), [0.2 * k for k in range(12)]
    V = F.volume(dims)
    gen = torch.Generator(device="cuda").manual_seed(3)

    def field(*shape):
        return torch.view_as_complex(torch.randn(shape + (2,), dtype=torch.float64, device="cuda", generator=gen))

    s, bs = S.Staggered(S.Layout(dims), 0.3 * field(8, 3, 3, V)), [field(3, V) for _ in range(3)]
    for b in bs:
        b[:, V // 2:] = 0
    ys = [[torch.zeros_like(b) for _ in sigmas] for b in bs]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (500 << 20), dtype=torch.uint8, device="cuda")
    sp = S.SolverParams(r2req=1e-20, sloppySolve=S.L.SLOPPY_SINGLE)
    r2 = s.cgm_ee(0.5, sigmas, bs, ys, sp)
    del fill
    assert sp.status == S.L.OK and (r2 <= 1e-20).all()
    for b, row in zip(bs, ys):
        for sg, y in zip(sigmas, row):
            ay = torch.zeros_like(b)
            s.stagD2ee(ay, y, 0.25 + 0.25 * sg)
            assert float((ay - b)[:, :V // 2].norm()) <= 1.01e-10 * float(b.norm())


# a thread whose first call of the library is in a graph that it captures
def test_first_call_of_a_thread_in_a_capture(cuda):
    import threading
    torch, dims = cuda, (4, 6, 6, 10)
    V = F.volume(dims)
    s = S.Staggered(S.Layout(dims), S.to_device_links(F.fat_naik_links(dims, 3)))
    x = S.to_device_vector(F.gaussian_vector(V, 4))
    want, got, graph = torch.empty_like(x), torch.zeros_like(x), torch.cuda.CUDAGraph()
    s.D(want, x, 0.1)
    torch.cuda.synchronize()
    done = []

    def capture():
        with torch.cuda.graph(graph):
            S.set_stream(torch.cuda.current_stream().cuda_stream)
            s.D(got, x, 0.1)
        done.append(True)

    t = threading.Thread(target=capture)
    t.start()
    t.join()
    assert done
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
