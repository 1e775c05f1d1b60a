"""The edges of the launch rules: quartets whose primitive quartets are shared by several lane groups
(prim_split; single-block calls and short lists of contracted shells, where the split is widest), roots at
the end of the table, and J/K contractions of every ket size, against the CPU oracle or the plain path."""
import numpy as np
import pytest

from cintx_b200 import molecules as M

pytestmark = pytest.mark.gpu



def contracted(ls, nprims, seed):
    """Three atoms, each with one shell per (l, nprim)."""
    rng = M.SplitMix64(seed)
    coords = [[0.0, 0.0, 0.0], [0.9, -0.7, 1.1], [-1.3, 0.4, 0.6]]
    return M.build_molecule("contracted", coords, [[M.make_shell(rng, l, n) for l, n in zip(ls, nprims)] for _ in coords])


def agree(got, ref):
    d = np.abs(got - ref)
    assert np.all((d <= 1e-12) | (d <= 1e-10 * np.abs(ref))), d.max()


@pytest.mark.parametrize("sph", [True, False])
@pytest.mark.parametrize("nij,nkl", [(1, 17), (17, 1), (3, 7), (8, 8), (13, 17)])
def test_single_block_calls(sph, nij, nkl):
    import cintx_b200 as cx
    from oracle import Restatement
    for la, lb, lc, ld in [(0, 0, 0, 0), (1, 0, 0, 0), (2, 0, 1, 0), (1, 1, 1, 0), (2, 1, 1, 1), (3, 0, 2, 0), (2, 2, 2, 1)]:
        mol = contracted([la, lb, lc, ld], [nij, 1 if nij > 8 else nij, nkl, 1 if nkl > 8 else nkl], 5 + la)
        q = np.array([[0, 5, 10, 3]], dtype=np.int32)  # one shell of each kind, over the three atoms
        ref, _ = Restatement().int2e_batch(q, mol, sph=sph)
        f = cx.int2e_sph if sph else cx.int2e_cart
        agree(f(q[0], mol.atm, mol.bas, mol.env)[0], ref)


@pytest.mark.parametrize("sph", [True, False])
def test_lists_mix_split_and_whole_quartets(sph):
    """A list long enough that only its contracted quartets are split."""
    import cintx_b200 as cx
    import torch
    from oracle import Restatement
    mol = contracted([0, 0, 0, 1, 1, 2], [13, 1, 8, 3, 1, 1], 9)
    rng = np.random.default_rng(3)
    q = rng.integers(0, mol.nbas, size=(6000, 4)).astype(np.int32)
    with cx.Optimizer(mol.atm, mol.bas, mol.env) as opt:
        plan = cx.Plan.shells(opt, cx.INT2E, q, sph=sph)
        out = torch.full((plan.stats.nintegrals,), np.nan, dtype=torch.float64, device="cuda")
        plan.execute(out.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        plan.close()
    ref, _ = Restatement().int2e_batch(q, mol, sph=sph)
    agree(got, ref)


@pytest.mark.parametrize("nsh", [3, 4])
@pytest.mark.parametrize("sph", [True, False])
def test_derivatives_of_contracted_shells(nsh, sph):
    """One derivative block per call (its primitive quartets over all lane groups) equals the same
    block out of a list of 4000 (few or none of them split)."""
    import cintx_b200 as cx
    import torch
    mol = contracted([0, 0, 1, 1, 2, 3], [13, 7, 3, 1, 1, 1], 11)
    rng = np.random.default_rng(4)
    t = rng.integers(0, mol.nbas, size=(4000, nsh)).astype(np.int32)
    t[:6] = np.arange(6)[:, None] + np.array([0, 6, 12, 6])[:nsh]
    fam = cx.INT2E if nsh == 4 else cx.INT3C2E
    out = torch.full((cx.ip1_len(fam, t, mol.bas, sph),), np.nan, dtype=torch.float64, device="cuda")
    off = cx.ip1_eval(fam, t, mol.atm, mol.bas, mol.env, out.data_ptr(), sph)
    got = out.cpu().numpy()
    assert np.isfinite(got).all()
    f = {(4, True): cx.int2e_ip1_sph, (4, False): cx.int2e_ip1_cart, (3, True): cx.int3c2e_ip1_sph,
         (3, False): cx.int3c2e_ip1_cart}[nsh, sph]
    with cx.Optimizer(mol.atm, mol.bas, mol.env) as opt:  # screened as the list is
        for q in range(40):
            one, _ = f(t[q], mol.atm, mol.bas, mol.env, opt=opt)
            # equal up to the order of at most 169 x 169 primitive terms of either sign
            assert np.allclose(one, got[off[q]:off[q] + one.size], rtol=1e-9, atol=1e-11)


XMAX = {1: 40, 2: 52, 3: 60, 4: 64, 5: 72, 6: 76, 7: 84, 8: 92, 9: 100}  # end of each order's table


def two_centres(ls, x, shift=0.0):
    """Shells 0 and 1 on one point, 2 and 3 on another, all of exponent 0.7 (a_ij = a_kl = 1.4, rho = 0.7),
    so that the quartet's only x is the given one; shell 0's atom moved by `shift` along z."""
    r = float(np.sqrt(x / 0.7))
    co = [[0.0, 0.0, shift], [0.0, 0.0, 0.0], [0.6 * r, 0.48 * r, 0.64 * r]]
    return M.build_molecule("ends", co, [[M.ShellSpec(ls[0], [0.7], [1.0])], [M.ShellSpec(ls[1], [0.7], [1.0])],
                                         [M.ShellSpec(l, [0.7], [1.0]) for l in ls[2:]]])


@pytest.mark.parametrize("ls", [(0, 0, 0, 0), (1, 0, 1, 0), (2, 0, 2, 0), (2, 1, 2, 1), (2, 2, 2, 2), (3, 2, 3, 2),
                                (3, 3, 3, 3), (4, 3, 4, 3), (4, 4, 4, 4)])
def test_roots_at_the_end_of_the_table(ls):
    """Quartets whose x lies on, just below and just above the last table interval of their order (1..9)
    and the 2^-20 before it where the large-x form starts, in single calls and in each launch shape."""
    import cintx_b200 as cx
    import torch
    from oracle import Restatement
    xmax = XMAX[sum(ls) // 2 + 1]
    orc = Restatement()
    s = torch.cuda.current_stream().cuda_stream
    for eps in (-1e-3, -2.0 ** -20 / xmax, -1e-9, 0.0, 1e-15, 1e-9, 1e-3):
        mol = two_centres(ls, xmax * (1.0 + eps))
        q = np.array([[0, 1, 2, 3]], dtype=np.int32)
        ref, _ = orc.int2e_batch(q, mol, sph=True)
        got, _ = cx.int2e_sph(q[0], mol.atm, mol.bas, mol.env)
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max() + 1e-15, (ls, eps)
        if sum(ls) not in (10, 12):  # (32|32), (33|33): sliced and split-transfer shapes exist
            continue
        with cx.Optimizer(mol.atm, mol.bas, mol.env) as opt:
            plan = cx.Plan.shells(opt, cx.INT2E, q)
            out = torch.empty(plan.stats.nintegrals, dtype=torch.float64, device="cuda")
            for v in range(12):
                plan.set_shape(v)
                plan.execute(out.data_ptr(), stream=s)
                d = np.abs(out.cpu().numpy() - ref).max()
                assert d <= 1e-12 * np.abs(ref).max() + 1e-15, (ls, eps, v)
            plan.close()


@pytest.mark.parametrize("ls", [(0, 0, 0, 0), (1, 0, 1, 0), (2, 1, 1, 1), (2, 1, 2, 2), (3, 2, 2, 2), (3, 3, 3, 3)])
def test_derivative_roots_at_the_end_of_the_table(ls):
    """First derivatives on both sides of the table's end of their order (one angular momentum more than
    the block's): minus the block's derivative by the shell's centre, from the oracle by differences."""
    import cintx_b200 as cx
    from oracle import Restatement
    xmax = XMAX[(sum(ls) + 1) // 2 + 1]
    q = np.array([[0, 1, 2, 3]], dtype=np.int32)
    orc = Restatement()
    h = 1e-2
    for eps in (-1e-3, -2.0 ** -20 / xmax, -1e-9, 0.0, 1e-9, 1e-3):
        x = xmax * (1.0 + eps)
        f = {k: orc.int2e_batch(q, two_centres(ls, x, k * h), sph=True)[0] for k in (-3, -2, -1, 1, 2, 3)}
        ref = -(45 * (f[1] - f[-1]) - 9 * (f[2] - f[-2]) + (f[3] - f[-3])) / (60 * h)
        mol = two_centres(ls, x)
        got, _ = cx.int2e_ip1_sph(q[0], mol.atm, mol.bas, mol.env)
        dz = got.reshape(3, -1)[2]
        # sixth-order differences: h^6 / 140 of the seventh derivative (up to some 10^5 in units of a^(7/2)
        # for f shells), and 1e-14 / h of rounding; a root out of a wrong interval is off by its whole value
        assert np.abs(dz - ref).max() <= 1e-7 * max(np.abs(ref).max(), np.abs(f[1]).max()), (ls, eps)


@pytest.mark.parametrize("sph", [True, False])
def test_lists_of_generally_contracted_shells_in_any_order(sph):
    """Every tuple of eight shells of one to two contractions: the blocks of a class come in all index
    orders, with extents that count the contractions."""
    import os

    import cintx_b200 as cx
    import torch
    from conftest import ROOT
    from oracle import Restatement
    g = np.load(os.path.join(ROOT, "tests", "golden", "libcint_ctr2.npz"))
    mol = M.Molecule("ctr2", g["atm"], g["bas"], g["env"], np.zeros((2, 3)))
    q = np.stack(np.meshgrid(*[np.arange(mol.nbas)] * 4, indexing="ij"), axis=-1).reshape(-1, 4).astype(np.int32)
    with cx.Optimizer(mol.atm, mol.bas, mol.env) as opt:
        plan = cx.Plan.shells(opt, cx.INT2E, q, sph=sph)
        out = torch.full((plan.stats.nintegrals,), np.nan, dtype=torch.float64, device="cuda")
        plan.execute(out.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
        got = out.cpu().numpy()
        plan.close()
    ref, _ = Restatement().int2e_batch(q, mol, sph=sph)
    agree(got, ref)


@pytest.mark.parametrize("sph", [True, False])
def test_jk_of_shells_up_to_g(sph):
    """J and K over every ket extent the contraction has a kernel for (spherical 1..9; cartesian up to
    10, and 15 in the general kernel) against einsum over the sweep's own s1 tensor."""
    import cintx_b200 as cx
    import torch
    mol = contracted([0, 1, 2, 3, 4], [2, 1, 1, 1, 1], 13)
    l = mol.bas[:, 1].astype(int)
    nao = int((2 * l + 1 if sph else (l + 1) * (l + 2) // 2).sum())
    g = torch.Generator(device="cuda").manual_seed(3)
    dm = torch.randn(nao, nao, generator=g, device="cuda", dtype=torch.float64)
    dm = dm + dm.T
    with cx.Optimizer(mol.atm, mol.bas, mol.env) as opt:
        plan = cx.Plan.screened(opt, 1e-14, sph=sph)
        eri = torch.full((nao ** 4,), np.nan, dtype=torch.float64, device="cuda")
        s = torch.cuda.current_stream().cuda_stream
        plan.execute_ao(eri.data_ptr(), eri.numel(), 1, s)
        vj, vk, j2, k2 = (torch.empty(nao, nao, dtype=torch.float64, device="cuda") for _ in range(4))
        plan.jk(dm.data_ptr(), nao, vj.data_ptr(), vk.data_ptr(), s)
        plan.jk(dm.data_ptr(), nao, j2.data_ptr(), 0, s)
        plan.jk(dm.data_ptr(), nao, 0, k2.data_ptr(), s)
        torch.cuda.synchronize()
        plan.close()
    eri = eri.reshape(nao, nao, nao, nao)
    assert torch.isfinite(eri).all()
    for got, ref in ((vj, torch.einsum("pqrs,rs->pq", eri, dm)), (vk, torch.einsum("pqrs,qs->pr", eri, dm))):
        # nao^2 products a sum; eps times their absolute sum bounds a difference in the order of addition
        assert (got - ref).abs().max() <= 1e-15 * nao ** 2 * float(eri.abs().max() * dm.abs().max())
    assert (j2 - vj).abs().max() <= 1e-11 * vj.abs().max() and (k2 - vk).abs().max() <= 1e-11 * vk.abs().max()


def test_forked_execution_from_two_threads_and_under_capture():
    """One explicit plan run by two host threads on streams of their own, and captured into a graph by
    the caller (where it stays on the captured stream), gives what a single run gives."""
    import threading

    import cintx_b200 as cx
    import torch
    mol = contracted([0, 0, 1, 1, 2], [8, 1, 3, 1, 1], 15)
    i, j = np.tril_indices(mol.nbas)
    a, b = np.tril_indices(i.size)
    q = np.stack([i[a], j[a], i[b], j[b]], axis=1).astype(np.int32)
    with cx.Optimizer(mol.atm, mol.bas, mol.env) as opt:
        plan = cx.Plan.shells(opt, cx.INT2E, q)
        n = plan.stats.nintegrals
        ref = torch.zeros(n, dtype=torch.float64, device="cuda")
        plan.execute(ref.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        bad, outs = [], [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(2)]

        def work(k):
            try:
                s = torch.cuda.Stream()
                with torch.cuda.stream(s):
                    for _ in range(20):
                        outs[k].zero_()
                        plan.execute(outs[k].data_ptr(), stream=s.cuda_stream)
                        got = outs[k].clone()
                        s.synchronize()
                        if not torch.equal(got, ref):
                            bad.append(k)
            except Exception as e:  # noqa: BLE001
                bad.append(e)

        th = [threading.Thread(target=work, args=(k,)) for k in range(2)]
        for t in th:
            t.start()
        for t in th:
            t.join()
        assert not bad
        out = torch.zeros(n, dtype=torch.float64, device="cuda")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            plan.execute(out.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, ref)
        del graph
        plan.close()


@pytest.mark.parametrize("sph", [True, False])
def test_jk_from_two_threads(sph):
    """Two host threads build J and K on plans of their own, streams of their own.  The kets of the f and
    g shells take shared memory that differs from bra to bra under one kernel ((gf|gf) and (gg|gf), or
    cartesian (fd|fd) and (ff|fd)), so a launch that set the kernel's limit to its own size would have
    the other thread's larger one refused."""
    import threading

    import cintx_b200 as cx
    import torch
    mol = contracted([3, 4] if sph else [0, 2, 3], [1, 1, 1], 17)
    l = mol.bas[:, 1].astype(int)
    nao = int((2 * l + 1 if sph else (l + 1) * (l + 2) // 2).sum())
    g = torch.Generator(device="cuda").manual_seed(5)
    dm = torch.randn(nao, nao, generator=g, device="cuda", dtype=torch.float64)
    dm = dm + dm.T
    torch.cuda.synchronize()
    bad, res = [], [None, None]

    def work(k):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s), cx.Optimizer(mol.atm, mol.bas, mol.env) as opt:
                plan = cx.Plan.screened(opt, 1e-14, sph=sph)
                vj, vk = (torch.empty(nao, nao, dtype=torch.float64, device="cuda") for _ in range(2))
                for _ in range(300):
                    plan.jk(dm.data_ptr(), nao, vj.data_ptr(), vk.data_ptr(), s.cuda_stream)
                s.synchronize()
                res[k] = (vj, vk)
                plan.close()
        except Exception as e:  # noqa: BLE001
            bad.append(e)

    th = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad, bad
    for a, b in zip(*res):  # the atomic adds of a sum come in any order
        assert (a - b).abs().max() <= 1e-12 * a.abs().max()


@pytest.mark.parametrize("ls", [(2, 1, 1, 1), (2, 0, 2, 0), (3, 2, 2, 1)])
def test_set_shape_runs_the_shape_on_split_quartets(ls):
    """Two contracted quartets, which a plan of their own shares over lane groups, and the same two
    repeated 6000 times, which no rule splits: in each forced shape both plans run the same kernel on one
    group per quartet, so their blocks agree to the last bit, and both report the shape's lanes."""
    import cintx_b200 as cx
    import torch
    mol = contracted(list(ls), [3, 3, 3, 3], 21)
    q = np.array([[0, 5, 10, 3], [4, 9, 2, 7]], dtype=np.int32)
    s = torch.cuda.current_stream().cuda_stream
    with cx.Optimizer(mol.atm, mol.bas, mol.env) as opt:
        few, many = cx.Plan.shells(opt, cx.INT2E, q), cx.Plan.shells(opt, cx.INT2E, np.tile(q, (6000, 1)))
        n = few.stats.nintegrals
        a = torch.empty(n, dtype=torch.float64, device="cuda")
        b = torch.empty(many.stats.nintegrals, dtype=torch.float64, device="cuda")
        split_lanes = few.segment_lanes(0)
        few.execute(a.data_ptr(), stream=s)
        split = a.clone()
        for v in range(12):
            few.set_shape(v), many.set_shape(v)
            assert few.set_shape(v) == 0  # nothing left to change
            lanes = few.segment_lanes(0)
            assert set(lanes) == set(many.segment_lanes(0)) and (v or (lanes < split_lanes).all())
            few.execute(a.data_ptr(), stream=s)
            many.execute(b.data_ptr(), stream=s)
            assert torch.equal(a, b[:n]), v
            # at most 81 terms of 1e-16 of the block's size each
            assert (a - split).abs().max() <= 1e-13 * split.abs().max()
        few.close(), many.close()


def test_tuning_a_small_molecule_leaves_larger_ones_their_shapes():
    """A plan whose quartets are all split has nothing to tune: it adds no choice for the process, counts
    as tuned itself, and a larger plan that picks up the process's choices afterwards runs the shapes it
    would have run before."""
    import cintx_b200 as cx
    import torch
    mol = contracted([3, 1, 3, 1], [3, 3, 3, 3], 23)
    q = np.array([[0, 5, 10, 3], [4, 9, 2, 7]], dtype=np.int32)
    s = torch.cuda.current_stream().cuda_stream
    with cx.Optimizer(mol.atm, mol.bas, mol.env) as opt:
        few, many = cx.Plan.shells(opt, cx.INT2E, q), cx.Plan.shells(opt, cx.INT2E, np.tile(q, (6000, 1)))
        buf = torch.empty(many.stats.nintegrals, dtype=torch.float64, device="cuda")
        many.use_tuned_shapes()  # of tests before this one
        lanes, recs, split = many.segment_lanes(0), cx.tuned_shapes(), few.segment_lanes(0)
        few.autotune(buf.data_ptr(), chunk=-1, stream=s, reps=1)
        assert cx.tuned_shapes() == recs
        assert few.use_tuned_shapes() == len(split) and np.array_equal(few.segment_lanes(0), split)
        many.use_tuned_shapes()
        assert np.array_equal(many.segment_lanes(0), lanes)
        few.set_shape(4)
        few.autotune(buf.data_ptr(), chunk=0, stream=s, reps=1)
        assert np.array_equal(few.segment_lanes(0), split)  # tuning ends a forced shape
        few.close(), many.close()


def test_work_behind_a_held_stream_holds_up_no_other():
    """A list of many classes queued behind a long kernel on one stream, then the same and a plain copy on
    others: they are done while the first is still held up."""
    import cintx_b200 as cx
    import torch
    mol = contracted([0, 0, 1, 1, 2], [8, 1, 3, 1, 1], 25)
    i, j = np.tril_indices(mol.nbas)
    a, b = np.tril_indices(i.size)
    q = np.stack([i[a], j[a], i[b], j[b]], axis=1).astype(np.int32)
    with cx.Optimizer(mol.atm, mol.bas, mol.env) as opt:
        plan = cx.Plan.shells(opt, cx.INT2E, q)
        streams = [torch.cuda.Stream() for _ in range(2)]
        outs = [torch.zeros(plan.stats.nintegrals, dtype=torch.float64, device="cuda") for _ in range(2)]
        torch.cuda.synchronize()
        for s, o in zip(streams, outs):
            plan.execute(o.data_ptr(), stream=s.cuda_stream)
        torch.cuda.synchronize()
        ref = outs[0].clone()
        torch.cuda.synchronize()
        with torch.cuda.stream(streams[0]):
            torch.cuda._sleep(1_000_000_000)  # cycles: half a second
            held = torch.cuda.Event()
            held.record()
        for s, o in zip(streams, outs):
            plan.execute(o.data_ptr(), stream=s.cuda_stream)
        rest = [torch.cuda.Stream() for _ in range(8)]  # as many as there are hardware queues
        for s in rest:
            with torch.cuda.stream(s):
                ref.clone()
        for s in streams[1:] + rest:
            s.synchronize()
        assert not held.query()
        torch.cuda.synchronize()
        assert torch.equal(outs[0], ref) and torch.equal(outs[1], ref)
        plan.close()


@pytest.mark.parametrize("sph", [True, False])
def test_j_of_an_infinite_density_element(sph):
    """An infinite density element makes every element of J infinite that it reaches by a nonzero
    integral, not NaN: lanes that pad a group or a warp add nothing."""
    import cintx_b200 as cx
    import torch
    mol = contracted([0, 1, 2, 3], [2, 1, 1, 1], 27)
    l = mol.bas[:, 1].astype(int)
    nao = int((2 * l + 1 if sph else (l + 1) * (l + 2) // 2).sum())
    s = torch.cuda.current_stream().cuda_stream
    with cx.Optimizer(mol.atm, mol.bas, mol.env) as opt:
        plan = cx.Plan.screened(opt, 0.0, sph=sph)
        eri = torch.empty(nao ** 4, dtype=torch.float64, device="cuda")
        plan.execute_ao(eri.data_ptr(), eri.numel(), 1, s)
        eri = eri.reshape(nao, nao, nao, nao)
        vj = torch.empty(nao, nao, dtype=torch.float64, device="cuda")
        n = 0
        for a in range(nao):
            b = (7 * a) % nao
            dm = torch.ones(nao, nao, dtype=torch.float64, device="cuda")
            dm[a, b] = dm[b, a] = float("inf")
            plan.jk(dm.data_ptr(), nao, vj.data_ptr(), 0, s)
            reached = eri[:, :, a, b].abs() > 1e-10  # zeros by symmetry are of either sign, or 0
            assert vj[reached].isinf().all(), (a, b)
            n += int(reached.sum())
        assert n > nao
        plan.close()
