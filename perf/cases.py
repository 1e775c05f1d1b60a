"""The work this library is timed on: its public entry points over the sizes they are used at.

Each case is one call pattern of a user's program:

  call    int2e_sph / int2e_cart for one block through the libcint signature (host in, host out)
  batch   an explicit list of every 8-fold-unique quartet of a small molecule (Plan.shells)
  sweep   every Schwarz-surviving quartet of a molecule into device memory (Plan.screened, or the
          tuned form: Plan.screened_mixed, autotuned launch shapes, one CUDA graph)
  jk      the Coulomb and exchange matrices of a density over such a sweep (direct SCF)
  ao      the sweep as an AO-indexed tensor (s1, s4 or s8)
  df3c    the density-fitting sweep (ab|k) (Plan.screened_3c)
  metric  the density-fitting metric (k|l) over all auxiliary pairs (an explicit int2c2e plan)
  grad    first-derivative integrals of a whole small molecule (ip1_eval; 4 or 3 centres)

Molecules are the package's synthetic ones (molecules.random_molecule, with_aux; g shells as in
its mol20_g), at the density of its 40- and 120-atom configurations.  A case has one molecule; each
seed moves its atoms and scales its exponents a little, as the steps of a geometry optimisation and
of a basis optimisation do, so the surviving quartets of two seeds differ by some percent.
"""
import math

import numpy as np
import torch

import cintx_b200 as cx
from cintx_b200 import molecules as M

CUTOFF = 1e-12       # Schwarz cut-off of every screened plan
PRIM_BUDGET = 5e-11  # primitive-screening budget of the tuned form (the package's default)
ONE_CHUNK = 1 << 31  # doubles: every sweep case below fits one chunk, so its output comes back whole


def listed():
    return [
        # a libcint caller that keeps its loop: one contracted block per call, latency of the call
        {"name": "call_psss", "op": "call", "l": "1000", "sph": True},
        # the whole of a 3-atom molecule in one list: few quartets, up to 4096 primitive quartets each
        {"name": "batch_water", "op": "batch", "natm": 3, "basis": "spd", "sph": True},
        # high angular momentum: every quartet of four atoms that carry g shells
        {"name": "batch_g4", "op": "batch", "natm": 4, "basis": "g", "sph": True},
        # the 40-atom s/p/d configuration, tuned form: the package's mid-size benchmark
        {"name": "sweep_spd40_tuned", "op": "sweep", "natm": 40, "basis": "spd", "sph": True, "tuned": True},
        # a mid-size s/p/d/f molecule without tuning: what a first call gets
        {"name": "sweep_spdf24", "op": "sweep", "natm": 24, "basis": "spdf", "sph": True, "tuned": False},
        # cartesian output, an odd number of atoms
        {"name": "sweep_spd19_cart", "op": "sweep", "natm": 19, "basis": "spd", "sph": False, "tuned": False},
        # a Fock build of the 120-atom s/p/d/f configuration, tuned: the largest
        {"name": "jk_spdf120_tuned", "op": "jk", "natm": 120, "basis": "spdf", "sph": True, "tuned": True},
        # a Fock build of a small molecule, as each step of a geometry optimisation does some ten of
        {"name": "jk_spd12", "op": "jk", "natm": 12, "basis": "spd", "sph": True, "tuned": False},
        # the full AO tensor of a small molecule, for a caller that indexes it directly
        {"name": "ao_s1_spd9", "op": "ao", "natm": 9, "basis": "spd", "sph": True, "aosym": 1},
        # density fitting, 3-centre part
        {"name": "df3c_spdf40", "op": "df3c", "natm": 40, "basis": "spdf", "sph": True},
        # density fitting, metric of 120 atoms: 2.9 million tiny blocks
        {"name": "metric_120", "op": "metric", "natm": 120, "sph": True},
        # nuclear gradient of a small molecule: host lists in, derivative blocks on the device
        {"name": "grad_spdf4", "op": "grad", "natm": 4, "basis": "spdf", "sph": True, "centres": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["call", "batch", "sweep", "sweep", "jk", "ao", "df3c", "metric", "grad"])
    sph = rng.random() < 0.7
    if op == "call":
        return {"op": op, "l": "".join(rng.choice("0123") for _ in range(4)), "sph": sph}
    if op == "batch":
        basis = rng.choice(["spd", "spdf", "g"])
        return {"op": op, "natm": rng.randint(2, 6 if basis == "spd" else 4), "basis": basis, "sph": sph}
    if op == "sweep":
        basis = rng.choice(["spd", "spdf"])
        tuned = sph and rng.random() < 0.5
        return {"op": op, "natm": _log_int(rng, 5, 40 if basis == "spd" else 24), "basis": basis, "sph": sph,
                "tuned": tuned}
    if op == "jk":
        basis = rng.choice(["spd", "spdf"])
        return {"op": op, "natm": _log_int(rng, 5, 60), "basis": basis, "sph": True, "tuned": rng.random() < 0.5}
    if op == "ao":
        aosym = rng.choice([1, 4, 8])
        return {"op": op, "natm": rng.randint(3, {1: 10, 4: 14, 8: 18}[aosym]), "basis": "spd", "sph": sph,
                "aosym": aosym}
    if op == "df3c":
        return {"op": op, "natm": _log_int(rng, 6, 40), "basis": rng.choice(["spd", "spdf"]), "sph": sph}
    if op == "metric":
        return {"op": op, "natm": _log_int(rng, 4, 120), "sph": sph}
    return {"op": op, "natm": rng.randint(2, 4), "basis": rng.choice(["spd", "spdf"]), "sph": sph,
            "centres": rng.choice([3, 4])}


# ------------------------------------------------------------------------------ molecules

def _molecule(case, seed):
    """The case's molecule, its atoms moved by up to 0.05 bohr and its exponents scaled by up to 2%."""
    natm = 5 if case["op"] == "call" else case["natm"]  # five: two heavy atoms
    box = 4.3 * natm ** (1.0 / 3.0) + 1.0  # the density of the 40- and 120-atom configurations
    basis = case.get("basis", "spdf")
    base = 1000 + natm
    if basis == "g":
        rng = M.SplitMix64(base)
        coords = M._place_atoms(rng, natm, box, 1.4)
        mol = M.build_molecule("g", coords, [[M.make_shell(rng, l, n) for l, n in M.G_ATOM] for _ in range(natm)])
    else:
        mol = M.random_molecule(basis, base, natm, box, with_f=basis == "spdf")
    norb = mol.nbas
    if case["op"] in ("df3c", "metric") or case.get("centres") == 3:
        mol = M.with_aux(mol, base + 1)
    rng = np.random.default_rng(seed)
    mol.coords = mol.coords + rng.uniform(-0.05, 0.05, size=mol.coords.shape)
    for a in range(mol.natm):
        at = mol.atm[a, M.PTR_COORD]
        mol.env[at:at + 3] = mol.coords[a]
    for r in mol.bas:
        at = r[M.PTR_EXP]
        mol.env[at:at + r[M.NPRIM_OF]] *= 1.0 + rng.uniform(-0.02, 0.02)
    return mol, norb


def _unique_quartets(n):
    """Every 8-fold-unique (i, j, k, l): i >= j, k >= l, ij >= kl, in lexicographic order."""
    a, b = np.tril_indices(n)
    p, q = np.tril_indices(a.size)
    return np.stack([a[p], b[p], a[q], b[q]], axis=1).astype(np.int32)


def _tuples(case, mol, norb):
    op = case["op"]
    if op == "call":
        # (ab| on one heavy atom and |cd) on the other, of each angular momentum the most contracted
        # shell first: a block that no screening removes
        l, atom = mol.bas[:, M.ANG_OF], mol.bas[:, M.ATOM_OF]
        heavy = [a for a in range(mol.natm) if ((atom == a) & (l == 2)).any()]
        seen, out = {}, []
        for x, c in enumerate(case["l"]):
            ids = np.nonzero((l == int(c)) & (atom == heavy[x // 2]))[0]
            out.append(int(ids[seen.get((x // 2, c), 0) % ids.size]))
            seen[(x // 2, c)] = seen.get((x // 2, c), 0) + 1
        return np.asarray([out], dtype=np.int32)
    if op == "batch":
        return _unique_quartets(mol.nbas)
    if op == "metric":
        a, b = np.tril_indices(mol.nbas - norb)
        return np.stack([a + norb, b + norb], axis=1).astype(np.int32)
    if op == "grad":
        n = norb
        if case["centres"] == 3:
            i, j, k = np.meshgrid(np.arange(n), np.arange(n), np.arange(norb, mol.nbas), indexing="ij")
            return np.stack([i.ravel(), j.ravel(), k.ravel()], axis=1).astype(np.int32)
        a, b = np.tril_indices(n)
        ij = np.stack(np.meshgrid(np.arange(n), np.arange(n), indexing="ij"), axis=-1).reshape(-1, 2)
        out = np.empty((ij.shape[0], a.size, 4), dtype=np.int32)
        out[:, :, :2] = ij[:, None, :]
        out[:, :, 2] = a[None, :]
        out[:, :, 3] = b[None, :]
        return out.reshape(-1, 4)
    raise ValueError(op)


def _nao(mol, norb, sph):
    l = mol.bas[:norb, M.ANG_OF].astype(np.int64)
    return int((2 * l + 1 if sph else (l + 1) * (l + 2) // 2).sum())


def _density(nao, seed):
    """A symmetric density-like matrix (occupied-orbital outer products, trace of some nao / 2)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    c = torch.randn(nao, max(1, nao // 4), generator=g, device="cuda", dtype=torch.float64)
    return 2.0 * (c @ c.T) / nao


def _tune(plan, buf):
    """Tuned launch shapes: this process's earlier choices, timed now for classes it has not met."""
    nseg = sum(len(plan.segments(c)[1]) for c in range(int(plan.stats.nchunks)))
    if plan.use_tuned_shapes() < nseg:
        plan.autotune(buf.data_ptr(), -1, torch.cuda.current_stream().cuda_stream, 1)


def _sweep_buffer(case, st):
    """The device buffer a sweep writes, of one size for all geometries of the case (zeros past the
    sweep's end): every quartet, or for larger molecules 1.2 times the survivors that work() estimates."""
    mol, norb = _molecule(case, 1)
    nf = (2 * mol.bas[:, M.ANG_OF].astype(np.int64) + 1 if case["sph"]
          else (mol.bas[:, M.ANG_OF] + 1) * (mol.bas[:, M.ANG_OF] + 2) // 2)
    pairs = (int(nf[:norb].sum()) ** 2 + int((nf[:norb] ** 2).sum())) // 2
    full = pairs * int(nf[norb:].sum()) if case["op"] == "df3c" else (pairs + int(nf[:norb].max()) ** 4) ** 2 // 2
    n = int(min(full, 1.2 * _screened_counts(case)[0] + 1e5))
    if st.nchunks != 1 or st.nintegrals > n:
        raise ValueError("the sweep of %r holds %d integrals, %d expected at most" % (case, st.nintegrals, n))
    return torch.zeros(n, dtype=torch.float64, device="cuda")


def prepare(case, seed):
    mol, norb = _molecule(case, seed)
    op, sph = case["op"], case.get("sph", True)
    s = {"case": case, "mol": mol}
    if op == "call":
        s["shls"] = _tuples(case, mol, norb)[0]
        s["opt"] = cx.Optimizer(mol.atm, mol.bas, mol.env)
    elif op in ("batch", "metric"):
        family = cx.INT2E if op == "batch" else cx.INT2C2E
        s["opt"] = cx.Optimizer(mol.atm, mol.bas, mol.env, pair_shells=norb if op == "metric" else None)
        s["plan"] = cx.Plan.shells(s["opt"], family, _tuples(case, mol, norb), sph=sph)
        s["out"] = torch.empty(s["plan"].stats.nintegrals, dtype=torch.float64, device="cuda")
    elif op in ("sweep", "jk", "ao"):
        s["opt"] = cx.Optimizer(mol.atm, mol.bas, mol.env)
        chunk = ONE_CHUNK if op == "sweep" else 1 << 28
        tuned = case.get("tuned", False)
        if tuned:
            s["plan"] = cx.Plan.screened_mixed(s["opt"], CUTOFF, prim_budget=PRIM_BUDGET, max_chunk_doubles=chunk)
        else:
            s["plan"] = cx.Plan.screened(s["opt"], CUTOFF, sph=sph, max_chunk_doubles=chunk)
        st = s["plan"].stats
        if op == "sweep":
            s["out"] = _sweep_buffer(case, st)
        elif tuned:
            s["out"] = torch.empty(st.max_chunk_doubles, dtype=torch.float64, device="cuda")
        if tuned:
            _tune(s["plan"], s["out"])
        if op == "sweep" and tuned:
            s["plan"].graph_build(s["out"].data_ptr())
        nao = s["nao"] = _nao(mol, norb, sph)
        if op == "jk":
            s.pop("out", None)  # jk works in a ring of the plan's own
            s["dm"] = _density(nao, seed)
            s["vj"], s["vk"] = (torch.empty(nao, nao, dtype=torch.float64, device="cuda") for _ in range(2))
        if op == "ao":
            np2 = nao * (nao + 1) // 2
            n = {1: nao ** 4, 4: np2 * np2, 8: np2 * (np2 + 1) // 2}[case["aosym"]]
            s["eri"] = torch.empty(n, dtype=torch.float64, device="cuda")
    elif op == "df3c":
        s["opt"] = cx.Optimizer(mol.atm, mol.bas, mol.env, pair_shells=norb)
        s["plan"] = cx.Plan.screened_3c(s["opt"], norb, CUTOFF, sph=sph, max_chunk_doubles=ONE_CHUNK)
        s["out"] = _sweep_buffer(case, s["plan"].stats)
    elif op == "grad":
        s["family"] = cx.INT2E if case["centres"] == 4 else cx.INT3C2E
        s["tuples"] = _tuples(case, mol, norb)
        n = cx.ip1_len(s["family"], s["tuples"], mol.bas, sph)
        s["out"] = torch.empty(n, dtype=torch.float64, device="cuda")
    return s


def run(s):
    case, mol = s["case"], s["mol"]
    op, sph = case["op"], case.get("sph", True)
    stream = torch.cuda.current_stream().cuda_stream
    if op == "call":
        f = cx.int2e_sph if sph else cx.int2e_cart
        return f(s["shls"], mol.atm, mol.bas, mol.env, opt=s["opt"])[0]
    if op in ("batch", "metric", "df3c"):
        s["plan"].execute(s["out"].data_ptr(), -1, stream)
        return s["out"]
    if op == "sweep":
        if case["tuned"]:
            s["plan"].graph_launch(stream)
        else:
            s["plan"].execute(s["out"].data_ptr(), -1, stream)
        return s["out"]
    if op == "jk":
        s["plan"].jk(s["dm"].data_ptr(), s["nao"], s["vj"].data_ptr(), s["vk"].data_ptr(), stream)
        return {"vj": s["vj"], "vk": s["vk"]}
    if op == "ao":
        s["plan"].execute_ao(s["eri"].data_ptr(), s["eri"].numel(), case["aosym"], stream)
        return s["eri"]
    offs = cx.ip1_eval(s["family"], s["tuples"], mol.atm, mol.bas, mol.env, s["out"].data_ptr(), sph)
    return {"out": s["out"], "offsets": offs}


# ------------------------------------------------------------------------------ work

def _nf(l, sph):
    return 2 * l + 1 if sph else (l + 1) * (l + 2) // 2


def _flops(li, lj, lk, ll):
    """FP64 operations of one primitive quartet: recurrences, transfers and products of the Rys path
    (root evaluation left out)."""
    if (lk, ll) > (li, lj):
        li, lj, lk, ll = lk, ll, li, lj
    n = (li + lj + lk + ll) // 2 + 1
    nij, nkl = li + lj + 1, lk + ll + 1
    hrr = sum((nij - j) * nkl for j in range(1, lj + 1))
    hrr += sum((li + 1) * (lj + 1) * (nkl - m) for m in range(1, ll + 1))
    cart = 1
    for l in (li, lj, lk, ll):
        cart *= (l + 1) * (l + 2) // 2
    return 15.0 * n * nij * nkl + 6.0 * n * hrr + 3.0 * n * cart


def _pair_stats(mol, norb):
    """Of every orbital shell pair of mol: (larger l, smaller l), primitive pairs that pass libcint's
    exponent cut-off, and an estimate of its Schwarz factor sqrt((ab|ab))."""
    bas, env, atm = mol.bas[:norb], mol.env, mol.atm
    xyz = np.stack([env[atm[bas[:, 0], 1] + c] for c in range(3)], axis=1)
    a, b = np.tril_indices(norb)
    la, lb = bas[a, 1], bas[b, 1]
    npr, q = np.zeros(a.size), np.zeros(a.size)
    r2 = ((xyz[a] - xyz[b]) ** 2).sum(1)
    kinds = bas[:, 1] * 100 + bas[:, 2]
    for ka in np.unique(kinds):
        for kb in np.unique(kinds):
            sel = np.nonzero((kinds[a] == ka) & (kinds[b] == kb))[0]
            if not sel.size:
                continue
            na, nb = int(ka) % 100, int(kb) % 100
            ea, eb = (env[bas[x[sel], 5][:, None] + np.arange(n)] for x, n in ((a, na), (b, nb)))
            ca, cb = (np.abs(env[bas[x[sel], 6][:, None] + np.arange(n)]) for x, n in ((a, na), (b, nb)))
            p = ea[:, :, None] + eb[:, None, :]
            eij = ea[:, :, None] * eb[:, None, :] / p * r2[sel][:, None, None]
            lij = int(ka) // 100 + int(kb) // 100
            log_rr = 1.7 - 1.5 * np.log(ea[:, -1] + eb[:, -1]) + lij * np.log(np.sqrt(r2[sel]) + 1.0)
            c = ca[:, :, None] * cb[:, None, :]
            npr[sel] = (eij - log_rr[:, None, None] - np.log(c) < 60.0).sum((1, 2))
            diag = c * np.exp(-eij) * np.sqrt(2 * math.pi ** 2.5 / (p * p * np.sqrt(2 * p)))
            r = np.sqrt(r2[sel])[:, None, None]
            diag = diag * (np.sqrt(0.5 / p) + eb[:, None, :] / p * r) ** (int(ka) // 100)
            diag = diag * (np.sqrt(0.5 / p) + ea[:, :, None] / p * r) ** (int(kb) // 100)
            q[sel] = diag.sum((1, 2)) / (4 * math.pi)
    return np.maximum(la, lb), np.minimum(la, lb), npr, q


_WORK = {}


def _screened_counts(case):
    """(integrals, primitive flops) of the surviving quartets or triples, estimated on the host."""
    key = (case["op"] == "df3c", case["natm"], case["basis"], case["sph"])
    if key in _WORK:
        return _WORK[key]
    mol, norb = _molecule(case, 1)
    la, lb, npr, q = _pair_stats(mol, norb)
    cls = {}
    for c in sorted(set(zip(la.tolist(), lb.tolist()))):
        sel = np.nonzero((la == c[0]) & (lb == c[1]) & (npr > 0))[0]
        sel = sel[np.argsort(-q[sel])]
        cls[c] = (q[sel], np.concatenate([[0.0], np.cumsum(npr[sel])]), npr[sel])
    if key[0]:  # columns: auxiliary shells, one primitive each, (k|k) of a normalised shell
        aux = {}
        for r in mol.bas[norb:]:
            l, e, c = int(r[1]), mol.env[r[5]], mol.env[r[6]]
            kk = 2 * math.pi ** 2.5 / (e * e * math.sqrt(2 * e)) * c * c * (0.5 / e) ** l / (4 * math.pi)
            aux.setdefault((l, 0), []).append(math.sqrt(kk))
        aux = {c: (np.sort(v)[::-1].copy(), np.arange(len(v) + 1.0), np.ones(len(v))) for c, v in aux.items()}
    nint = flops = 0.0
    for c, (qr, _, nr) in cls.items():
        for d, (qc, cum, _) in (aux if key[0] else cls).items():
            if not key[0] and d > c:
                continue
            cnt = np.searchsorted(-qc, -(CUTOFF / np.maximum(qr, 1e-300)), side="right")
            half = 0.5 if not key[0] and c == d else 1.0
            nq = half * float(cnt.sum())
            blk = 1
            for l in c + d:
                blk *= _nf(l, case["sph"])
            nint += nq * blk
            flops += half * float((nr * cum[cnt]).sum()) * _flops(*c, *d)
    _WORK[key] = (nint, flops)
    return nint, flops


def work(case):
    op, sph = case["op"], case.get("sph", True)
    mol, norb = _molecule(case, 1)
    if op in ("sweep", "df3c", "jk", "ao"):
        nint, flops = _screened_counts(case)
        nao = _nao(mol, norb, sph)
        np2 = nao * (nao + 1) // 2
        if op == "jk":
            return {"bytes": 3 * 8.0 * nao * nao, "flops": flops + 12.0 * nint}
        if op == "ao":
            return {"bytes": 8.0 * {1: nao ** 4, 4: np2 ** 2, 8: np2 * (np2 + 1) // 2}[case["aosym"]], "flops": flops}
        return {"bytes": 8.0 * nint, "flops": flops}
    t = _tuples(case, mol, norb)
    l, npr = mol.bas[:, M.ANG_OF].astype(np.int64), mol.bas[:, M.NPRIM_OF].astype(np.int64)
    lt = np.zeros((t.shape[0], 4), dtype=np.int64)
    col = [0, 2] if t.shape[1] == 2 else list(range(t.shape[1]))
    lt[:, col] = l[t]
    code, inv = np.unique(lt @ np.array([125, 25, 5, 1]), return_inverse=True)
    nprq = np.bincount(inv, weights=np.prod(npr[t].astype(np.float64), axis=1))
    nq = np.bincount(inv)
    nint = flops = 0.0
    for c, k, n in zip(code.tolist(), nprq, nq):
        ls = (c // 125, c // 25 % 5, c // 5 % 5, c % 5)
        blk = 1
        for x, v in enumerate(ls):
            blk *= _nf(v, sph) if x in col else 1
        pairs = sorted((tuple(sorted(ls[:2], reverse=True)), tuple(sorted(ls[2:], reverse=True))), reverse=True)
        if op == "grad":  # three components over the raised recurrence
            nint += 3.0 * n * blk
            flops += k * 3.0 * _flops(ls[0] + 1, ls[1], ls[2], ls[3])
        else:
            nint += 1.0 * n * blk
            flops += k * _flops(*pairs[0], *pairs[1])
    return {"bytes": 8.0 * nint + 4.0 * t.size, "flops": flops}


# Double precision throughout.  Against exact(): blocks 4e-16 to 1e-14, tensors and matrices of
# screened sweeps up to 1.2e-12 (the Schwarz cut-off), of the tuned form up to 2.4e-12 (its primitive
# budget); largest single differences 2.5e-11 (gradients: cancelling terms of tight shells) and 7e-11
# (tuned).  Two runs of one J/K build differ by 4e-16 (atomic sums).
def tolerance(case):
    return {"rel": 1e-11, "max": 3e-10}


# ------------------------------------------------------------------------------ exact values
#
# McMurchie-Davidson in 64-bit torch: Hermite expansion of each primitive pair, Boys function from a
# Taylor grid, Hermite Coulomb tensors by recursion, contraction, cartesian -> spherical.

_BOYS = {}


def _boys_table(device):
    if device not in _BOYS:
        top, step, xmax = 28, 0.1, 100.0
        x = np.arange(int(xmax / step) + 2) * step
        f = np.zeros((x.size, top + 1))
        term = np.full(x.size, 1.0 / (2 * top + 1))
        acc = term.copy()
        for k in range(1, 400):
            term = term * 2 * x / (2 * top + 2 * k + 1)
            acc += term
        f[:, top] = np.exp(-x) * acc
        for m in range(top - 1, -1, -1):
            f[:, m] = (2 * x * f[:, m + 1] + np.exp(-x)) / (2 * m + 1)
        _BOYS[device] = (torch.as_tensor(f, device=device), step, xmax)
    return _BOYS[device]


def _boys(mmax, x):
    """F_0..F_mmax at x, as a list."""
    tab, step, xmax = _boys_table(x.device)
    small = x < xmax
    xs = torch.where(small, x, torch.zeros_like(x))
    k = torch.round(xs / step).long()
    d = k.double() * step - xs
    row = tab[k]
    top = torch.zeros_like(x)
    for t in range(9, -1, -1):
        top = top * d / (t + 1) + row[:, mmax + t]
    e = torch.exp(-xs)
    out = [None] * (mmax + 1)
    out[mmax] = top
    for m in range(mmax - 1, -1, -1):
        out[m] = (2 * xs * out[m + 1] + e) / (2 * m + 1)
    inv = 0.5 / torch.where(small, torch.ones_like(x), x)
    big = 0.5 * torch.sqrt(2 * math.pi * inv)
    for m in range(mmax + 1):
        out[m] = torch.where(small, out[m], big)
        big = big * (2 * m + 1) * inv
    return out


def _carts(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _herms(n):
    return [(t, u, v) for t in range(n + 1) for u in range(n + 1 - t) for v in range(n + 1 - t - u)]


def _c2s(l, sph):
    """Rows: functions, columns: cartesians.  libcint's factors: s and p carry theirs in both forms."""
    nc = (l + 1) * (l + 2) // 2
    if l == 0:
        return np.array([[0.5 / math.sqrt(math.pi)]])
    if l == 1:
        return math.sqrt(0.75 / math.pi) * np.eye(3)
    if not sph:
        return np.eye(nc)
    # real solid harmonics (Helgaker, Jorgensen, Olsen 6.4.47-50) times sqrt((2l+1)/4pi), m = -l..l
    fact, comb = math.factorial, math.comb
    idx = {c: i for i, c in enumerate(_carts(l))}
    out = np.zeros((2 * l + 1, nc))
    for m in range(-l, l + 1):
        am = abs(m)
        norm = math.sqrt(2.0 * fact(l + am) * fact(l - am) / (2.0 if m == 0 else 1.0)) / (2 ** am * fact(l))
        v0 = 0.5 if m < 0 else 0.0
        for t in range((l - am) // 2 + 1):
            for u in range(t + 1):
                v = v0
                while v <= am / 2.0:
                    w = (-1) ** int(t + v - v0) * 0.25 ** t * comb(l, t) * comb(l - t, am + t) * comb(t, u)
                    w *= comb(am, int(2 * v))
                    x, y = int(2 * t + am - 2 * (u + v)), int(2 * (u + v))
                    out[m + l, idx[(x, y, l - x - y)]] += norm * w
                    v += 1.0
    return out * math.sqrt((2 * l + 1) / (4 * math.pi))


class _Exact:
    """Blocks of shell tuples; a missing shell (-1) is the constant 1."""

    def __init__(self, mol, sph, deriv=False):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.mol, self.sph, self.deriv = mol, sph, deriv
        self.l = [int(r[M.ANG_OF]) for r in mol.bas]
        self.cache = {}

    def _shell(self, s):
        r, env = self.mol.bas[s], self.mol.env
        n = int(r[M.NPRIM_OF])
        return env[r[M.PTR_EXP]:r[M.PTR_EXP] + n], env[r[M.PTR_COEFF]:r[M.PTR_COEFF] + n], self.mol.coords[r[0]]

    def _pairs(self, pairs, first):
        key = (first, pairs.tobytes())
        if key not in self.cache:
            self.cache[key] = self._make_pairs([tuple(x) for x in pairs.tolist()], first)
        return self.cache[key]

    def _make_pairs(self, pairs, first):
        """Primitive pairs of shell pairs of one (la, lb): Hermite matrices [np, ncomp*na*nb, nherm]
        (first: the derivative pair, three components), exponents, centres, and offsets per pair."""
        la = self.l[pairs[0][0]]
        lb = 0 if pairs[0][1] < 0 else self.l[pairs[0][1]]
        p, P, PA, PB, K, A2, cnt = [], [], [], [], [], [], []
        for a, b in pairs:
            ea, ca, ra = self._shell(a)
            eb, cb, rb = (np.zeros(1), np.ones(1), ra) if b < 0 else self._shell(b)
            pp = (ea[:, None] + eb[None, :]).ravel()
            cen = (ea[:, None, None] * ra + eb[None, :, None] * rb).reshape(-1, 3) / pp[:, None]
            mu = (ea[:, None] * eb[None, :]).ravel() / pp
            K.append((ca[:, None] * cb[None, :]).ravel() * np.exp(-mu * ((ra - rb) ** 2).sum()))
            p.append(pp)
            P.append(cen)
            # P - A from the exponents, without cancellation
            PA.append((np.broadcast_to(eb[None, :], (ea.size, eb.size)).ravel() / pp)[:, None] * (rb - ra))
            PB.append((np.broadcast_to(ea[:, None], (ea.size, eb.size)).ravel() / pp)[:, None] * (ra - rb))
            A2.append(np.repeat(2.0 * ea, eb.size))
            cnt.append(pp.size)
        t = lambda v: torch.as_tensor(np.concatenate(v), device=self.dev)  # noqa: E731
        p, P, PA, PB, K, A2 = (t(v) for v in (p, P, PA, PB, K, A2))
        ra_ = la + (1 if first and self.deriv else 0)
        half = 0.5 / p
        E = []  # per axis: E[i][j] = list over t
        for ax in range(3):
            e = [[None] * (lb + 1) for _ in range(ra_ + 1)]
            e[0][0] = [torch.ones_like(p)]

            def up(src, x):
                n = len(src)
                out = []
                for k in range(n + 1):
                    v = torch.zeros_like(p)
                    if k > 0:
                        v = v + half * src[k - 1]
                    if k < n:
                        v = v + x * src[k]
                    if k + 1 < n:
                        v = v + (k + 1) * src[k + 1]
                    out.append(v)
                return out

            for i in range(ra_ + 1):
                if i > 0:
                    e[i][0] = up(e[i - 1][0], PA[:, ax])
                for j in range(1, lb + 1):
                    e[i][j] = up(e[i][j - 1], PB[:, ax])
            E.append(e)
        L = ra_ + lb
        herm = _herms(L)
        zero = torch.zeros_like(p)

        def pick(ax, i, j, t, diff):
            if not diff:
                return E[ax][i][j][t] if t <= i + j else zero
            v = zero
            if t <= i + 1 + j:
                v = v - A2 * E[ax][i + 1][j][t]
            if i > 0 and t <= i - 1 + j:
                v = v + i * E[ax][i - 1][j][t]
            return v

        comps = range(3) if first and self.deriv else [None]
        rows = []
        for c in comps:
            for ci in _carts(la):
                for cj in _carts(lb):
                    f = [[pick(ax, ci[ax], cj[ax], t, c == ax) for t in range(L + 1)] for ax in range(3)]
                    rows.append(torch.stack([K * f[0][h[0]] * f[1][h[1]] * f[2][h[2]] for h in herm], dim=1))
        H = torch.stack(rows, dim=1)
        off = np.concatenate([[0], np.cumsum(cnt)])
        return {"H": H, "p": p, "P": P, "off": off, "cnt": np.asarray(cnt), "L": L, "n": len(rows)}

    def blocks(self, tuples):
        """Yields (indices of tuples, blocks [n, (3,) ni, nj, nk, nl]) class by class."""
        tuples = np.asarray(tuples)
        l = np.array(self.l + [0])  # -1 -> 0
        code = l[tuples] @ np.array([1000, 100, 10, 1]) * 16 + (tuples < 0) @ np.array([8, 4, 2, 1])
        for c in np.unique(code):
            sel = np.nonzero(code == c)[0]
            tt = tuples[sel]
            ab, iab = np.unique(tt[:, :2], axis=0, return_inverse=True)
            cd, icd = np.unique(tt[:, 2:], axis=0, return_inverse=True)
            ls = [int(v) for v in l[tt[0]]]
            prt = [self._pairs(ab, True), self._pairs(cd, False)]
            nprq = prt[0]["cnt"][iab.ravel()] * prt[1]["cnt"][icd.ravel()]
            hab, hcd = _herms(prt[0]["L"]), _herms(prt[1]["L"])
            Lt = prt[0]["L"] + prt[1]["L"]
            per = len(hab) * len(hcd) + (Lt + 1) * (Lt + 2) * (Lt + 3) // 3 + prt[0]["n"] * (len(hab) + len(hcd) + prt[1]["n"])
            budget = max(1, int(4e8 / per))  # primitive quartets at once
            start = 0
            cum = np.concatenate([[0], np.cumsum(nprq)])
            while start < sel.size:
                stop = max(start + 1, int(np.searchsorted(cum, cum[start] + budget, side="right")) - 1)
                yield sel[start:stop], self._run(prt, iab.ravel()[start:stop], icd.ravel()[start:stop], ls, tt[0], hab, hcd)
                start = stop

    def _run(self, prt, iab, icd, ls, unit, hab, hcd):
        dev = self.dev
        A, C = prt
        na, nc = torch.as_tensor(A["cnt"][iab], device=dev), torch.as_tensor(C["cnt"][icd], device=dev)
        n = na * nc
        q = torch.repeat_interleave(torch.arange(len(iab), device=dev), n)
        r = torch.arange(int(n.sum()), device=dev) - torch.repeat_interleave(torch.cumsum(n, 0) - n, n)
        oa = torch.as_tensor(A["off"][:-1][iab], device=dev)
        oc = torch.as_tensor(C["off"][:-1][icd], device=dev)
        ip = oa[q] + torch.div(r, nc[q], rounding_mode="floor")
        kp = oc[q] + r % nc[q]
        p, k = A["p"][ip], C["p"][kp]
        d = A["P"][ip] - C["P"][kp]
        al = p * k / (p + k)
        L = A["L"] + C["L"]
        f = _boys(L, al * (d * d).sum(1))
        fac = 2 * math.pi ** 2.5 / (p * k * torch.sqrt(p + k))
        lev = {}
        for m in range(L, -1, -1):  # R^(m)_{tuv}, t + u + v <= L - m
            new = {(0, 0, 0): fac * (-2 * al) ** m * f[m]}
            for t, u, v in sorted(_herms(L - m), key=sum):
                if t + u + v == 0:
                    continue
                ax = 0 if t else (1 if u else 2)
                e = [t, u, v]
                e[ax] -= 1
                x = d[:, ax] * lev[tuple(e)]
                if e[ax] > 0:
                    w = e[ax]
                    e[ax] -= 1
                    x = x + w * lev[tuple(e)]
                new[(t, u, v)] = x
            lev = new
        R = torch.stack([lev[h] for h in _herms(L)], dim=1)
        at = {h: i for i, h in enumerate(_herms(L))}
        idx = torch.as_tensor([[at[tuple(x + y for x, y in zip(a, c))] for c in hcd] for a in hab], device=dev)
        sgn = torch.as_tensor([(-1.0) ** sum(c) for c in hcd], device=dev, dtype=torch.float64)
        T = torch.bmm(A["H"][ip], R[:, idx])
        B = torch.bmm(T, (C["H"][kp] * sgn).transpose(1, 2))
        out = torch.zeros(len(iab), A["n"], C["n"], dtype=torch.float64, device=dev).index_add_(0, q, B)
        ncar = [(x + 1) * (x + 2) // 2 for x in ls]
        out = out.reshape([len(iab), A["n"] // (ncar[0] * ncar[1])] + ncar)
        for ax in range(4):
            if unit[ax] < 0:
                continue
            m = torch.as_tensor(_c2s(ls[ax], self.sph), device=dev)
            out = torch.movedim(torch.tensordot(out, m, dims=([ax + 2], [1])), -1, ax + 2)
        return out


def exact(case, seed):
    op, sph = case["op"], case.get("sph", True)
    if op in ("sweep", "df3c"):
        return None  # the order of a sweep's blocks is the plan's own
    mol, norb = _molecule(case, seed)
    if op in ("jk", "ao"):
        if case["natm"] > (9 if case["basis"] == "spdf" else 14):
            return None
        t = _unique_quartets(norb)
    elif op == "batch" and case["basis"] == "g" and case["natm"] > 3:
        return None  # half a minute
    else:
        t = _tuples(case, mol, norb)
    if t.shape[1] == 3:
        t = np.concatenate([t, np.full((t.shape[0], 1), -1, dtype=t.dtype)], axis=1)
    elif t.shape[1] == 2:
        m1 = np.full((t.shape[0], 1), -1, dtype=t.dtype)
        t = np.concatenate([t[:, :1], m1, t[:, 1:], m1], axis=1)
    eng = _Exact(mol, sph, deriv=op == "grad")
    nf = np.array([_nf(v, sph) for v in eng.l] + [1])
    size = np.prod(nf[t], axis=1) * (3 if op == "grad" else 1)
    dev = eng.dev
    if op in ("jk", "ao"):
        loc = np.concatenate([[0], np.cumsum(nf[:norb])])
        nao = int(loc[-1])
        eri = torch.zeros(nao, nao, nao, nao, dtype=torch.float64, device=dev)
        for sel, b in eng.blocks(t):
            b = b[:, 0]
            ax = [torch.as_tensor(loc[t[sel, c]], device=dev).reshape(-1, 1, 1, 1, 1)
                  + torch.arange(b.shape[c + 1], device=dev).reshape([-1 if x == c else 1 for x in range(4)]) for c in range(4)]
            ax = [a.expand(b.shape) for a in ax]
            for o in ((0, 1, 2, 3), (1, 0, 2, 3), (0, 1, 3, 2), (1, 0, 3, 2)):
                i, j, k, l = (ax[x] for x in o)
                eri[i, j, k, l] = b
                eri[k, l, i, j] = b
        if op == "jk":
            dm = _density(nao, seed)
            return {"vj": torch.einsum("pqrs,rs->pq", eri, dm), "vk": torch.einsum("pqrs,qs->pr", eri, dm)}
        if case["aosym"] == 1:
            return eri.reshape(-1)
        i, j = (torch.as_tensor(v, device=dev) for v in np.tril_indices(nao))
        pair = eri[i, j][:, i, j]
        if case["aosym"] == 4:
            return pair.reshape(-1)
        a, b = (torch.as_tensor(v, device=dev) for v in np.tril_indices(i.numel()))
        return pair[a, b]
    off = np.concatenate([[0], np.cumsum(size)])
    out = torch.empty(int(off[-1]), dtype=torch.float64, device=dev)
    for sel, b in eng.blocks(t):
        flat = b.permute(0, 1, 5, 4, 3, 2).reshape(len(sel), -1)  # component, then l, k, j, i (i fastest)
        out[torch.as_tensor(off[:-1][sel], device=dev)[:, None] + torch.arange(flat.shape[1], device=dev)] = flat
    if op == "call":
        return out.cpu().numpy()
    if op == "grad":
        return {"out": out, "offsets": None}
    return out
