"""The work that users of this framework have it do, as timed cases.

A case is a dict of plain values; `listed()` names twelve of them, `draw(rng)` gives more of the same
ranges, `prepare(case, seed)` makes what a program has in hand before the call, `run(state)` is one
pass through the public entry points, `work(case)` the bytes and operations a pass cannot do without
and `exact(case, seed)` the same results in plain 64-bit torch where that is cheap enough.

Operations (`op`):
  solve   vhci_b200.solve(path): the whole procedure on an input file (heat-bath iterations, PT2)
  build   build_h + apply_h: the Hamiltonian of a given basis, and a product with it
  eigs    set_basis + eigs: the lowest k states in a given basis, from a cold start
  apply   apply_h: H X for a block of host vectors
  resid   residual_norms_noalloc: residual norms of device-resident vectors
  pt2     set_vectors + pt2: the perturbative correction on given (e.g. checkpointed) vectors

Potentials are the seeded synthetic ones of vhci_b200/pes.py (the first admissible draw of each
workload, restricted to its first `modes` modes); a case's seed scales every force constant by about
2 % and every frequency by about 0.5 %, so each seed is another molecule of the same kind.  Bases
are like the ones that heat-bath selection leaves: half of the n product states are a core of low
harmonic energy, the others are reached from it through the stronger force constants in two more
rounds; each round is appended in ascending key order, as the library does.
"""
import functools
import itertools
import math
import os
import tempfile

import numpy as np
import torch

from vhci_b200 import VHCI, pes, solve

#: workload of pes.WORKLOADS whose potential a case uses
POTENTIALS = {"quartic12": 0, "quartic15": 1, "quartic48": 2, "sextic30": 4}


def listed():
    return [
        # the smallest request of the serving range: a triatomic-sized solve, latency counts
        dict(name="solve_6modes", op="solve", pes="quartic12", modes=6, eps=3.0, k=10, pt2=1),
        # the benchmark's 12-mode solve (fifty states, no PT2), whole
        dict(name="solve_12modes", op="solve", pes="quartic12", modes=12, eps=1.0, k=50, pt2=0),
        # Hamiltonian of a large 15-mode basis (one 64-bit word a key)
        dict(name="build_15modes", op="build", pes="quartic15", modes=15, n=150001, b=1, precision=0),
        # Hamiltonian of a 48-mode basis (three words a key, many groups a state)
        dict(name="build_48modes", op="build", pes="quartic48", modes=48, n=200000, b=1, precision=0),
        # terms up to sixth order, FP32 storage: the memory-bound form
        dict(name="build_30modes_f32", op="build", pes="sextic30", modes=30, n=40000, b=1, precision=1),
        # a heat-bath iteration's eigensolve with many states wanted
        dict(name="eigs_15modes", op="eigs", pes="quartic15", modes=15, n=120011, k=200, precision=0),
        # the same in mixed precision on many modes
        dict(name="eigs_48modes_f32", op="eigs", pes="quartic48", modes=48, n=60011, k=100, precision=1),
        # a small basis, solved densely
        dict(name="eigs_dense", op="eigs", pes="quartic12", modes=12, n=1500, k=20, precision=0),
        # a block product on host vectors, as a caller's own iteration would ask for
        dict(name="apply_15modes", op="apply", pes="quartic15", modes=15, n=150001, b=16, precision=0),
        # convergence check of a few vectors of a small basis, on the device: latency
        dict(name="resid_small", op="resid", pes="quartic12", modes=10, n=3001, k=10, precision=0),
        # convergence check of a full set of states of a large basis, on the device
        dict(name="resid_15modes", op="resid", pes="quartic15", modes=15, n=150001, k=200, precision=0),
        # PT2 on given vectors
        dict(name="pt2_15modes", op="pt2", pes="quartic15", modes=15, n=60000, k=100, eps=0.01, precision=0),
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    op = rng.choice(["solve", "build", "eigs", "apply", "resid", "pt2"])
    if op == "solve":
        return dict(op=op, pes="quartic12", modes=rng.randint(6, 12), eps=round(log(1.0, 3.0), 4), k=rng.randint(10, 50),
                    pt2=rng.randint(0, 1))
    if op == "pt2":
        return dict(op=op, pes="quartic15", modes=rng.randint(10, 15), n=int(log(500, 60000)), k=rng.randint(5, 100),
                    eps=round(log(0.01, 0.5), 4), precision=0)
    kind, most = rng.choice([("quartic15", 15), ("quartic15", 15), ("quartic48", 48), ("sextic30", 30)])
    # fewer modes reach a size only by states of many quanta, which the force fields are not made for
    modes = rng.randint(10 if most == 15 else 15, most)
    precision = rng.randint(0, 1)
    if op == "build":
        return dict(op=op, pes=kind, modes=modes, n=int(log(1000, 30000 if kind == "sextic30" else 150000)), b=rng.randint(1, 4),
                    precision=precision)
    if op == "eigs":
        return dict(op=op, pes=kind, modes=modes, n=int(log(400, 20000 if kind == "sextic30" else 60000)), k=rng.randint(5, 100),
                    precision=precision)
    if op == "apply":
        return dict(op=op, pes=kind, modes=modes, n=int(log(1000, 30000 if kind == "sextic30" else 150000)), b=rng.randint(1, 40),
                    precision=precision)
    return dict(op=op, pes=kind, modes=modes, n=int(log(1000, 30000 if kind == "sextic30" else 150000)), k=rng.randint(1, 200),
                precision=precision)


@functools.lru_cache(maxsize=None)
def _potential(kind, modes):
    """(frequencies, force constants) of the workload's potential over its first `modes` modes."""
    w = POTENTIALS[kind]
    full = pes.generate(pes.WORKLOADS[w][0], pes.workload_seed(w))
    return tuple(full.freqs[:modes]), tuple((ms, v) for ms, v in full.fcs if max(ms) < modes)


def _molecule(case, seed):
    """The case's potential for one seed: (frequencies, [(modes, value)])."""
    freqs, fcs = _potential(case["pes"], case["modes"])
    rng = np.random.Generator(np.random.PCG64([seed, 11]))
    f = np.array(freqs) * (1 + 0.005 * rng.standard_normal(len(freqs)))
    v = np.array([x for _, x in fcs]) * (1 + 0.02 * rng.standard_normal(len(fcs)))
    return [float("%.6f" % x) for x in f], [(ms, float("%.10f" % x)) for (ms, _), x in zip(fcs, v)]


@functools.lru_cache(maxsize=None)
def _changes(kind, modes):
    """(quanta changes, cumulated share of each) of a potential, shares by size of force constant."""
    found = _patterns(_potential(kind, modes)[1])
    found.pop((), None)
    delta = np.zeros((len(found), modes), np.int8)
    for i, d in enumerate(found):
        for m, x in d:
            delta[i, m] = x
    size = np.array([sum(abs(c) for c, _ in terms) for terms in found.values()])
    return delta, np.cumsum(size / size.sum())


def _core(freq, n, cap):
    """The n states of lowest harmonic energy."""
    step, emax = 5.0, 320.0
    while True:  # an energy bound that holds them, by counting on a grid
        count = np.zeros(int(emax / step) + 1)
        count[0] = 1
        for w in freq:
            s = max(1, int(w / step))
            for e in range(s, len(count)):
                count[e] += count[e - s]
        if count.sum() >= 1.2 * n + 10:
            break
        emax *= 1.3
    emax = step * (np.searchsorted(np.cumsum(count), 1.2 * n + 10) + 8)
    while True:
        q, e = np.zeros((1, len(freq)), np.uint8), np.zeros(1)
        for i, w in enumerate(freq):
            reps = np.minimum(cap, np.floor((emax - e) / w)).astype(np.int64) + 1
            at = np.repeat(np.arange(len(e)), reps)
            j = np.arange(len(at)) - np.repeat(np.cumsum(reps) - reps, reps)
            q, e = q[at], e[at] + j * w
            q[:, i] = j
        if len(e) >= n:
            return q[np.argsort(e, kind="stable")[:n]]
        emax *= 1.1


def _basis(case, freq, seed, cap=12):
    """n states (quanta, harmonic energies above the zero point): a core and two rounds of growth."""
    n, modes = case["n"], len(freq)
    rng = np.random.Generator(np.random.PCG64([seed, 14]))
    delta, share = _changes(case["pes"], modes)
    mult = np.random.Generator(np.random.PCG64(5)).integers(-2**62, 2**62, modes)
    q = _core(freq, -(-n // 2), cap)
    parts = [q]
    for want in (n // 4, n - len(q) - n // 4):
        have = np.sort(q.astype(np.int64) @ mult)  # a linear hash tells states apart
        new, keys = np.zeros((0, modes), np.uint8), np.zeros(0, np.int64)
        while len(new) < want:
            m = 2 * (want - len(new)) + 1000
            t = q[rng.integers(0, len(q), m)].astype(np.int8) + delta[np.searchsorted(share, rng.random(m)).clip(max=len(delta) - 1)]
            t = t[((t >= 0) & (t <= cap)).all(1)].astype(np.uint8)
            new = np.concatenate([new, t])
            keys = np.concatenate([keys, t.astype(np.int64) @ mult])
            at = np.searchsorted(have, keys).clip(max=len(have) - 1)
            first = np.zeros(len(keys), bool)
            first[np.unique(keys, return_index=True)[1]] = True
            new, keys = new[first & (have[at] != keys)], keys[first & (have[at] != keys)]
        parts.append(new[:want])
        q = np.concatenate([q, new[:want]])
    for i, part in enumerate(parts):
        key = np.zeros((-(-modes // 16), len(part)), np.uint64)
        for m in range(modes):
            key[m // 16] |= part[:, m].astype(np.uint64) << np.uint64(4 * (m % 16))
        parts[i] = part[np.lexsort(key)]
    q = np.ascontiguousarray(np.concatenate(parts))
    return q, q @ np.array(freq)


def _context(case, seed):
    freq, fcs = _molecule(case, seed)
    q, e = _basis(case, freq, seed)
    v = VHCI(problem=dict(freq=freq, cap=[8] * len(freq), ntot=1, fcs=fcs, eps1=0.0, nstate=case.get("k", 1), pt2=1, eps2=case.get("eps", 0.0)),
             precision=case["precision"])
    return v, freq, q, e


def _block(n, b, seed):
    """A block of b unit vectors, n x b, as a Krylov iteration holds it."""
    x = np.random.Generator(np.random.PCG64([seed, 12])).standard_normal((n, b))
    return x / np.linalg.norm(x, axis=0)


def _vectors(freq, e, k, seed):
    """Vectors and energies like an eigensolve's: each column spread around one low state, its
    coefficients falling off over decades; energies of the lowest states."""
    rng = np.random.Generator(np.random.PCG64([seed, 13]))
    low = np.sort(e)[:k]
    c = rng.standard_normal((len(e), k)) * np.exp(-np.abs(e[:, None] - low) / 900.0)
    c *= 10.0 ** (-2.5 * rng.random((len(e), 1)))
    c[np.argsort(e, kind="stable")[:k], np.arange(k)] = 1.0
    return np.asfortranarray(c / np.linalg.norm(c, axis=0)), 0.5 * sum(freq) + 0.99 * low


def prepare(case, seed):
    op = case["op"]
    if op == "solve":
        freq, fcs = _molecule(case, seed)
        folder = tempfile.TemporaryDirectory(prefix="vhci_cases_")
        path = os.path.join(folder.name, "input.inp")
        pes.write_input(path, pes.PES(freqs=freq, caps=[8] * len(freq), fcs=fcs),
                        pes.RunSettings(eps1=case["eps"], nstate=case["k"], pt2=case["pt2"], eps2=0.1 * case["eps"] * case["pt2"]))
        return dict(op=op, path=path, folder=folder, pt2=case["pt2"])
    v, freq, q, e = _context(case, seed)
    state = dict(op=op, v=v, q=q, k=case.get("k"), eps=case.get("eps"))
    if op == "eigs":
        return state
    v.set_basis(q)
    if op in ("build", "apply"):
        state["X"] = np.asfortranarray(_block(case["n"], case["b"], seed))
    if op == "resid":
        state["X"] = torch.from_numpy(_block(case["n"], case["k"], seed)).cuda()
        state["theta"] = torch.from_numpy(0.5 * sum(freq) + np.sort(e)[: case["k"]]).cuda()
        state["r"] = torch.zeros(case["k"], dtype=torch.float64, device="cuda")
    if op in ("apply", "resid"):
        v.build_h()
    if op == "pt2":
        state["C"], state["E"] = _vectors(freq, e, case["k"], seed)
    return state


def run(state):
    op, v = state["op"], state.get("v")
    if op == "solve":
        r = solve(state["path"])
        return {"E": r["E"], "E_var": r["E_var"], "n_basis": int(r["n_basis"]), "n_pert": int(r["n_pert"])}
    if op == "build":
        return {"nnz": v.build_h(), "Y": v.apply_h(state["X"])}
    if op == "eigs":
        v.set_basis(state["q"])
        return v.eigs(state["k"])
    if op == "apply":
        return v.apply_h(state["X"])
    if op == "resid":
        v.residual_norms_noalloc(state["X"].data_ptr(), state["theta"].data_ptr(), state["r"].data_ptr(), state["k"])
        return state["r"]
    v.set_vectors(state["C"], state["E"])
    dE, n_pert = v.pt2(state["eps"])
    return {"dE": dE, "n_pert": int(n_pert), "E": v.energies()}


def work(case):
    """Of one pass: the stored matrix (12 bytes an entry, 8 in FP32 storage) written once by a build
    and read once by a product, an eigensolve reading it at least once per 16 wanted states and
    rotating its vectors once; PT2 reads each connection once and gathers its row of the vectors."""
    k = case.get("k", 1)
    if case["op"] == "solve":
        s = prepare(case, 0)
        with VHCI(s["path"]) as v:
            v.hci()
            n, nnz = v.n, int(v.info.h_nnz)
            if case["pt2"]:
                v.pt2()
            ent = v.stats()["pt2_entries"]
        return {"bytes": 12.0 * nnz * (1 + -(-k // 16)) + 8.0 * n * k + ent * (12.0 + 8.0 * k),
                "flops": 2.0 * nnz * k + 2.0 * n * k * k + 2.0 * ent * k}
    v, _, q, e = _context(case, 0)
    n = case["n"]
    with v:
        v.set_basis(q)
        if case["op"] == "pt2":
            freq, _ = _molecule(case, 0)
            v.set_vectors(*_vectors(freq, e, k, 0))
            _, p = v.pt2(case["eps"])
            ent = v.stats()["pt2_entries"]
            return {"bytes": 8.0 * n * k + 12.0 * ent + 8.0 * p, "flops": 2.0 * ent * k}
        nnz = v.build_h() - n
    h = nnz * (8.0 if case["precision"] else 12.0) + 16.0 * n
    b = case.get("b", k)
    if case["op"] == "build":
        return {"bytes": 2 * h + 16.0 * n * b, "flops": 2.0 * nnz * b + 8.0 * nnz}
    if case["op"] == "apply":
        return {"bytes": h + 16.0 * n * b, "flops": 2.0 * nnz * b}
    if case["op"] == "resid":
        return {"bytes": h + 8.0 * n * b, "flops": 2.0 * nnz * b}
    return {"bytes": h * (1 + -(-k // 16)) + 8.0 * n * k, "flops": 2.0 * nnz * k + 2.0 * n * k * k}


# ---- the Hamiltonian in plain 64-bit torch ------------------------------------------------------

#: change patterns beyond which the plain form takes too long
MOST_PATTERNS = 30000


def _patterns(fcs):
    """{quanta change: [(coefficient, [(mode, power, change)])]} of V = sum phi/prod(p!) prod q^p with
    q = (a + a^+)/sqrt(2)."""
    found = {}
    for ms, v in fcs:
        modes = sorted(set(ms))
        pw = [ms.count(m) for m in modes]
        c = v / math.sqrt(2.0 ** len(ms)) / math.prod(math.factorial(p) for p in pw)
        for d in itertools.product(*[range(-p, p + 1, 2) for p in pw]):
            delta = tuple((m, x) for m, x in zip(modes, d) if x)
            found.setdefault(delta, []).append((c, list(zip(modes, pw, d))))
    return found


def _apply(freq, fcs, quanta, x):
    """H x over the basis `quanta` for the columns of x, in 64 bits; None where it takes too long."""
    found = _patterns(fcs)
    if len(found) > MOST_PATTERNS:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    size = 40  # ladder matrix of q * sqrt(2), powers of it exact for quanta well below `size`
    up = np.diag(np.sqrt(np.arange(1.0, size)), 1)
    power = [np.eye(size)]
    for _ in range(6):
        power.append(power[-1] @ (up + up.T))
    q = torch.from_numpy(quanta.astype(np.int64)).to(dev)
    mult = torch.from_numpy(np.random.Generator(np.random.PCG64(5)).integers(-2**62, 2**62, quanta.shape[1])).to(dev)
    key = (q * mult).sum(1)  # a linear hash: a change of quanta adds a constant
    skey, place = torch.sort(key)
    x = torch.from_numpy(np.ascontiguousarray(x)).to(dev) if isinstance(x, np.ndarray) else x.to(dev)
    factors = {}

    def factor(m, p, d):
        if (m, p, d) not in factors:
            col = np.array([power[p][a, a + d] if a + d >= 0 else 0.0 for a in range(20)])
            factors[m, p, d] = torch.from_numpy(col).to(dev)[q[:, m]]
        return factors[m, p, d]

    y = x * ((q.double() + 0.5) * torch.tensor(freq, dtype=torch.float64, device=dev)).sum(1)[:, None]
    mults = [int(t) for t in mult.cpu()]
    for delta, terms in found.items():
        c = 0.0
        for fc, parts in terms:
            t = fc
            for part in parts:
                t = t * factor(*part)
            c = c + t
        if not delta:
            y += c[:, None] * x
            continue
        shift = (sum(mults[m] * d for m, d in delta) + 2**63) % 2**64 - 2**63
        want = key + shift
        at = torch.searchsorted(skey, want).clamp_(max=len(skey) - 1)
        hit = skey[at] == want
        y += torch.where(hit, c, 0.0)[:, None] * x[place[at]]
    return y


def exact(case, seed):
    if case["op"] in ("solve", "pt2") or (case["op"] == "eigs" and case["n"] > 2000):
        return None
    freq, fcs = _molecule(case, seed)
    q, e = _basis(case, freq, seed)
    if case["op"] == "eigs":
        h = _apply(freq, fcs, q, np.eye(case["n"]))
        return None if h is None else torch.linalg.eigvalsh((0.5 * (h + h.T)).cpu())[: case["k"]]
    x = torch.from_numpy(_block(case["n"], case.get("b", case.get("k")), seed))
    y = _apply(freq, fcs, q, x)
    if y is None:
        return None
    if case["op"] == "resid":
        theta = torch.from_numpy(0.5 * sum(freq) + np.sort(e)[: case["k"]]).to(y.device)
        return (y - theta * x.to(y.device)).norm(dim=0)
    return {"nnz": None, "Y": y} if case["op"] == "build" else y
