"""Workloads of the simulator, one dict of plain values per case, timed and
compared through the package's public entry points.

Kinds of case:

``layer``      one brickwork layer (a one-qudit gate on every site, two-qudit
               gates on every pair) on a chain in the steady state, where the
               bonds have reached the truncation: ``MPS.apply_layer`` on a
               copy of the state.  This is what a simulation spends its time
               in.  Outputs: for every pair of the layer the merged two-site
               tensor (left factor times right factor), and any site outside a
               pair; the two factors of a truncated SVD are only defined up to
               a phase per singular value, their product is not.
``circuit``    a whole small circuit through the reference's own call,
               ``MPS.apply`` on a list of ``MPSOperation`` from the product
               state, no truncation, then the wavefunction.
``plan``       a batch of independent circuits as one ``CircuitPlan``, run once,
               then amplitudes of sampled bitstrings of every circuit.
``overlap``    squared norm of a state and its inner product with a nearby
               one (fidelity of a perturbed or further truncated copy).
``amplitudes`` amplitudes of sampled bitstrings (cross-entropy checks).
``marginals``  every single-site marginal, what ``MPS.sample`` draws from.
``vector``     a state vector split into a matrix product state and contracted
               back: ``MPS.from_wavefunction``, then ``wavefunction``.
"""

import math

import numpy as np
import torch

from mpsim_gb300 import MPS, MPSOperation
from mpsim_gb300 import circuits as C
from mpsim_gb300.plan import CircuitPlan


# -- cases --------------------------------------------------------------------

def listed():
    return [
        # the smallest calls: a 10-qubit, depth-10 circuit as a user of the
        # gate-by-gate interface writes it; latency and launches count
        {"name": "circuit_10q_d10", "kind": "circuit", "n": 10, "d": 2, "depth": 10},
        # a small chain with an odd bond dimension
        {"name": "layer_24q_chi37", "kind": "layer", "n": 24, "d": 2, "chi": 37, "first": 1,
         "left": True, "precision": "plain"},
        # a layer of the 48-qubit, maxsvals=128 circuit
        {"name": "layer_48q_chi128", "kind": "layer", "n": 48, "d": 2, "chi": 128, "first": 0,
         "left": True, "precision": "plain"},
        # a layer of the 64-qubit, maxsvals=256 circuit
        {"name": "layer_64q_chi256", "kind": "layer", "n": 64, "d": 2, "chi": 256, "first": 0,
         "left": True, "precision": "plain"},
        # a right-canonical layer (the way back of a two-way sweep), ragged
        # sizes, an odd number of sites
        {"name": "layer_33q_chi100_right", "kind": "layer", "n": 33, "d": 2, "chi": 100, "first": 1,
         "left": False, "precision": "plain"},
        # a layer of the 32-qutrit, maxsvals=192 circuit
        {"name": "layer_32t_chi192", "kind": "layer", "n": 32, "d": 3, "chi": 192, "first": 0,
         "left": True, "precision": "plain"},
        # a long chain in the tensor-core (split-precision) form
        {"name": "layer_128q_chi256_mixed", "kind": "layer", "n": 128, "d": 2, "chi": 256, "first": 0,
         "left": True, "precision": "mixed"},
        # many small circuits together (the batched form)
        {"name": "plan_24x20q_d8_chi128", "kind": "plan", "count": 24, "n": 20, "d": 2,
         "depth": 8, "maxsvals": 128, "bits": 64},
        # read-outs of the steady states above
        {"name": "overlap_64q_chi256", "kind": "overlap", "n": 64, "d": 2, "chi": 256},
        {"name": "amplitudes_64q_chi256", "kind": "amplitudes", "n": 64, "d": 2, "chi": 256,
         "bits": 4096},
        {"name": "marginals_48q_chi128", "kind": "marginals", "n": 48, "d": 2, "chi": 128},
        # state vector in, state vector out
        {"name": "vector_14q", "kind": "vector", "n": 14, "d": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["layer"] * 8 + ["circuit", "plan", "overlap", "amplitudes", "marginals",
                                       "vector"])
    d = 3 if rng.random() < 0.25 else 2
    top = 256 if d == 2 else 192
    if kind == "layer":
        chi = _log_int(rng, 16, top)
        precision = rng.choice(["plain", "plain", "plain", "mixed", "auto"])
        n = rng.randint(12, 96 if precision == "mixed" else 64)
        if chi * d > 512:
            n = min(n, 40)
        return {"kind": kind, "n": n, "d": d, "chi": chi, "first": rng.randint(0, 1),
                "left": rng.random() < 0.75, "precision": precision}
    if kind == "circuit":
        return {"kind": kind, "n": rng.randint(3, 12 if d == 2 else 7), "d": d,
                "depth": rng.randint(2, 12)}
    if kind == "plan":
        return {"kind": kind, "count": _log_int(rng, 4, 32), "n": rng.randint(12, 24), "d": 2,
                "depth": 8, "maxsvals": rng.choice([64, 128]), "bits": rng.randint(16, 128)}
    if kind == "overlap":
        return {"kind": kind, "n": rng.randint(12, 80), "d": d, "chi": _log_int(rng, 16, top)}
    if kind == "amplitudes":
        return {"kind": kind, "n": rng.randint(12, 64), "d": d, "chi": _log_int(rng, 16, top),
                "bits": _log_int(rng, 64, 4096)}
    if kind == "marginals":
        return {"kind": kind, "n": rng.randint(12, 64), "d": d, "chi": _log_int(rng, 16, top)}
    return {"kind": "vector", "n": rng.randint(3, 13) if d == 2 else rng.randint(2, 9), "d": d}


# -- inputs -------------------------------------------------------------------

def _bonds(n, d, chi):
    """Bond dimensions min(chi, d^i, d^(n-i)) of a state truncated to chi."""
    out = []
    for i in range(n + 1):
        e = min(i, n - i)
        out.append(chi if e * math.log(d) > math.log(chi) + 1 else min(chi, d ** e))
    return out


def _sites(n, d, chi, seed):
    """Random sites with the norm of a state near 1: complex Gaussian entries
    of variance 1 / (chi_left d), one buffer drawn on the GPU and cut up."""
    b = _bonds(n, d, chi)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    sizes = [b[i] * d * b[i + 1] for i in range(n)]
    flat = torch.randn(sum(sizes), dtype=torch.complex64, device="cuda", generator=gen)
    out = []
    for i, t in enumerate(torch.split(flat, sizes)):
        out.append((t * (1.0 / math.sqrt(b[i] * d))).reshape(b[i], d, b[i + 1]))
    return out


def _layer_gates(case, seed):
    """Haar gates of a layer whose pairs start at site 0 or 1."""
    n, d = case["n"], case["d"]
    lefts = list(range(case["first"], n - 1, 2))
    base = 7 + 1000 * seed
    one = C.haar_batch(1, d, [(base + i) % (1 << 32) for i in range(n)])
    two = C.haar_batch(2, d, [(base + 500 + i) % (1 << 32) for i in lefts])
    return one.astype(np.complex64), lefts, two.astype(np.complex64)


def _operations(case, seed):
    circ = C.brickwork(case["n"], case["depth"], d=case["d"], seed=seed % (1 << 31))
    d = case["d"]
    return [(sites, g.astype(np.complex64).reshape((d,) * (2 * k)))
            for k, sites, g in circ.operations()]


def _bits(case, seed, n):
    return C.sample_bitstrings(n, case["d"], case["bits"], seed=seed % (1 << 31)).astype(np.int8)


def _circuits(case, seed):
    """Circuits of n - 4 .. n + 4 qudits, gates as complex64."""
    out = []
    for q in range(case["count"]):
        circ = C.brickwork(case["n"] - 4 + q % 9, case["depth"], d=case["d"],
                           maxsvals=case["maxsvals"], seed=seed % (1 << 31), instance=q)
        for lay in circ.layers:
            lay.one_q = lay.one_q.astype(np.complex64)
            lay.two_q = lay.two_q.astype(np.complex64)
        out.append(circ)
    return out


def _perturbed(sites, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed + 77)
    return [t + 0.02 * t.abs().mean() * torch.randn(t.shape, dtype=torch.complex64, device="cuda",
                                                    generator=gen) for t in sites]


def _vector(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    v = torch.randn(case["d"] ** case["n"], dtype=torch.complex64, device="cuda", generator=gen)
    return (v / v.norm()).cpu().numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "layer":
        one, lefts, two = _layer_gates(case, seed)
        mps = MPS.from_sites(_sites(case["n"], case["d"], case["chi"], seed), case["d"],
                             precision=case["precision"])
        return {"kind": kind, "mps": mps, "one": one, "lefts": lefts, "two": two,
                "chi": case["chi"], "left": case["left"]}
    if kind == "circuit":
        ops = [MPSOperation(g, sites, qudit_dimension=case["d"])
               for sites, g in _operations(case, seed)]
        return {"kind": kind, "ops": ops, "n": case["n"], "d": case["d"]}
    if kind == "plan":
        circs = _circuits(case, seed)
        return {"kind": kind, "plan": CircuitPlan(circs),
                "bits": [_bits(case, seed + q, c.nqudits) for q, c in enumerate(circs)]}
    if kind == "vector":
        return {"kind": kind, "vector": _vector(case, seed), "n": case["n"], "d": case["d"]}
    sites = _sites(case["n"], case["d"], case["chi"], seed)
    state = {"kind": kind, "mps": MPS.from_sites(sites, case["d"])}
    if kind == "overlap":
        state["other"] = MPS.from_sites(_perturbed(sites, seed), case["d"])
    elif kind == "amplitudes":
        state["bits"] = _bits(case, seed, case["n"])
    return state


# -- one pass -----------------------------------------------------------------

def _merged(sites, lefts):
    """The layer's state without the gauge of its cuts, as one vector: the merged
    tensors of the pairs (those of one shape together), and the sites outside
    every pair."""
    groups, inside = {}, set()
    for i in lefts:
        inside.update((i, i + 1))
        a, b = sites[i], sites[i + 1]
        groups.setdefault((tuple(a.shape), tuple(b.shape)), []).append(
            (a.reshape(-1, a.shape[2]), b.reshape(b.shape[0], -1)))
    out = [torch.bmm(torch.stack([a for a, _ in g]), torch.stack([b for _, b in g]))
           for g in groups.values()] + [t for i, t in enumerate(sites) if i not in inside]
    return torch.cat([t.reshape(-1) for t in out])


def run(state):
    kind = state["kind"]
    if kind == "layer":
        mps = state["mps"].copy()
        mps.apply_layer(state["one"], state["lefts"], state["two"], maxsvals=state["chi"],
                        keep_left_canonical=state["left"])
        return _merged(mps.sites, state["lefts"])
    if kind == "circuit":
        mps = MPS(state["n"], state["d"])
        mps.apply(state["ops"])
        return mps.wavefunction()
    if kind == "plan":
        plan = state["plan"]
        plan.run()
        return np.stack([plan.state(q).amplitudes(b) for q, b in enumerate(state["bits"])])
    if kind == "overlap":
        mps, other = state["mps"], state["other"]
        return np.array([mps.inner_product(mps), mps.inner_product(other)], dtype=np.complex64)
    if kind == "amplitudes":
        return state["mps"].amplitudes(state["bits"])
    if kind == "marginals":
        return state["mps"].site_marginals()
    mps = MPS.from_wavefunction(state["vector"], state["n"], state["d"])
    return mps.wavefunction()


# -- what a pass cannot do without ----------------------------------------------

def _svd_flops(m, n):
    """Complex SVD with both factors, the usual count for an m x n matrix."""
    big, small = max(m, n), min(m, n)
    return 4.0 * (14.0 * big * small ** 2 + 8.0 * small ** 3)


def _pair_work(d, cl, cm, cr, k):
    m, n = cl * d, d * cr
    flops = 8.0 * m * n * cm + 8.0 * m * n * d * d + _svd_flops(m, n)
    nbytes = 8.0 * (cl * d * cm + cm * d * cr + m * k + k * n + d ** 4)
    return nbytes, flops


def _circuit_work(n, d, depth, maxsvals):
    b = [1] * (n + 1)
    nbytes = flops = 0.0
    for t in range(depth):
        nbytes += 8.0 * n * d * d
        flops += 8.0 * sum(b[i] * b[i + 1] * d * d for i in range(n))
        for i in range(t % 2, n - 1, 2):
            k = min(b[i] * d, d * b[i + 2])
            k = k if maxsvals is None else min(k, maxsvals)
            x, f = _pair_work(d, b[i], b[i + 1], b[i + 2], k)
            nbytes, flops = nbytes + x, flops + f
            b[i + 1] = k
    return nbytes, flops, b


def _env_flops(b, d):
    return sum(8.0 * d * b[i] * b[i + 1] * (b[i] + b[i + 1]) for i in range(len(b) - 1))


def _site_bytes(b, d):
    return sum(8.0 * d * b[i] * b[i + 1] for i in range(len(b) - 1))


def work(case):
    kind, n, d = case["kind"], case["n"], case["d"]
    if kind == "layer":
        b = _bonds(n, d, case["chi"])
        nbytes = 2.0 * 8 * sum(b[i] * d * b[i + 1] for i in range(n)) + 8.0 * n * d * d
        flops = 8.0 * d * d * sum(b[i] * b[i + 1] for i in range(n))
        for i in range(case["first"], n - 1, 2):
            k = min(case["chi"], b[i] * d, d * b[i + 2])
            flops += _pair_work(d, b[i], b[i + 1], b[i + 2], k)[1]
            nbytes += 8.0 * d ** 4
        return {"bytes": nbytes, "flops": flops}
    if kind == "circuit":
        # the gates in, the wavefunction out; the state stays on the chip
        _, flops, _ = _circuit_work(n, d, case["depth"], None)
        gates = case["depth"] * (n * d * d + (n // 2) * d ** 4)
        return {"bytes": 8.0 * (gates + d ** n), "flops": flops + 8.0 * d ** (n + 1)}
    if kind == "plan":
        nbytes = flops = 0.0
        for q in range(case["count"]):
            x, f, b = _circuit_work(n - 4 + q % 9, d, case["depth"], case["maxsvals"])
            nbytes += x + _site_bytes(b, d)
            flops += f + 8.0 * case["bits"] * sum(b[i] * b[i + 1] for i in range(len(b) - 1))
        return {"bytes": nbytes, "flops": flops}
    if kind == "vector":
        # the vector in and out, and its left half's Gram matrix at the
        # middle cut (the other cuts are smaller)
        half = d ** (n // 2)
        return {"bytes": 16.0 * d ** n, "flops": _svd_flops(d ** n // half, half)}
    b = _bonds(n, d, case["chi"])
    if kind == "overlap":
        return {"bytes": 3.0 * _site_bytes(b, d), "flops": 2.0 * _env_flops(b, d)}
    if kind == "amplitudes":
        return {"bytes": _site_bytes(b, d) + case["bits"] * (n + 8.0),
                "flops": 8.0 * case["bits"] * sum(b[i] * b[i + 1] for i in range(n))}
    return {"bytes": _site_bytes(b, d) + 4.0 * n * d, "flops": 2.0 * _env_flops(b, d)}


# -- the same in 64 bits --------------------------------------------------------

def _truncated(theta, k):
    u, s, vh = np.linalg.svd(theta, full_matrices=False)
    return (u[:, :k] * s[:k]) @ vh[:k]


def _exact_layer(case, seed):
    one, lefts, two = _layer_gates(case, seed)
    d, chi = case["d"], case["chi"]
    sites = [np.einsum("ba,lar->lbr", g.astype(np.complex128), t.cpu().numpy().astype(np.complex128))
             for g, t in zip(one, _sites(case["n"], d, chi, seed))]
    groups, inside = {}, set()
    for p, i in enumerate(lefts):
        inside.update((i, i + 1))
        a, b = sites[i], sites[i + 1]
        m = np.tensordot(a, b, (2, 0))                          # l a b r
        g = two[p].astype(np.complex128).reshape(d, d, d, d)    # a' b' a b
        th = np.einsum("xyab,labr->lxyr", g, m, optimize=True)
        th = th.reshape(a.shape[0] * d, d * b.shape[2])
        k = min(chi, *th.shape)
        groups.setdefault((a.shape[0], k, b.shape[2]), []).append(_truncated(th, k))
    out = [t for g in groups.values() for t in g] + \
        [t for i, t in enumerate(sites) if i not in inside]
    return np.concatenate([t.reshape(-1) for t in out])


def _exact_circuit(case, seed):
    n, d = case["n"], case["d"]
    psi = np.zeros((d,) * n, np.complex128)
    psi[(0,) * n] = 1.0
    for sites, g in _operations(case, seed):
        k = len(sites)
        psi = np.tensordot(g.astype(np.complex128), psi, (list(range(k, 2 * k)), sites))
        psi = np.moveaxis(psi, list(range(k)), sites)
    return psi.reshape(-1)


def _amplitudes64(sites, bits):
    env = np.ones((len(bits), 1), np.complex128)
    for i, t in enumerate(sites):
        out = np.zeros((len(bits), t.shape[2]), np.complex128)
        for x in range(t.shape[1]):
            rows = bits[:, i] == x
            out[rows] = env[rows] @ t[:, x]
        env = out
    return env[:, 0]


def _exact_plan(case, seed):
    out = []
    d = case["d"]
    for q, circ in enumerate(_circuits(case, seed)):
        sites = [np.zeros((1, d, 1), np.complex128) for _ in range(circ.nqudits)]
        for t in sites:
            t[0, 0, 0] = 1.0
        for lay in circ.layers:
            sites = [np.einsum("ba,lar->lbr", g.astype(np.complex128), t)
                     for g, t in zip(lay.one_q, sites)]
            for p, i in enumerate(lay.pair_left):
                a, b = sites[i], sites[i + 1]
                g = lay.two_q[p].astype(np.complex128).reshape(d, d, d, d)
                th = np.einsum("xyab,labr->lxyr", g, np.tensordot(a, b, (2, 0)))
                cl, cr = a.shape[0], b.shape[2]
                u, s, vh = np.linalg.svd(th.reshape(cl * d, d * cr), full_matrices=False)
                k = min(case["maxsvals"], len(s))
                sites[i] = u[:, :k].reshape(cl, d, k)
                sites[i + 1] = (s[:k, None] * vh[:k]).reshape(k, d, cr)
        out.append(_amplitudes64(sites, _bits(case, seed + q, circ.nqudits)))
    return np.stack(out)


def _left_step(env, a, b):
    """E'[r, r'] = sum E[l, l'] a[l, x, r] conj(b[l', x, r'])."""
    t = np.tensordot(env, b.conj(), (1, 0))
    return np.tensordot(a, t, ((0, 1), (0, 1)))


def _exact_overlap(case, seed):
    sites = _sites(case["n"], case["d"], case["chi"], seed)
    other = _perturbed(sites, seed)
    a = [t.cpu().numpy().astype(np.complex128) for t in sites]
    b = [t.cpu().numpy().astype(np.complex128) for t in other]
    out = []
    for bra in (a, b):
        env = np.ones((1, 1), np.complex128)
        for x, y in zip(a, bra):
            env = _left_step(env, x, y)
        out.append(env[0, 0])
    return np.array(out)


def _exact_marginals(case, seed):
    a = [t.cpu().numpy().astype(np.complex128)
         for t in _sites(case["n"], case["d"], case["chi"], seed)]
    right = [np.ones((1, 1), np.complex128)]
    for t in reversed(a[1:]):
        u = np.tensordot(t, right[-1], (2, 0))                  # l x r'
        right.append(np.tensordot(u, t.conj(), ((1, 2), (1, 2))))
    right.reverse()
    left = np.ones((1, 1), np.complex128)
    out = []
    for t, r in zip(a, right):
        u = np.tensordot(left, t, (0, 0))                       # l' x r
        w = np.tensordot(u, r, (2, 0))                          # l' x r'
        out.append(np.einsum("lxr,lxr->x", w, t.conj()).real)
        left = _left_step(left, t, t)
    return np.array(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "layer":
        return _exact_layer(case, seed)
    if kind == "circuit":
        return _exact_circuit(case, seed)
    if kind == "plan":
        return _exact_plan(case, seed)
    if kind == "overlap":
        return _exact_overlap(case, seed)
    if kind == "amplitudes":
        sites = [t.cpu().numpy().astype(np.complex128)
                 for t in _sites(case["n"], case["d"], case["chi"], seed)]
        return _amplitudes64(sites, _bits(case, seed, case["n"]))
    if kind == "marginals":
        return _exact_marginals(case, seed)
    return _vector(case, seed).astype(np.complex128)
