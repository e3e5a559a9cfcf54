"""The timed cases: the calls in which a user of the framework spends the time of a sweep.

Every case is a dict of plain values; ``prepare`` makes a program's inputs, maps and caches
from a seed, ``run`` is one pass through the public entry points, ``exact`` the same outputs
from plain torch tensordots in complex128.  The sizes are those of the workloads that the
repository's benchmark and tests name (63- and 31-site binary trees, the 63-site chain, the
star and 4-ary trees, 64 batched one-site maps, U(1) Heisenberg blocks) and sizes between
them, odd ones among them.
"""
import itertools
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "graft.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import grafttn as G  # noqa: E402
from grafttn import blocksparse as B  # noqa: E402
from grafttn import contractions as GC  # noqa: E402
from grafttn import networks as GN  # noqa: E402

C128 = torch.complex128


# ---------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------

def listed():
    return [
        # Two-site map of the root edge of star_topology(3, 2), transverse-field Ising, FP64:
        # its bonds saturate at 4 below maxdim 32, so a pass is launches and host work.
        {"name": "h2_star_d32_fp64", "kind": "h2", "tree": "star", "D": 32, "precision": "fp64",
         "spectrum": "flat"},
        # Two-site map in the middle of a chain at an odd bond dimension, in the default FP64
        # (what dmrg2 applies when no precision is given), on a state in canonical form.
        {"name": "h2_chain_d250_fp64", "kind": "h2", "tree": "chain", "D": 250, "precision": "fp64",
         "spectrum": "decaying"},
        # The site gradient dE/d conj(A_n) = eff_h1 A_n at a degree-3 node of the 31-site
        # binary tree at bond dimension 128, FP64: the largest FP64 call of the gradients.
        {"name": "h1_bin31_d128_fp64", "kind": "h1", "tree": "binary", "D": 128, "precision": "fp64",
         "spectrum": "flat"},
        # Two-site map of a chain in the bf16x6 mode at an odd, ragged bond dimension.
        {"name": "h2_chain_d333_bf16x6", "kind": "h2", "tree": "chain", "D": 333, "precision": "bf16x6",
         "spectrum": "flat"},
        # The headline: the depth-3 -> depth-2 edge of the 63-site binary tree at bond
        # dimension 1024 in the fp16x3 mode.
        {"name": "h2_bin63_d1024_fp16x3", "kind": "h2", "tree": "binary", "D": 1024, "precision": "fp16x3",
         "spectrum": "flat"},
        # Environment update after a move of the centre, chain, default FP64, odd size.
        {"name": "env_chain_d193_fp64", "kind": "env", "tree": "chain", "D": 193, "precision": "fp64"},
        # The same at bond dimension 1024 in the FP64-grade tensor-core mode of mixed sweeps.
        {"name": "env_chain_d1024_fp64e", "kind": "env", "tree": "chain", "D": 1024, "precision": "fp64e"},
        # 64 independent one-site maps, bond dimensions 16-256, one CUDA graph.
        {"name": "batched_h1_64_bf16x6", "kind": "batched", "count": 64, "dmin": 16, "dmax": 256, "shapes": 64,
         "precision": "bf16x6"},
        # U(1) block-sparse two-site map of the same binary-tree edge at total bond
        # dimension 1024, replayed as a graph as the sweeps' eigensolver host does.
        {"name": "u1_bin63_d1024_fp16x3", "kind": "u1", "D": 1024, "precision": "fp16x3"},
        # One-site Krylov exponential of TDVP1 at an inner node of the 4-ary tree
        # (degree 5, transverse-field Ising), dz = -0.05i, bf16x6 maps.
        {"name": "expm_kary_d13_bf16x6", "kind": "expm", "tree": "kary", "D": 13, "precision": "bf16x6"},
        # One local update of dmrg2 in its defaults (FP64): merge, map build, Lanczos,
        # truncated SVD, and the merge of the split tensors.
        {"name": "dmrg2_step_chain_d96_fp64", "kind": "dmrg2", "D": 96, "sites": 16, "precision": "fp64"},
        # Pullback of the one-site map (adjoints of the site tensor and of the TTNO tensor,
        # the coupling gradients' route) at the 31-site binary tree, odd bond dimension.
        {"name": "vjp_bin31_d75_fp64", "kind": "vjp", "tree": "binary", "D": 75, "spectrum": "flat"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["h2", "h2", "h2", "h1", "h1", "env", "env", "batched", "u1", "expm", "dmrg2", "vjp"])
    spectrum = rng.choice(["flat", "decaying"])
    if kind == "h2":
        prec = rng.choice(["fp64", "fp64", "fp64e", "bf16x6", "fp16x3", "bf16x3"])
        tree = rng.choice(["star", "chain", "chain", "binary"])
        hi = {"star": 64, "chain": 400 if prec == "fp64" else 1024, "binary": 96 if prec == "fp64" else 700}[tree]
        return {"kind": kind, "tree": tree, "D": _log_int(rng, 2 if tree == "star" else 8, hi), "precision": prec,
                "spectrum": spectrum}
    if kind == "h1":
        prec = rng.choice(["fp64", "fp64", "fp64e", "bf16x6", "fp16x3"])
        tree = rng.choice(["chain", "binary"])
        hi = {"chain": 512 if prec == "fp64" else 1024, "binary": 120}[tree]
        return {"kind": kind, "tree": tree, "D": _log_int(rng, 4, hi), "precision": prec, "spectrum": spectrum}
    if kind == "env":
        prec = rng.choice(["fp64", "fp64e"])
        tree = rng.choice(["chain", "chain", "binary"])
        hi = {"chain": 400 if prec == "fp64" else 1024, "binary": 80 if prec == "fp64" else 120}[tree]
        return {"kind": kind, "tree": tree, "D": _log_int(rng, 4, hi), "precision": prec}
    if kind == "batched":
        return {"kind": kind, "count": _log_int(rng, 4, 64), "dmin": 16, "dmax": rng.randint(40, 256),
                "shapes": rng.randint(1, 10000), "precision": rng.choice(["bf16x6", "fp16x3", "fp64"])}
    if kind == "u1":
        return {"kind": kind, "D": _log_int(rng, 64, 1024), "precision": rng.choice(["fp16x3", "bf16x6"])}
    if kind == "expm":
        tree = rng.choice(["kary", "chain", "binary"])
        hi = {"kary": 14, "chain": 200, "binary": 40}[tree]
        return {"kind": kind, "tree": tree, "D": _log_int(rng, 4, hi), "precision": rng.choice(["bf16x6", "fp64"])}
    if kind == "dmrg2":
        return {"kind": kind, "D": _log_int(rng, 8, 120), "sites": rng.choice([14, 16, 20]), "precision": "fp64"}
    return {"kind": "vjp", "tree": rng.choice(["chain", "binary"]), "D": _log_int(rng, 4, 80), "spectrum": spectrum}


# ---------------------------------------------------------------------------------------
# structures: the tree, its node or edge, its bond dimensions, its operator tensors
# ---------------------------------------------------------------------------------------

def _tree(name, kind):
    """(topology, node, Hamiltonian): the node of a one-site call, the child of a two-site one."""
    if name == "star":
        t = G.star_topology(3, 2)
        return t, t.index["b1_1"], G.tfi(t, J=1.0, g=0.9)
    if name == "chain":
        t = G.mps_topology(63)
        return t, t.index["site32"], G.heisenberg(t)
    if name == "kary":
        t = G.kary_topology(4, 3)
        return t, t.index["k1_2"], G.tfi(t, J=1.0, g=0.9)
    t = G.binary_topology(5 if kind == "h2" else 4)
    return t, t.index["n3_1" if kind == "h2" else "n1_1"], G.heisenberg(t)


def _bonds(t, D, d=2):
    """Bond of every node to its parent: the saturated min(D, states of either side)."""
    below = {}
    for v in t.postorder():
        below[v] = min(1 << 40, d * math.prod(below[c] for c in t.children[v]))
    return {v: min(D, below[v], d ** min(40, t.nnodes - len(t.subtree_nodes(v, t.parent[v])))) if t.parent[v] >= 0
            else 1 for v in range(t.nnodes)}


def _h1_graph(K):
    """x (children.., phys, parent), W (children.., out, in, parent), environments (ket, op,
    bra) of the children and of the parent; the children's environments are absorbed first."""
    x = [10 + j for j in range(K)] + [1, 2]
    W = [30 + j for j in range(K)] + [-(K + 1), 1, 3]
    envs = [[10 + j, 30 + j, -(j + 1)] for j in range(K)] + [[2, 3, -(K + 2)]]
    return [x, W] + envs, [0] + [2 + j for j in range(K)] + [1, 2 + K]


def _h2_graph(Kn, Km, k):
    pos = [Kn + 1 + (j if j < k else j - 1) for j in range(Km)]
    last = Kn + Km + 1
    x = [10 + j for j in range(Kn)] + [1] + [50 + j for j in range(Km) if j != k] + [2, 3]
    Wn = [30 + j for j in range(Kn)] + [-(Kn + 1), 1, 4]
    Wm = [4 if j == k else 70 + j for j in range(Km)] + [-last, 2, 5]
    envs = [[10 + j, 30 + j, -(j + 1)] for j in range(Kn)]
    envs += [[50 + j, 70 + j, -(pos[j] + 1)] for j in range(Km) if j != k]
    envs.append([3, 5, -(last + 1)])
    n1, n2 = 3 + Kn, 3 + Kn + Km - 1
    return [x, Wn, Wm] + envs, [0] + list(range(3, n1)) + [1] + list(range(n1, n2)) + [2, n2]


def _env_graph(K):
    """A, environments of the children, W, conj(A); the parent's legs open (ket, op, bra)."""
    A = [10 + j for j in range(K)] + [1, -1]
    W = [30 + j for j in range(K)] + [2, 1, -2]
    bra = [50 + j for j in range(K)] + [2, -3]
    return [A] + [[10 + j, 30 + j, 50 + j] for j in range(K)] + [W, bra]


def _structure(case):
    """(x shape, labels, order, operator tensors on the host, environment bonds, W's bond)."""
    kind = "h2" if case["kind"] == "h2" else "h1"
    t, n, H = _tree(case["tree"], kind)
    bond = _bonds(t, case["D"])
    Ws = G.ttno_tensors(H)
    if kind == "h1":
        legs = [bond[c] for c in t.children[n]] + [bond[n]]
        shape = tuple(legs[:-1]) + (2, legs[-1])
        labels, order = _h1_graph(t.nchildren(n))
        return shape, labels, order, [Ws[n]], legs, False
    m = t.parent[n]
    k = t.childslot(m, n)
    root = t.parent[m] < 0
    legs = [bond[c] for c in t.children[n]] + [bond[c] for c in t.children[m] if c != n] + ([] if root else [bond[m]])
    shape = tuple([bond[c] for c in t.children[n]] + [2] + [bond[c] for c in t.children[m] if c != n] + [2, bond[m]])
    labels, order = _h2_graph(t.nchildren(n), t.nchildren(m), k)
    return shape, labels, order, [Ws[n], Ws[m]], legs, root


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------

def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + salt)
    return g


def _randn(g, shape):
    re_im = torch.randn(tuple(shape) + (2,), generator=g, device="cuda", dtype=torch.float64)
    return torch.view_as_complex(re_im.mul_(math.sqrt(0.5)))


def _environment(g, D, w):
    """Hermitian in (ket, bra) for every operator index, as a converged environment is."""
    e = _randn(g, (D, w, D)) / math.sqrt(D)
    return ((e + e.conj().permute(2, 1, 0)) / 2).resolve_conj().contiguous()


def _state(g, shape, spectrum):
    """A normalised centre tensor; "decaying": Schmidt weights 1 ... 1e-4 on every bond leg."""
    x = _randn(g, shape)
    if spectrum == "decaying":
        for j, s in enumerate(shape):
            if s > 2:
                wgt = torch.logspace(0, -4, s, dtype=torch.float64, device="cuda")
                x = x * wgt.view([-1 if i == j else 1 for i in range(len(shape))])
    return (x / torch.linalg.vector_norm(x)).contiguous()


def _map_inputs(case, seed):
    shape, labels, order, Ws, legs, root = _structure(case)
    g = _gen(seed)
    statics = [torch.from_numpy(np.ascontiguousarray(W, dtype=np.complex128)).cuda() for W in Ws]
    statics += [_environment(g, D, Ws[0].shape[0]) for D in legs]
    if root:
        statics.append(torch.ones((1, 1, 1), dtype=C128, device="cuda"))
    x = _state(g, shape, case.get("spectrum", "flat"))
    return shape, labels, order, statics, x


def _env_inputs(case, seed):
    """A_u isometric towards its parent, W_u, and the children's environments."""
    t, n, H = _tree(case["tree"], "h1")
    bond = _bonds(t, case["D"])
    g = _gen(seed, 1)
    legs = [bond[c] for c in t.children[n]]
    A = _randn(g, tuple(legs) + (2, bond[n]))
    q, _ = torch.linalg.qr(A.reshape(-1, bond[n]))
    A = q.reshape(tuple(legs) + (2, q.shape[1])).contiguous()
    W = G.ttno_tensors(H)[n]
    envs = [_environment(g, D, W.shape[0]) for D in legs]
    W = torch.from_numpy(np.ascontiguousarray(W, dtype=np.complex128)).cuda()
    K = len(legs)
    return [A] + envs + [W, A], _env_graph(K), [False] * (K + 2) + [True], list(range(K + 3))


def _batch_shapes(case):
    """Chain nodes with two bonds and tree nodes with three bonds of at most 48, in turn."""
    r = random.Random(case["shapes"])
    out = []
    for i in range(case["count"]):
        hi = case["dmax"] if i % 2 == 0 else min(case["dmax"], 48)
        out.append([r.randint(case["dmin"], hi) for _ in range(2 if i % 2 == 0 else 3)])
    return out


def _batch_inputs(case, seed):
    g = _gen(seed, 2)
    out = []
    for dims in _batch_shapes(case):
        K = len(dims) - 1
        labels, order = _h1_graph(K)
        statics = [_randn(g, (5,) * K + (2, 2, 5))] + [_environment(g, D, 5) for D in dims]
        x = _state(g, tuple(dims[:-1]) + (2, dims[-1]), "flat")
        out.append((labels, order, statics, x))
    return out


_PHYS = {0: 1, 1: 1}


def _u1_structure(case):
    """Legs of every operand of the two-site map of the depth-3 -> depth-2 edge of the 63-site
    binary tree, Sz-conserving Heisenberg; charges count up spins."""
    t = G.binary_topology(5)
    n = t.index["n3_1"]
    m = t.parent[n]
    H = G.NNHamiltonian(t)
    for e in t.edges():
        H.bonds[e] = list(B.u1_heisenberg_terms())
    Ws = G.ttno_tensors(H)
    out_leg, perm = B.op_leg(+1)
    in_leg, _ = B.op_leg(-1)

    def sectors(c):
        return B.binomial_sectors(len(t.subtree_nodes(c, t.parent[c])), case["D"])
    labels, order = _h2_graph(2, 2, t.childslot(m, n))
    others = [c for c in t.children[m] if c != n]
    xlegs = [B.U1Leg(sectors(c), 1) for c in t.children[n]] + [B.U1Leg(_PHYS, 1)]
    xlegs += [B.U1Leg(sectors(c), 1) for c in others] + [B.U1Leg(_PHYS, 1), B.U1Leg(sectors(m), -1)]
    operands = []
    for u in (n, m):
        W = Ws[u]
        for ax in (0, 1, 4):
            W = np.take(W, perm, axis=ax)
        operands.append(([out_leg, out_leg, B.U1Leg(_PHYS, 1), B.U1Leg(_PHYS, -1), in_leg], np.ascontiguousarray(W)))
    for c in list(t.children[n]) + others:
        operands.append(([B.U1Leg(sectors(c), -1), in_leg, B.U1Leg(sectors(c), 1)], None))
    operands.append(([B.U1Leg(sectors(m), 1), out_leg, B.U1Leg(sectors(m), -1)], None))
    return xlegs, labels, order, operands


def _u1_inputs(case, seed):
    xlegs, labels, order, operands = _u1_structure(case)
    rng = np.random.default_rng(seed)
    statics = []
    for (legs, W), lab in zip(operands, labels[1:]):
        T = B.BlockTensor(legs)
        statics.append((T, lab, T.from_dense(W) if W is not None else T.random(rng) / math.sqrt(legs[0].total)))
    xs = B.BlockTensor(xlegs)
    x = xs.random(rng)
    return xs, labels, order, statics, x / np.linalg.norm(x)


def _dmrg_state(case, seed):
    t = G.mps_topology(case["sites"])
    ctx = G.default_context()
    psi = GN.random_ttns(np.random.default_rng(seed), t, 2, _bonds(t, case["D"]), ctx=ctx)
    n = t.index["site%d" % (case["sites"] // 2)]
    G.move_center(psi, n)
    psi.tensors[n] = _decayed(ctx, psi.tensors[n])
    H = G.TTNO.from_hamiltonian(G.heisenberg(t), ctx)
    cache = GC.EnvCache(t)
    m = t.parent[n]
    for u, v in [(w, n) for w in t.neighbors(n) if w != m] + [(w, m) for w in t.neighbors(m) if w != n]:
        cache.env(psi, H, u, v)
    return psi, H, cache, n, m


def _decayed(ctx, A):
    """The centre tensor with Schmidt weights on its parent bond, normalised."""
    wgt = torch.logspace(0, -5, A.shape[-1], dtype=torch.float64, device="cuda")
    A = A * wgt
    return (A / torch.linalg.vector_norm(A)).contiguous()


# ---------------------------------------------------------------------------------------
# prepare, run
# ---------------------------------------------------------------------------------------

def prepare(case, seed):
    ctx = G.default_context()
    kind = case["kind"]
    s = {"kind": kind, "ctx": ctx}
    if kind in ("h1", "h2", "expm", "vjp"):
        shape, labels, order, statics, x = _map_inputs(case, seed)
        order = GC.choose_order([shape] + [tuple(a.shape) for a in statics], labels, order)
        s["x"] = x
        s["map"] = GC.EffectiveMap(ctx, shape, labels, order, statics, case.get("precision", "fp64"))
        if kind == "vjp":
            s["ybar"] = _state(_gen(seed, 3), shape, "flat")
    elif kind == "env":
        ops, labels, conj, order = _env_inputs(case, seed)
        order = GC.choose_order([tuple(o.shape) for o in ops], labels, order)
        s.update(ops=ops, labels=labels, conj=conj, order=order, precision=G._lib.PRECISIONS[case["precision"]])
    elif kind == "batched":
        items = _batch_inputs(case, seed)
        s["maps"] = [GC.EffectiveMap(ctx, x.shape, labels, order, statics, case["precision"])
                     for labels, order, statics, x in items]
        s["xs"] = [x for _, _, _, x in items]
        s["ys"] = [ctx.empty(m.y_shape) for m in s["maps"]]
        s["batch"] = GC.MapBatch(s["maps"], s["xs"], s["ys"], graph=True)
    elif kind == "u1":
        xs, labels, order, statics, x = _u1_inputs(case, seed)
        plan = B.BlockPlan(xs, labels[0], statics, order)
        s["map"] = B.BlockEffectiveMap(ctx, plan, case["precision"], graph=True)
        s["x"] = ctx.upload(x)
        s["y"] = ctx.empty((plan.y.size,))
    else:
        psi, H, cache, n, m = _dmrg_state(case, seed)
        s.update(psi=psi, H=H, cache=cache, n=n, m=m, trunc=GN.TruncationScheme(maxdim=case["D"]))
        s["precision"] = G._lib.PRECISIONS[case["precision"]]
    return s


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind in ("h1", "h2"):
        return s["map"](s["x"])
    if kind == "expm":
        y, _ = s["map"].exponentiate(-0.05j, s["x"], krylovdim=30, tol=1e-10)
        return y
    if kind == "vjp":
        return [s["map"].vjp(s["x"], s["ybar"], 0), s["map"].vjp(s["x"], s["ybar"], 1)]
    if kind == "env":
        return ctx.contract(s["ops"], s["labels"], s["conj"], s["order"], s["precision"])
    if kind == "batched":
        return s["batch"].run()
    if kind == "u1":
        return s["map"].apply_into(s["x"], s["y"])
    psi, n, m = s["psi"], s["n"], s["m"]
    psi = GN.TTNS(psi.topo, list(psi.tensors), psi.center, ctx)  # a pass leaves the state as it was
    theta = GN.two_site_tensor(psi, n, m)
    h2 = GC.eff_h2(s["cache"], psi, s["H"], n, m, s["precision"])
    E, v, _ = h2.lanczos_min(theta, krylovdim=20, tol=1e-10, maxiter=2)
    h2.close()
    discarded = GN.split_two_site(psi, v, n, m, s["trunc"], "m")
    return {"energy": E, "discarded": discarded, "theta": GN.two_site_tensor(psi, n, m)}


# ---------------------------------------------------------------------------------------
# work, exact
# ---------------------------------------------------------------------------------------

def _chain_work(shapes, labels, order):
    """(complex multiply-adds, output elements) of the pairwise chain in this order."""
    dims = {}
    for shp, lab in zip(shapes, labels):
        dims.update(zip(lab, shp))
    cur, macs = list(labels[order[0]]), 0
    for j in order[1:]:
        shared = [l for l in cur if l > 0 and l in labels[j]]
        free_t = [l for l in cur if l not in shared]
        free_s = [l for l in labels[j] if l not in shared]
        macs += math.prod(dims[l] for l in free_t + shared + free_s)
        cur = free_s + free_t
    return macs, math.prod(dims[l] for l in cur)


def _map_work(shape, labels, order, Ws, legs, root):
    w = Ws[0].shape[0]
    shapes = [shape] + [W.shape for W in Ws] + [(D, w, D) for D in legs] + ([(1, 1, 1)] if root else [])
    order = GC.choose_order(shapes, labels, order)
    macs, out = _chain_work(shapes, labels, order)
    return macs, sum(math.prod(p) for p in shapes) + out


def work(case):
    kind = case["kind"]
    if kind in ("h1", "h2", "expm", "vjp"):
        shape, labels, order, Ws, legs, root = _structure(case)
        macs, elems = _map_work(shape, labels, order, Ws, legs, root)
        if kind == "expm":  # a Krylov basis of about 12 vectors
            return {"bytes": 16 * (elems + 12 * math.prod(shape)), "flops": 8 * 12 * macs}
        if kind == "vjp":  # the adjoints of x and of W are chains of the same cost
            return {"bytes": 2 * 16 * elems, "flops": 2 * 8 * macs}
        return {"bytes": 16 * elems, "flops": 8 * macs}
    if kind == "env":
        t, n, H = _tree(case["tree"], "h1")
        bond = _bonds(t, case["D"])
        legs = [bond[c] for c in t.children[n]]
        W = G.ttno_tensors(H)[n].shape
        A = tuple(legs) + (2, bond[n])
        shapes = [A] + [(D, W[0], D) for D in legs] + [W, A]
        labels = _env_graph(len(legs))
        order = GC.choose_order(shapes, labels, list(range(len(shapes))))
        macs, out = _chain_work(shapes, labels, order)
        return {"bytes": 16 * (sum(math.prod(p) for p in shapes[:-1]) + out), "flops": 8 * macs}
    if kind == "batched":
        macs = elems = 0
        for dims in _batch_shapes(case):
            K = len(dims) - 1
            labels, order = _h1_graph(K)
            a, b = _map_work(tuple(dims[:-1]) + (2, dims[-1]), labels, order, [np.empty((5,) * K + (2, 2, 5))], dims,
                             False)
            macs, elems = macs + a, elems + b
        return {"bytes": 16 * elems, "flops": 8 * macs}
    if kind == "u1":
        xlegs, labels, order, operands = _u1_structure(case)
        sizes = [B.BlockTensor(legs).size for legs in [xlegs] + [legs for legs, _ in operands]]
        # per coupled charge, the dense chain restricted to the charge-conserving blocks: about
        # the share of the dense elements that the blocks hold
        shapes = [tuple(l.total for l in legs) for legs in [xlegs] + [legs for legs, _ in operands]]
        macs, _ = _chain_work(shapes, labels, order)
        share = sizes[0] / math.prod(shapes[0])
        return {"bytes": 16 * (sum(sizes) + sizes[0]), "flops": 8 * macs * share * share}
    D = _bonds(G.mps_topology(case["sites"]), case["D"])
    d = D[G.mps_topology(case["sites"]).index["site%d" % (case["sites"] // 2)]]
    x = (d, 2, 2, d)
    labels, order = _h2_graph(1, 1, 0)
    macs, elems = _map_work(x, labels, order, [np.empty((5, 2, 2, 5))] * 2, [d, d], False)
    svd = 22 * 8 * (2 * d) ** 3 / 3  # a complex SVD with both factors
    return {"bytes": 16 * (elems + 30 * math.prod(x)), "flops": 8 * 30 * macs + svd}


def _ncon(ops, labels, conj, order):
    """Pairwise chain of torch tensordots; the legs of the result in the order -1, -2, ..."""
    cur, lab = ops[order[0]], list(labels[order[0]])
    for j in order[1:]:
        b = ops[j].conj() if conj and conj[j] else ops[j]
        shared = [l for l in lab if l > 0 and l in labels[j]]
        cur = torch.tensordot(cur, b, dims=([lab.index(l) for l in shared], [labels[j].index(l) for l in shared]))
        lab = [l for l in lab if l not in shared] + [l for l in labels[j] if l not in shared]
    return cur.permute([lab.index(-(k + 1)) for k in range(len(lab))]).contiguous()


def _dense(legs, data):
    """The dense array of a block vector: the charge-conserving blocks in lexicographic order."""
    out, off = np.zeros([l.total for l in legs], dtype=np.complex128), 0
    for sl, shape in _blocks(legs):
        n = math.prod(shape)
        out[sl] = data[off: off + n].reshape(shape)
        off += n
    return out


def _blocks(legs):
    for qs in itertools.product(*[l.charges for l in legs]):
        if sum(l.sign * q for l, q in zip(legs, qs)) == 0:
            at = [l.charges.index(q) for l, q in zip(legs, qs)]
            dims = tuple(l.dims[i] for l, i in zip(legs, at))
            lo = [sum(l.dims[:i]) for l, i in zip(legs, at)]
            yield tuple(slice(a, a + d) for a, d in zip(lo, dims)), dims


def exact(case, seed):
    kind = case["kind"]
    if kind in ("h1", "h2"):
        _, labels, order, statics, x = _map_inputs(case, seed)
        return _ncon([x] + statics, labels, None, order)
    if kind == "expm":
        _, labels, order, statics, x = _map_inputs(case, seed)
        return _exp_taylor(lambda v: _ncon([v] + statics, labels, None, order), -0.05j, x)
    if kind == "vjp":
        _, labels, order, statics, x = _map_inputs(case, seed)
        ybar = _state(_gen(seed, 3), tuple(x.shape), "flat")
        return [_adjoint([x] + statics, labels, ybar, slot) for slot in (0, 1)]
    if kind == "env":
        ops, labels, conj, order = _env_inputs(case, seed)
        return _ncon(ops, labels, conj, order)
    if kind == "batched":
        return [_ncon([x] + statics, labels, None, order) for labels, order, statics, x in _batch_inputs(case, seed)]
    if kind == "u1":
        xs, labels, order, statics, x = _u1_inputs(case, seed)
        ops = [_dense(xs.legs, x)] + [_dense(T.legs, d) for T, _, d in statics]
        y = _ncon([torch.from_numpy(o).cuda() for o in ops], labels, None, order).cpu().numpy()
        return torch.from_numpy(np.concatenate([y[sl].reshape(-1) for sl, _ in _blocks(xs.legs)])).cuda()
    return None  # a solver that stops after two restarts has no value of its own


def _adjoint(ops, labels, ybar, slot):
    """The cotangent of operand `slot`: ybar contracted with the conjugates of the others."""
    to = {l: -(k + 1) for k, l in enumerate(labels[slot])}            # its legs are the result's
    ylab = [to.get(-(k + 1), 100 + k) for k in range(ybar.dim())]
    new = [[to.get(l, l) if l > 0 else 99 - l for l in lab] for lab in labels]
    chain, labs, todo = [ybar], [ylab], [j for j in range(len(ops)) if j != slot]
    while todo:  # connected operands, small ones before x
        have = {l for lab in labs for l in lab if l > 0}
        todo.sort(key=lambda j: (not have & set(new[j]), j == 0, ops[j].dim()))
        j = todo.pop(0)
        chain.append(ops[j].conj())
        labs.append(new[j])
    return _ncon(chain, labs, None, list(range(len(chain))))


def _exp_taylor(apply, dz, x):
    """exp(dz H) x: Taylor series over steps of |dz| |H| at most 1."""
    v, norm = x, 0.0
    for _ in range(12):
        v = apply(v)
        norm = float(torch.linalg.vector_norm(v))
        v = v / norm
    steps = max(1, math.ceil(1.5 * norm * abs(dz)))
    for _ in range(steps):
        term, k = x, 0
        while k < 60:
            k += 1
            term = apply(term) * (dz / steps / k)
            x = x + term
            if float(torch.linalg.vector_norm(term)) < 1e-19:
                break
    return x
