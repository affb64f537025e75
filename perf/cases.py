"""The calls that users of this library make, at the sizes they make them.

Every case is one pass through the Python interface (xped_gb300): tensor operations on device-resident
blocks, or a whole CTMRG / simple-update step.  Sizes are those of the benchmark, the profiles and the
tests: U(1) legs with charges -2..2 and degeneracies 2..60, SU(2) legs, power-law block matrices of 16 to
1024 columns, iPEPS of D = 2..6 with chi up to 128.  Inputs are drawn on the GPU from the seed alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from xped_gb300 import CTM, Basis, SimpleUpdate, Tensor, lib
from xped_gb300.tensor import set_gemm_precision

CHARGES = (-2, -1, 0, 1, 2)
PROFILE = (1 / 3, 2 / 3, 1.0, 2 / 3, 1 / 3)  # shape of a U(1) leg's degeneracies around charge 0
PERMS = ("0,2,1,3", "2,3,0,1", "1,0,3,2", "2,0,3,1", "3,1,0,2", "1,3,0,2", "0,3,2,1")


# ----------------------------------------------------------------------------- the cases
def listed():
    return [
        # two-site operator chain on small blocks (9 sectors up to 76 wide): T1*T2, permute, truncated SVD;
        # the smallest call a user makes, where launches and latency count
        {"name": "chain", "kind": "chain", "legs": "2,4,6,4,2", "keep": 16},
        # operator* at the sector sizes of the CTM projector products (up to 616 wide), plain FP64,
        # the left operand an adjoint
        {"name": "product_fp64", "kind": "product", "legs": "6,12,16,12,6", "form": "fp64", "adj": "TN"},
        # operator* on blocks up to 2464 wide in the FP64-accurate tensor-core form
        {"name": "product_f64tc", "kind": "product", "legs": "12,24,32,24,12", "form": "f64tc", "adj": "NN"},
        # fusion-tree permute of a large U(1) tensor (1.4 GB): memory bandwidth
        {"name": "permute_u1", "kind": "permute", "sym": "U1", "legs": "20,40,60,40,20", "perm": "0,2,1,3", "shift": 0},
        # SU(2) recoupling permute (several source trees add into each output tree)
        {"name": "permute_su2", "kind": "permute", "sym": "SU2", "legs": "12,16,12,6", "perm": "2,0,3,1", "shift": 0},
        # exact truncated SVD of power-law blocks, as in the plain projector step: ragged sizes, one block
        # above 512 columns
        {"name": "tsvd_exact", "kind": "tsvd", "sizes": "24x24,61x61,134x134,210x180,347x347,560x600,90x90,17x17",
         "form": "exact", "keep": 128, "alpha": 2.0},
        # the randomized form of the same decomposition (sketch widths from the kept counts)
        {"name": "tsvd_randomized", "kind": "tsvd",
         "sizes": "24x24,61x61,134x134,347x347,821x821,1024x1024,560x600,210x180,90x90,37x37,17x17",
         "form": "randomized", "keep": 128, "alpha": 2.0},
        # left-canonicalisation of a matrix-product tensor: (bond, phys | bond) with tall blocks
        {"name": "tqr", "kind": "tqr", "legs": "40,90,128,90,40", "phys": 3},
        # reverse rules of operator* and of the per-sector SVD (gradient of a two-site contraction)
        {"name": "backward", "kind": "backward", "legs": "4,8,11,8,4"},
        # one plain FP64 CTMRG step, exact projector SVDs
        {"name": "ctm_plain", "kind": "ctm", "sym": "U1", "aux": "1,2,1", "chi": 32, "form": "plain"},
        # one CTMRG step of the chosen form at the benchmark's size
        {"name": "ctm_chosen", "kind": "ctm", "sym": "U1", "aux": "2,2,2", "chi": 128, "form": "chosen"},
        # one simple-update step (8 bond updates) of the checkerboard Heisenberg iPEPS
        {"name": "simple_update", "kind": "su", "aux": "2,2,2"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_legs(rng, lo, hi):
    peak = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return ",".join(str(max(1, min(int(hi), int(round(peak * w * rng.uniform(0.8, 1.0)))))) for w in PROFILE)


def draw(rng):
    kind = rng.choice(["chain", "product", "product", "permute", "permute", "tsvd", "tsvd", "tqr", "backward", "ctm",
                       "ctm", "su"])
    if kind == "chain":
        return {"kind": kind, "legs": _draw_legs(rng, 2, 16), "keep": _log_int(rng, 8, 64)}
    if kind == "product":
        form = rng.choice(["fp64", "f64tc"])
        return {"kind": kind, "legs": _draw_legs(rng, 3, 16 if form == "fp64" else 32), "form": form,
                "adj": rng.choice(["NN", "TN", "NT"])}
    if kind == "permute":
        sym = rng.choice(["U1", "U1", "SU2"])
        if sym == "U1":
            return {"kind": kind, "sym": sym, "legs": _draw_legs(rng, 4, 60), "perm": rng.choice(PERMS),
                    "shift": rng.choice([0, 0, 1, -1])}
        legs = ",".join(str(_log_int(rng, 2, 16)) for _ in range(4))
        return {"kind": kind, "sym": sym, "legs": legs, "perm": rng.choice(PERMS), "shift": rng.choice([0, 0, 1, -1])}
    if kind == "tsvd":
        form = rng.choice(["exact", "randomized"])
        sizes = []
        for _ in range(rng.randint(3, 10)):
            m = _log_int(rng, 16, 520 if form == "exact" else 1024)
            n = m if rng.random() < 0.6 else max(8, int(m * rng.uniform(0.6, 1.0)))
            sizes.append("%dx%d" % ((m, n) if rng.random() < 0.5 else (n, m)))
        return {"kind": kind, "sizes": ",".join(sizes), "form": form, "keep": _log_int(rng, 16, 128),
                "alpha": rng.choice([1.0, 2.0, 3.0])}
    if kind == "tqr":
        return {"kind": kind, "legs": _draw_legs(rng, 4, 128), "phys": rng.choice([2, 3])}
    if kind == "backward":
        return {"kind": kind, "legs": _draw_legs(rng, 2, 11)}
    if kind == "ctm":
        form = rng.choice(["plain", "chosen"])
        sym = rng.choice(["U1", "U1", "fZ2"])
        if sym == "U1":
            aux = rng.choice(["1,1,1", "1,2,1"]) if form == "plain" else rng.choice(["1,2,1", "1,3,1", "2,2,2"])
        else:
            aux = rng.choice(["1,1", "2,1"]) if form == "plain" else rng.choice(["2,1", "2,2", "3,2"])
        return {"kind": kind, "sym": sym, "aux": aux, "chi": _log_int(rng, 9, 30) if form == "plain" else
                _log_int(rng, 24, 112), "form": form}
    return {"kind": "su", "aux": ",".join(str(rng.randint(1, 2)) for _ in range(3))}


# ----------------------------------------------------------------------------- structure of the inputs
def _ints(s):
    return [int(x) for x in s.split(",")]


def _u1_pairs(case):
    return list(zip(CHARGES, _ints(case["legs"])))


def _aux_pairs(case):
    a = _ints(case["aux"])
    return list(zip((-1, 0, 1) if len(a) == 3 else (0, 1), a))


def _fused(l1, l2):
    """{q: [((q1, q2), offset, (d1, d2)), ...]} of two U(1) legs: fusion trees in order of (q1, q2), the row
    index of a tree running over leg 1 first."""
    out = {}
    for q1, d1 in sorted(l1):
        for q2, d2 in sorted(l2):
            rows = out.setdefault(q1 + q2, [])
            off = rows[-1][1] + rows[-1][2][0] * rows[-1][2][1] if rows else 0
            rows.append(((q1, q2), off, (d1, d2)))
    return {q: out[q] for q in sorted(out)}


def _width(rows):
    return sum(d1 * d2 for _, _, (d1, d2) in rows)


def _blocks22(pairs):
    """(rows, cols) per coupled charge of a Tensor<2,2> with four equal legs."""
    f = _fused(pairs, pairs)
    return [(_width(r), _width(r)) for r in f.values()]


def _spectrum_scales(n_sec):
    return [0.1 + 0.9 * ((5 * i + 3) % n_sec) / max(n_sec - 1, 1) for i in range(n_sec)]


def _sizes(case):
    return [tuple(int(x) for x in s.split("x")) for s in case["sizes"].split(",")]


def _kept(case):
    """Kept counts per sector of the power-law spectra (known by construction)."""
    sizes = _sizes(case)
    vals = []
    for i, ((m, n), c) in enumerate(zip(sizes, _spectrum_scales(len(sizes)))):
        vals += [(-c * (j + 1.0) ** -case["alpha"], i) for j in range(min(m, n))]
    keep = [0] * len(sizes)
    for v, i in sorted(vals)[:case["keep"]]:
        if -v >= 1e-10:
            keep[i] += 1
    return keep


# ----------------------------------------------------------------------------- data
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _normal(n, gen):
    return torch.randn(n, dtype=torch.float64, device="cuda", generator=gen)


class _Shared:
    """A tensor's device buffer for torch (kept alive by the torch tensor)."""

    def __init__(self, t):
        self.t = t
        self.__cuda_array_interface__ = {"shape": (t.size,), "typestr": "<f8", "strides": None, "version": 3,
                                         "data": (lib().xgb_tensor_device_data(t._h), False)}


def _view(t):
    return torch.as_tensor(_Shared(t), device="cuda")


def _tensor(dom, cod, flat):
    t = Tensor.zeros(dom, cod)
    lib().xgb_synchronize()
    _view(t).copy_(flat)
    torch.cuda.synchronize()
    return t


def _random(dom, cod, gen):
    t = Tensor.zeros(dom, cod)
    return _tensor(dom, cod, _normal(t.size, gen))


def _split(flat, shapes):
    """The column-major blocks of a flat buffer as matrices."""
    out, o = [], 0
    for r, c in shapes:
        out.append(flat[o:o + r * c].view(c, r).T)
        o += r * c
    return out


def _join(blocks):
    return torch.cat([b.T.reshape(-1) for b in blocks])


def _haar(n, gen):
    q, r = torch.linalg.qr(_normal(n * n, gen).view(n, n))
    return q * torch.sign(torch.diagonal(r))


def _chain_flats(case, seed):
    """T1, T2 whose legs (outer ones per charge, inner ones per coupled sector) are rotated by Haar matrices of
    the seed: other inputs with every seed, the same truncation pattern."""
    pairs = _u1_pairs(case)
    f, shapes = _fused(pairs, pairs), _blocks22(pairs)
    base, g = _gen(0), _gen(seed + 1)
    n = sum(r * c for r, c in shapes)
    flats = [_normal(n, base) for _ in range(2)]
    legs = [torch.block_diag(*[_haar(d, g) for _, d in pairs]).cpu().numpy() for _ in range(4)]
    inner = [_haar(r, g) for r, _ in shapes]
    one = _dense22(flats[0].cpu().numpy(), f, f, [pairs] * 4)[0]
    two = _dense22(flats[1].cpu().numpy(), f, f, [pairs] * 4)[0]
    one = np.einsum("xa,yb,abcd->xycd", legs[0], legs[1], one, optimize=True)
    two = np.einsum("zc,wd,abcd->abzw", legs[2], legs[3], two, optimize=True)
    outs = []
    for dense, left in ((one, False), (two, True)):
        flat = torch.from_numpy(np.concatenate([b.ravel(order="F") for b in _blocked22(dense, f, f, [pairs] * 4)])).cuda()
        blocks = [(o @ b if left else b @ o.T) for o, b in zip(inner, _split(flat, shapes))]
        outs.append(_join(blocks))
    return outs


def _rotated(t, gauges):
    """`t` with leg i rotated by gauges[i] (a Tensor<1,1> of orthogonal blocks, or None): W on a domain leg,
    its adjoint on a codomain leg, so that rotations of the two ends of a bond cancel."""
    r, c = t.rank
    for i, w in enumerate(gauges):
        if w is None:
            continue
        a1 = [1 if j == i else -(j + 1) for j in range(r + c)]
        t = t.contract(w.twist(1), a1, [-(i + 1), 1], r) if i < r else t.contract(w.adjoint(), a1, [1, -(i + 1)], r)
    return t


def _gauge(leg, gen):
    w = Tensor.zeros([leg], [leg])
    w.set_blocks({q: _haar(r, gen).cpu().numpy() for q, r in zip(*w.sectors()[:2])})
    return w


def _power_law_flat(case, seed):
    """Blocks U diag(c (i+1)^-alpha) V^T with Haar factors."""
    g = _gen(seed)
    sizes = _sizes(case)
    parts = []
    for (m, n), c in zip(sizes, _spectrum_scales(len(sizes))):
        k = min(m, n)
        u = torch.linalg.qr(_normal(m * k, g).view(m, k))[0]
        v = torch.linalg.qr(_normal(n * k, g).view(n, k))[0]
        s = c * torch.arange(1, k + 1, dtype=torch.float64, device="cuda") ** -case["alpha"]
        parts.append((u * s) @ v.T)
    return _join(parts)


def _backward_flats(case, seed):
    """A, B, dC of C = A B and the factors and cotangents of A's SVD, per sector (square blocks)."""
    g = _gen(seed)
    shapes = _blocks22(_u1_pairs(case))
    total = sum(r * c for r, c in shapes)
    a, b, dc = (_normal(total, g) for _ in range(3))
    us, ss, vs, dus, dss, dvs = [], [], [], [], [], []
    for blk in _split(a, shapes):
        u, s, vh = np.linalg.svd(blk.cpu().numpy())
        us.append(torch.from_numpy(u).cuda())
        ss.append(torch.diag(torch.from_numpy(s).cuda()))
        vs.append(torch.from_numpy(np.ascontiguousarray(vh)).cuda())
        n = blk.shape[0]
        dus.append(_normal(n * n, g).view(n, n))
        dss.append(torch.diag(_normal(n, g)))
        dvs.append(_normal(n * n, g).view(n, n))
    return a, b, dc, us, ss, vs, dus, dss, dvs


def _ctm_environment(ctm, case, seed):
    """A saturated environment of bond dimension chi: random edges and corners with decaying spectra, its bonds
    rotated by Haar matrices of the seed (another environment with the same projector spectra)."""
    sym, chi = case["sym"], case["chi"]
    base, g = _gen(1), _gen(seed + 1)
    D2 = sum(_ints(case["aux"])) ** 2
    weights = {-2: 0.1, -1: 0.22, 0: 0.36, 1: 0.22, 2: 0.1} if sym == "U1" else {0: 0.5, 1: 0.5}
    pairs = [(q, max(1, int(round(chi * w)))) for q, w in weights.items()]
    pairs = [(q, d + (chi - sum(x for _, x in pairs) if q == 0 else 0)) for q, d in pairs]
    leg = Basis.from_pairs(sym, pairs)
    decay = Tensor.zeros([leg], [leg])
    qs, rs, _ = decay.sectors()
    decay.set_blocks({q: np.diag(np.arange(1.0, r + 1.0) ** -1.0) for q, r in zip(qs, rs)})
    side = {i: _gauge(leg, g) for i in "1234"}
    env = {}
    for name, bonds in (("C1", "41"), ("C2", "12"), ("C3", "23"), ("C4", "43"), ("T1", "11"), ("T2", "22"),
                        ("T3", "33"), ("T4", "44")):
        t = ctm.get(name)
        r, c = t.rank
        legs = [t.leg(i) for i in range(r + c)]
        chis = [i for i, b in enumerate(legs) if sum(b.dims) == D2]
        for i in chis:
            legs[i] = leg.conj() if legs[i].info()[2] else leg
        t = _random(legs[:r], legs[r:], base)
        if name[0] == "C":
            t = _rotated(t, [decay, decay])
        gauges = [None] * (r + c)
        for i, b in zip(chis, bonds):
            gauges[i] = side[b]
        env[name] = _rotated(t, gauges).normalize_max()
    return env


# ----------------------------------------------------------------------------- prepare / run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "chain":
        B = Basis.from_pairs("U1", _u1_pairs(case))
        one, two = _chain_flats(case, seed)
        return dict(case, T1=_tensor([B, B], [B, B], one), T2=_tensor([B, B], [B, B], two))
    if kind == "product":
        B = Basis.from_pairs("U1", _u1_pairs(case))
        g = _gen(seed)
        return dict(case, T1=_random([B, B], [B, B], g), T2=_random([B, B], [B, B], g))
    if kind == "permute":
        legs = _ints(case["legs"])
        pairs = list(zip(CHARGES if case["sym"] == "U1" else (1, 2, 3, 4), legs))
        B = Basis.from_pairs(case["sym"], pairs)
        return dict(case, T1=_random([B, B], [B, B], _gen(seed)), p=_ints(case["perm"]))
    if kind == "tsvd":
        sizes = _sizes(case)
        left = Basis.from_pairs("U1", [(i, m) for i, (m, _) in enumerate(sizes)])
        right = Basis.from_pairs("U1", [(i, n) for i, (_, n) in enumerate(sizes)])
        widths = [min(min(s), k + max(16, -(-k // 2))) for s, k in zip(sizes, _kept(case))]
        return dict(case, T1=_tensor([left], [right], _power_law_flat(case, seed)), widths=widths)
    if kind == "tqr":
        bond = Basis.from_pairs("U1", _u1_pairs(case))
        phys = Basis.from_pairs("U1", [(-1, 1), (1, 1)] if case["phys"] == 2 else [(-1, 1), (0, 1), (1, 1)])
        return dict(case, T1=_random([bond, phys], [bond], _gen(seed)))
    if kind == "backward":
        B = Basis.from_pairs("U1", _u1_pairs(case))
        a, b, dc, us, ss, vs, dus, dss, dvs = _backward_flats(case, seed)
        st = dict(case, A=_tensor([B, B], [B, B], a), B=_tensor([B, B], [B, B], b), dC=_tensor([B, B], [B, B], dc))
        mid = Basis.from_pairs("U1", [(q, _width(r)) for q, r in _fused(_u1_pairs(case), _u1_pairs(case)).items()])
        for k, blocks in (("U", us), ("dU", dus)):
            st[k] = _tensor([B, B], [mid], _join(blocks))
        for k, blocks in (("S", ss), ("dS", dss)):
            st[k] = _tensor([mid], [mid], _join(blocks))
        for k, blocks in (("V", vs), ("dV", dvs)):
            st[k] = _tensor([mid], [B, B], _join(blocks))
        return st
    base, g = _gen(0), _gen(seed + 1)
    aux = Basis.from_pairs(case.get("sym", "U1"), _aux_pairs(case))
    if kind == "ctm":
        phys = Basis.from_pairs(case["sym"], [(-1, 1), (1, 1)] if case["sym"] == "U1" else [(0, 1), (1, 1)])
        A = _random([aux, aux], [aux, aux, phys], base)
        ctm = CTM(A, case["chi"]).init()
        env = _ctm_environment(ctm, case, seed)
        if case["form"] == "chosen":
            ctm.set_svd("randomized", power_iters=8, seed=1234, oversample=16, growth=0.5)
            ctm.set_sketch_unseen(True)
            ctm.set_gemm("f64tc")
        return dict(case, ctm=ctm, env=env, A=A)
    phys = Basis.from_pairs("U1", [(-1, 1), (1, 1)])
    U = Tensor.zeros([phys, phys], [phys, phys])
    tau = 0.05
    h = np.linalg.eigh(np.array([[-0.25, 0.5], [0.5, -0.25]]))
    mid = (h[1] * np.exp(-tau * h[0])) @ h[1].T
    e = np.exp(-0.25 * tau) * np.ones((1, 1))
    U.set_blocks({-2: e, 0: mid, 2: e})
    # site tensors with legs (left, top | right, bottom, phys); every bond rotated by a Haar matrix of the seed
    w = [_gauge(aux, g) for _ in range(4)]
    G = [_random([aux, aux], [aux, aux, phys], base) for _ in range(2)]
    G = [_rotated(G[0], [w[0], w[1], w[2], w[3], None]), _rotated(G[1], [w[2], w[3], w[0], w[1], None])]
    return dict(case, U=U, G=[t * float(1.0 + 0.1 * _normal(1, g).abs().item()) for t in G])


def run(s):
    kind = s["kind"]
    if kind == "chain":
        c = s["T1"].matmul(s["T2"])
        p = c.permute(0, [0, 2, 1, 3])
        U, S, V, tw, ent, keep = p.tSVD(s["keep"], 1e-10)
        return {"product": _view(c), "permuted": _view(p), "U": _view(U), "S": _view(S), "V": _view(V),
                "weight": tw, "entropy": ent, "keep": np.array(keep)}
    if kind == "product":
        set_gemm_precision(s["form"])
        c = s["T1"].matmul(s["T2"], adj_a=s["adj"][0] == "T", adj_b=s["adj"][1] == "T")
        set_gemm_precision("fp64")
        return _view(c)
    if kind == "permute":
        return _view(s["T1"].permute(s["shift"], s["p"]))
    if kind == "tsvd":
        if s["form"] == "exact":
            U, S, V, tw, ent, keep = s["T1"].tSVD(s["keep"], 1e-10)
        else:
            U, S, V, tw, ent, keep, _, _ = s["T1"].tSVD_randomized(s["keep"], 1e-10, s["widths"], power_iters=8, seed=7)
        return {"U": _view(U), "S": _view(S), "V": _view(V), "entropy": ent, "keep": np.array(keep)}
    if kind == "tqr":
        Q, R = s["T1"].tQR()
        return {"Q": _view(Q), "R": _view(R)}
    if kind == "backward":
        da, db = s["A"].matmul_backward(s["B"], s["dC"])
        ds = s["A"].svd_backward(s["U"], s["S"], s["V"], s["dU"], s["dS"], s["dV"])
        return {"dA": _view(da), "dB": _view(db), "dA_svd": _view(ds)}
    if kind == "ctm":
        ctm = s["ctm"]
        for k, t in s["env"].items():
            ctm.set(k, t)
        ctm.grow_all()
        return {k: _view(t) for k, t in ctm.env().items()}
    su = SimpleUpdate([[0, 1], [1, 0]], s["G"], sum(_ints(s["aux"])))
    su.step(s["U"], s["U"])
    return {"%s%d" % (k, i): _view(su.get(k, i)) for k in ("G", "wh", "wv") for i in range(2)}


# ----------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind in ("chain", "product", "backward"):
        blocks = _blocks22(_u1_pairs(case))
        size = sum(r * c for r, c in blocks)
        gemm = sum(2.0 * r * r * c for r, c in blocks)
        if kind == "product":
            return {"bytes": 24.0 * size, "flops": gemm}
        if kind == "chain":  # product, permute, and a thin SVD of each block of the permuted tensor
            return {"bytes": 8.0 * 4 * size, "flops": gemm + sum(26.0 * r * r * c for r, c in blocks)}
        return {"bytes": 8.0 * (5 + 7) * size, "flops": 7 * gemm}
    if kind == "permute":
        legs = _ints(case["legs"])
        if case["sym"] == "U1":
            size = sum(r * c for r, c in _blocks22(_u1_pairs(case)))
        else:
            rows = {}
            for j1, d1 in enumerate(legs):
                for j2, d2 in enumerate(legs):
                    for q in range(abs(j1 - j2), j1 + j2 + 1, 2):
                        rows[q] = rows.get(q, 0) + d1 * d2
            size = sum(r * r for r in rows.values())
        return {"bytes": 16.0 * size, "flops": 0.0}
    if kind == "tsvd":
        sizes = _sizes(case)
        size = sum(m * n for m, n in sizes)
        if case["form"] == "exact":  # thin R-SVD, 6 m n^2 + 20 n^3 (Golub and Van Loan)
            flops = sum(6.0 * max(s) * min(s) ** 2 + 20.0 * min(s) ** 3 for s in sizes)
        else:  # eighteen products with the sketch and the small factorisations
            flops = sum(2.0 * m * n * min(m, n, k + max(16, k // 2)) * 18 for (m, n), k in zip(sizes, _kept(case)))
        kept = _kept(case)
        return {"bytes": 8.0 * (size + sum(k * (m + n) for (m, n), k in zip(sizes, kept))), "flops": flops}
    if kind == "tqr":
        flops, size = 0.0, 0
        phys = [(-1, 1), (1, 1)] if case["phys"] == 2 else [(-1, 1), (0, 1), (1, 1)]
        rows = _fused(_u1_pairs(case), phys)
        for q, n in _u1_pairs(case):
            m = _width(rows[q]) if q in rows else 0
            k = min(m, n)
            flops += 4.0 * m * n * k
            size += 2 * m * n + n * n
        return {"bytes": 8.0 * size, "flops": flops}
    D = sum(_ints(case["aux"]))
    nq = 5.0 if case.get("sym", "U1") == "U1" else 2.0  # charges that share the blocks
    if kind == "ctm":
        chi = case["chi"]
        corner = 2.0 * (chi ** 3 * D * D * 2 + 2 * chi * chi * D ** 6 * 2) / nq
        renorm = 2.0 * (chi ** 3 * D ** 4 * 2 + 2 * chi * chi * D ** 6 * 2) / nq
        prod = 2.0 * (chi * D * D) ** 3 / nq ** 2
        n = chi * D * D
        if case["form"] == "plain":
            svd = 26.0 * n ** 3 / nq ** 2
        else:
            prod = min(prod, 4.0 * n * n * chi * 1.5 / nq)
            svd = 18 * 2.0 * n * n * chi * 1.5 / nq
        env = 4 * chi * chi + 4 * chi * chi * D * D
        return {"bytes": 8.0 * 2 * env / nq, "flops": 4 * (2 * corner + prod + svd + renorm)}
    size = 2 * D ** 4 * 2 / 3.0
    return {"bytes": 8.0 * 2 * size, "flops": 8 * (2 * 26.0 * D ** 3 * (2 * D) ** 2 + 26.0 * (2 * D * 2) ** 3) / 9.0}


# ----------------------------------------------------------------------------- the same in 64 bits without the library
def _signed(u, v):
    """The library's sign rule: r.u > 0 for the generic vector r_i = frac((i+1) * 0.7548776662466927) + 0.25."""
    y = np.arange(1, u.shape[0] + 1) * 0.7548776662466927
    r = (y - np.floor(y)) + 0.25
    for j in range(u.shape[1]):
        d = r @ u[:, j]
        if abs(d) <= 1e-8 * (r @ np.abs(u[:, j])):
            d = u[np.argmax(np.abs(u[:, j])), j]
        if d < 0:
            u[:, j] = -u[:, j]
            v[j, :] = -v[j, :]
    return u, v


def _truncated(blocks, max_keep, eps=1e-10):
    """(U, S, V flat, weight, entropy, keep) of the globally truncated blockwise SVD."""
    facs = [np.linalg.svd(b, full_matrices=False) for b in blocks]
    order = sorted(((-float(x), i, j) for i, f in enumerate(facs) for j, x in enumerate(f[1])))
    keep, ent = [0] * len(facs), 0.0
    for x, i, _ in order[:max_keep]:
        if -x >= eps:
            keep[i] += 1
            ent -= x * x * math.log(x * x)
    weight = sum(x * x for x, _, _ in order[max_keep:])
    us, ss, vs = [], [], []
    for (u, s, v), k in zip(facs, keep):
        if k:
            u, v = _signed(u[:, :k].copy(), v[:k].copy())
            us.append(u.ravel(order="F"))
            ss.append(np.diag(s[:k]).ravel(order="F"))
            vs.append(v.ravel(order="F"))
    return np.concatenate(us), np.concatenate(ss), np.concatenate(vs), weight, ent, np.array(keep)


def _dense22(flat, f_dom, f_cod, legs):
    """Dense array (a, b, c, d) of a U(1) Tensor<2,2> with the legs' charge offsets, from its flat blocks."""
    offs = []
    for leg in legs:
        o, m = 0, {}
        for q, d in sorted(leg):
            m[q] = o
            o += d
        offs.append((m, o))
    out = np.zeros([o for _, o in offs])
    pos = 0
    for q in f_dom:
        if q not in f_cod:
            continue
        r, c = _width(f_dom[q]), _width(f_cod[q])
        blk = flat[pos:pos + r * c].reshape((r, c), order="F")
        pos += r * c
        for (qa, qb), ro, (da, db) in f_dom[q]:
            for (qc, qd), co, (dc, dd) in f_cod[q]:
                sub = blk[ro:ro + da * db, co:co + dc * dd].reshape((da, db, dc, dd), order="F")
                a, b, c_, d_ = (offs[k][0][x] for k, x in enumerate((qa, qb, qc, qd)))
                out[a:a + da, b:b + db, c_:c_ + dc, d_:d_ + dd] = sub
    return out, offs


def _blocked22(dense, f_dom, f_cod, legs, sign=(1, 1, 1, 1)):
    """The blocks of a dense (dom, dom, cod, cod) array; sign[k] = -1: charge q of leg k lies where -q lay."""
    offs = []
    for leg in legs:
        o, m = 0, {}
        for q, d in sorted(leg):
            m[q] = o
            o += d
        offs.append(m)
    blocks = []
    for q in f_dom:
        if q not in f_cod:
            continue
        blk = np.zeros((_width(f_dom[q]), _width(f_cod[q])))
        for qd, ro, dd in f_dom[q]:
            for qc, co, dc in f_cod[q]:
                at = [offs[k][sign[k] * x] for k, x in enumerate(qd + qc)]
                sub = dense[tuple(slice(a, a + d) for a, d in zip(at, dd + dc))]
                blk[ro:ro + dd[0] * dd[1], co:co + dc[0] * dc[1]] = sub.reshape((dd[0] * dd[1], -1), order="F")
        blocks.append(blk)
    return blocks


def exact(case, seed):
    kind = case["kind"]
    if kind == "product":
        shapes = _blocks22(_u1_pairs(case))
        g = _gen(seed)
        n = sum(r * c for r, c in shapes)
        a, b = _split(_normal(n, g), shapes), _split(_normal(n, g), shapes)
        ta, tb = case["adj"]
        return _join([(x.T if ta == "T" else x) @ (y.T if tb == "T" else y) for x, y in zip(a, b)])
    if kind == "chain":
        pairs = _u1_pairs(case)
        f = _fused(pairs, pairs)
        shapes = _blocks22(pairs)
        prod = _join([x @ y for x, y in zip(*(_split(t, shapes) for t in _chain_flats(case, seed)))])
        prod = prod.cpu().numpy()
        dense = _dense22(prod, f, f, [pairs] * 4)[0]
        # permute<0>(0, 2, 1, 3): the second leg of each side turns around, its charges change sign
        turned = [(-q, d) for q, d in pairs]
        fd, fc = _fused(pairs, turned), _fused(turned, pairs)
        # an index of charge q on a turned leg is the one of -q before
        blocks = _blocked22(dense.transpose(0, 2, 1, 3), fd, fc, [pairs, pairs, pairs, pairs], (1, -1, -1, 1))
        U, S, V, weight, ent, keep = _truncated(blocks, case["keep"])
        return {"product": prod, "permuted": np.concatenate([b.ravel(order="F") for b in blocks]), "U": U, "S": S,
                "V": V, "weight": weight, "entropy": ent, "keep": keep}
    if kind == "tsvd" and case["form"] == "exact":
        blocks = [b.cpu().numpy() for b in _split(_power_law_flat(case, seed), _sizes(case))]
        U, S, V, _, ent, keep = _truncated(blocks, case["keep"])
        return {"U": U, "S": S, "V": V, "entropy": ent, "keep": keep}
    if kind == "tqr":
        phys = [(-1, 1), (1, 1)] if case["phys"] == 2 else [(-1, 1), (0, 1), (1, 1)]
        rows = _fused(_u1_pairs(case), phys)
        shapes = [(_width(rows[q]), n) for q, n in _u1_pairs(case) if q in rows]
        flat = _normal(sum(m * n for m, n in shapes), _gen(seed))
        qs, rs = [], []
        for b in _split(flat, shapes):
            m, n = b.shape
            q, r = np.linalg.qr(b.cpu().numpy())
            qf, rf = np.zeros((m, n)), np.zeros((n, n))
            qf[:, :q.shape[1]] = q
            rf[:r.shape[0]] = r
            qs.append(qf.ravel(order="F"))
            rs.append(rf.ravel(order="F"))
        return {"Q": np.concatenate(qs), "R": np.concatenate(rs)}
    if kind == "backward":
        shapes = _blocks22(_u1_pairs(case))
        a, b, dc, us, ss, vs, dus, dss, dvs = _backward_flats(case, seed)
        da = _join([x @ y.T for x, y in zip(_split(dc, shapes), _split(b, shapes))])
        db = _join([x.T @ y for x, y in zip(_split(a, shapes), _split(dc, shapes))])
        out = []
        for u, s, v, du, ds, dv in zip(us, ss, vs, dus, dss, dvs):
            s1 = torch.diagonal(s)
            gap = s1[None, :] ** 2 - s1[:, None] ** 2
            small = gap.abs() < 1e-12
            F = torch.where(small, gap / (gap * gap + 1e-12), 1.0 / torch.where(small, torch.ones_like(gap), gap))
            J, K = F * (u.T @ du), F * (v @ dv.T)
            eye = torch.eye(u.shape[0], dtype=torch.float64, device=u.device)
            g = u @ (ds + (J + J.T) @ s + s @ (K + K.T)) @ v
            g = g + (eye - u @ u.T) @ du @ torch.diag(1 / s1) @ v
            out.append(g + u @ torch.diag(1 / s1) @ dv @ (eye - v.T @ v))
        return {"dA": da, "dB": db, "dA_svd": _join(out)}
    # permutes move entries (SU(2): times fixed coefficients); the randomized SVD approximates by its
    # sketch; whole CTM and simple-update steps have no short restatement
    return None
