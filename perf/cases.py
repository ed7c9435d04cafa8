"""Cases of the hot path of a two-site DMRG step, for timing and comparing.

A case is one call (or the few calls a step makes in a row) of the package's
public interface, with inputs of the shapes a run of bond dimension D meets:
bond sectors 2j = 0..max2j with multiplet counts from a discretised Gaussian
summing to D, spin-1/2 sites, spin-1 operators.  Block entries decay along
their rows and columns over a few decades, as the entries of a truncated wave
function and of its environments do (multiplets are kept in ascending order of
their singular values), and the truncation's input has singular values that
fall exponentially.

Kinds of cases:
  apply    HeffPlan.apply on a plan the caller keeps (the inner loop of any
           eigensolver a user brings; the benchmark's workload)
  solve    HeffPlan + lanczos + close: the eigensolve of one step
  env      env_batch: one site update (operators carried over the site, the
           block Hamiltonian with its on-site pairing, the new site operator)
  svd      the truncation of a step
  input    prepare_input_vector: the start vector of the next step
  combine  operator_combine: a summed partner of H_eff, once per step
"""
from __future__ import annotations

import math

import numpy as np
import torch

from su2dmrg_gb300 import su2 as S
from su2dmrg_gb300.workloads import gaussian_sector_counts

F64, SPLIT, FAST = 0, 1, 2  # plain FP64, 7 digit slices, 6 digit slices


def listed():
    return [
        # the small steps near the ends of a chain and of a warm-up: latency
        {"name": "apply_f64_d40", "kind": "apply", "D": 40, "nops": 4, "mode": F64, "max2j": 6},
        # parity runs and small production runs in plain FP64, odd sizes
        {"name": "apply_f64_d251", "kind": "apply", "D": 251, "nops": 9, "mode": F64, "max2j": 12},
        # the 6x4 D = 200 configuration with the split engine
        {"name": "apply_split_d200", "kind": "apply", "D": 200, "nops": 6, "mode": SPLIT, "max2j": 10},
        # the early sweeps of a large run, at the lower of the two split precisions, odd sizes
        {"name": "apply_fast_d777", "kind": "apply", "D": 777, "nops": 11, "mode": FAST, "max2j": 12},
        # the headline step: D = 2000, 18 operator pairs and two block Hamiltonians
        {"name": "apply_split_d2000", "kind": "apply", "D": 2000, "nops": 18, "mode": SPLIT, "max2j": 12},
        # a whole eigensolve of a small step (plan, five Lanczos vectors, release) and of a middling one
        {"name": "solve_f64_d123", "kind": "solve", "D": 123, "nops": 5, "mode": F64, "max2j": 9},
        {"name": "solve_split_d600", "kind": "solve", "D": 600, "nops": 12, "mode": SPLIT, "max2j": 12},
        # site updates of a left-moving small run and of a right-moving large one
        {"name": "env_f64_d150", "kind": "env", "D": 150, "nops": 6, "mode": F64, "max2j": 9, "flag": 1},
        {"name": "env_split_d1100", "kind": "env", "D": 1100, "nops": 14, "mode": SPLIT, "max2j": 12, "flag": 0},
        # the truncation of a step of a middling run
        {"name": "svd_d400", "kind": "svd", "D": 400, "max2j": 12},
        # the start vector of the next step of a large run
        {"name": "input_split_d1500", "kind": "input", "D": 1500, "mode": SPLIT, "max2j": 12},
        # one summed partner of a large run
        {"name": "combine_d900", "kind": "combine", "D": 900, "nops": 6, "max2j": 12},
    ]


def draw(rng):
    def log_int(a, b):
        return max(a, min(b, int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))))

    kind = rng.choice(["apply", "apply", "apply", "solve", "solve", "env", "env", "svd", "input", "combine"])
    c = {"kind": kind, "max2j": rng.randint(5, 12)}
    if kind == "svd":
        c["D"] = log_int(24, 400)
    elif kind == "input":
        c["mode"] = rng.choice([F64, SPLIT])
        c["D"] = log_int(32, 1500 if c["mode"] else 800)
    elif kind == "combine":
        c["D"], c["nops"] = log_int(32, 1200), rng.randint(2, 8)
    else:
        c["mode"] = rng.choice([F64, SPLIT, SPLIT, FAST])
        most = 2000 if kind == "apply" else 900 if kind == "solve" else 1100
        c["D"] = log_int(24, most if c["mode"] else 500)
        c["nops"] = rng.randint(1, 18 if kind == "apply" else 12)
        if kind == "env":
            c["flag"] = rng.randint(0, 1)
    return c


# ------------------------------------------------------------- structures
def _bond(case, direction):
    counts = gaussian_sector_counts(case["D"], case["max2j"])
    angm = [k for k in range(case["max2j"] + 1) if counts[k] > 0]
    return S.Su2Bond(direction, angm, [counts[k] for k in angm])


def _half(direction=1):
    return S.Su2Bond(direction, [1], [1])


def _fuse(b):
    """bond (x) spin 1/2 with direction -1: the enlarged leg of a step."""
    dim = {}
    for a, d in zip(b.angm, b.dim):
        for c in (a - 1, a + 1):
            if c >= 0:
                dim[c] = dim.get(c, 0) + d
    return S.Su2Bond(-1, sorted(dim), [dim[c] for c in sorted(dim)])


def _blocks(struct):
    """{(2j of each leg): (offset, shape)} of the legal blocks, leg 0 fastest
    (every leg's spin reachable from the others), and the packed length."""
    got, total = {}, 0
    n = [len(b.angm) for b in struct.bonds]
    for idx in range(int(np.prod(n))):
        key, shape = [], []
        for b, m in zip(struct.bonds, n):
            key.append(b.angm[idx % m])
            shape.append(b.dim[idx % m])
            idx //= m
        if len(key) == 2:
            legal = key[0] == key[1]
        else:
            legal = abs(key[0] - key[1]) <= key[2] <= key[0] + key[1] and sum(key) % 2 == 0
        if legal:
            got[tuple(key)] = (total, tuple(shape))
            total += int(np.prod(shape))
    return got, total


def _view(x, blk):
    """One block with an inner leg of multiplicity 1 (or none) as a matrix."""
    off, shape = blk
    r, c = shape[0], int(np.prod(shape[1:]))
    return x[off: off + r * c].view(c, r).t()


def _mat(x, blk, flag):
    """An MPS block as (bond x new bond); the physical leg has one multiplet."""
    off, shape = blk
    r, c = shape[flag], shape[2]
    return x[off: off + r * c].view(c, r).t()


def _ramp(n, decades, dev):
    return torch.logspace(-decades, 0.0, n, dtype=torch.float64, device=dev) if n > 1 else \
        torch.ones(n, dtype=torch.float64, device=dev)


class _Random:
    def __init__(self, seed):
        self.dev = torch.device("cuda")
        self.g = torch.Generator(device=self.dev)
        self.g.manual_seed(seed)

    def normal(self, n):
        return torch.randn(n, generator=self.g, dtype=torch.float64, device=self.dev)

    def tensor(self, struct, rows=0.0, cols=0.0, norm=True):
        """Normal entries, every block over sqrt(rows) and falling over
        `rows` and `cols` decades towards its first row and column."""
        blks, total = _blocks(struct)
        x = self.normal(total)
        for key, (off, shape) in blks.items():
            m = _view(x, (off, shape))
            f = 1.0 / math.sqrt(max(shape)) if norm else 1.0
            if rows or cols:
                m *= f * _ramp(m.shape[0], rows, self.dev)[:, None] * _ramp(m.shape[1], cols, self.dev)[None, :]
            else:
                m *= f
        return x


def _symmetric(rnd, struct, blks, scale_back):
    """Operator data that makes H_eff symmetric: the block (j', s, j) is the
    transpose of (j, s, j'), on the right-hand operator times the inverse
    ratio of the two recoupling factors."""
    x = rnd.tensor(struct)
    for key, blk in blks.items():
        a, c = key[0], key[-1]
        if a > c:
            continue
        m = _view(x, blk)
        if a == c:
            m.copy_(0.5 * (m + m.t()))
        else:
            back = (c,) + key[1:-1] + (a,)
            if back in blks:
                _view(x, blks[back]).copy_(m.t() * ((c + 1) / (a + 1) if scale_back else 1.0))
    return x


# ---------------------------------------------------------------- prepare
def _prepare_heff(case, rnd):
    enl = _fuse(_bond(case, 1))
    inb = enl.inverted()
    psi = S.Su2Struct([enl, enl], 0).with_legal_flags()
    x = rnd.tensor(psi, 1.5, 1.5, norm=False)
    x /= x.norm()
    spin = S.Su2Bond(1, [2], [1])
    op = S.Su2Struct([inb, spin, enl], 0).with_legal_flags()
    oblk, _ = _blocks(op)
    hs = S.Su2Struct([inb, enl], 0).with_legal_flags()
    hblk, _ = _blocks(hs)
    terms = []
    for t in range(case["nops"]):
        terms.append((op, _symmetric(rnd, op, oblk, False), op, _symmetric(rnd, op, oblk, True), (0.5, 1.0, -0.75)[t % 3]))
    hl = (hs, _symmetric(rnd, hs, hblk, False), 1.0)
    hr = (hs, _symmetric(rnd, hs, hblk, False), 1.0)
    return psi, x, terms, hl, hr


def _sigma():
    s = S.Su2Struct([S.Su2Bond(-1, [1], [1]), S.Su2Bond(-1, [2], [1]), S.Su2Bond(1, [1], [1])], 0)
    return s.with_legal_flags()


def _env_parts(case, rnd):
    flag = case["flag"]
    a, c = _bond(case, 1), _bond(case, -1)
    legs = [a, _half(), c] if flag == 0 else [_half(), a, c]
    uu = S.Su2Struct(legs, 0).with_legal_flags()
    ublk, total = _blocks(uu)
    xu = rnd.normal(total)
    for blk in ublk.values():
        m = _mat(xu, blk, flag)
        m *= 1.0 / math.sqrt(max(m.shape))
    op = S.Su2Struct([a.inverted(), S.Su2Bond(-1, [2], [1]), a], 0).with_legal_flags()
    hs = S.Su2Struct([a.inverted(), a], 0).with_legal_flags()
    ops = [rnd.tensor(op, 1.0, 1.0) for _ in range(case["nops"])]
    return uu, xu, op, ops, hs, rnd.tensor(hs, 1.0, 1.0)


def _mps_pair(case, rnd):
    """Left and right MPS tensors of a step sharing their last leg."""
    a, c = _bond(case, 1), _bond(case, -1)
    out = []
    for legs in ([a, _half(), c], [_half(), a, c]):
        s = S.Su2Struct(legs, 0).with_legal_flags()
        blks, total = _blocks(s)
        x = rnd.normal(total)
        for blk in blks.values():
            m = _mat(x, blk, 1 if legs[0].angm == [1] else 0)
            m *= _ramp(m.shape[1], 2.0, rnd.dev)[None, :] / math.sqrt(max(m.shape))
        out.append((s, x))
    return out


def _svd_vector(case, rnd):
    """A two-site vector with singular values that fall by 2j and
    exponentially within each sector (16 digits over the whole sector)."""
    enl = _fuse(_bond(case, 1))
    psi = S.Su2Struct([enl, enl], 0).with_legal_flags()
    blks, total = _blocks(psi)
    x = torch.empty(total, dtype=torch.float64, device=rnd.dev)
    for (j, _), (off, (n, _)) in blks.items():
        q, _ = torch.linalg.qr(rnd.normal(n * n).view(n, n))
        p, _ = torch.linalg.qr(rnd.normal(n * n).view(n, n))
        k = torch.arange(n, dtype=torch.float64, device=rnd.dev) + 0.6 * (0.618 * (j + 1) % 1.0)  # no ties between sectors
        s = torch.exp(-0.25 * abs(j - 4) - 18.0 * k / max(n, 8))
        _view(x, blks[(j, j)]).copy_((q * s[None, :]) @ p.t())
    return psi, x / x.norm()


def prepare(case, seed):
    rnd = _Random(seed)
    kind = case["kind"]
    if kind in ("apply", "solve"):
        psi, x, terms, hl, hr = _prepare_heff(case, rnd)
        st = {"case": case, "psi": psi, "x": x, "terms": terms, "hl": hl, "hr": hr}
        torch.cuda.synchronize()  # a plan reads its operators on its own stream
        if kind == "apply":
            st["plan"] = S.HeffPlan(psi, terms, hl, hr, mode=case["mode"])
            st["y"] = torch.empty_like(x)
        return st
    if kind == "env":
        uu, xu, op, ops, hs, xh = _env_parts(case, rnd)
        sg = _sigma()
        jobs = [{"kind": "transform", "slot": t, "x": (op, x)} for t, x in enumerate(ops)]
        n = case["nops"]
        jobs.append({"kind": "init", "slot": n, "site1": (sg, np.array([math.sqrt(0.75)]))})
        jobs.append({"kind": "overlap", "slot": n + 1, "x": (hs, xh)})
        for t in range(min(n, 3)):
            jobs.append({"kind": "pair", "slot": n + 1, "coef": 0.5 + t, "x": (op, ops[t]),
                         "site1": (sg, np.array([-math.sqrt(0.75)]))})
        return {"case": case, "uu": uu, "xu": xu, "jobs": jobs}
    if kind == "svd":
        psi, x = _svd_vector(case, rnd)
        b = _bond(case, 1)
        tu = S.Su2Struct([b, _half(), _bond(case, -1)], 0)
        tv = S.Su2Struct([b, _half(), _bond(case, -1)], 0)
        return {"case": case, "psi": psi, "x": x, "tu": tu, "tv": tv}
    if kind == "input":
        (sl, xl), (sr, xr) = _mps_pair(case, rnd)
        return {"case": case, "sl": sl, "xl": xl, "sr": sr, "xr": xr}
    b = _bond(case, 1)
    op = S.Su2Struct([b.inverted(), S.Su2Bond(1, [2], [1]), b], 0).with_legal_flags()
    return {"case": case, "ops": [(op, rnd.tensor(op, 1.0, 1.0)) for _ in range(case["nops"])], "coefs": _coefs(case)}


def _coefs(case):
    return [(-1.0) ** t * (1.0 + 0.5 * t) for t in range(case["nops"])]


# -------------------------------------------------------------------- run
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "apply":
        st["plan"].apply(st["x"], st["y"])
        return st["y"]
    if kind == "solve":
        x = st["x"].clone()
        plan = S.HeffPlan(st["psi"], st["terms"], st["hl"], st["hr"], mode=case["mode"])
        e, n = plan.lanczos(x)
        plan.close()
        return {"energy": e, "matvecs": n, "psi": x}
    if kind == "env":
        return [y for _, y in S.env_batch(st["uu"], st["xu"], st["uu"], st["xu"], case["flag"], st["jobs"], mode=case["mode"])]
    if kind == "svd":
        tu, xu, tv, xv, w = S.svd(st["psi"], st["x"], st["tu"], 1.0, st["tv"], 0.0, case["D"])
        return {"bond": np.array([tu.bonds[2].angm, tu.bonds[2].dim]), "tu": xu, "tv": xv, "w": w}
    if kind == "input":
        return S.prepare_input_vector(st["sl"], st["xl"], st["sr"], st["xr"], mode=case["mode"])[1]
    return S.operator_combine(st["ops"], st["coefs"])[1]


# ------------------------------------------------------------------- work
def _heff_work(case):
    enl = _fuse(_bond(case, 1))
    d = dict(zip(enl.angm, enl.dim))
    pairs = [(a, c) for a in d for c in d if abs(a - 2) <= c <= a + 2 and (a + c) % 2 == 0]
    flops = nbytes = 0.0
    for a, c in pairs:  # psi(a,a)^T L(a,c), then T^T R(a,c)
        flops += case["nops"] * (2.0 * d[a] * d[a] * d[c] + 2.0 * d[c] * d[a] * d[c])
        nbytes += case["nops"] * 2 * 8.0 * d[a] * d[c]
    for a in d:
        flops += 4.0 * d[a] ** 3
        nbytes += 2 * 8.0 * d[a] ** 2 + 2 * 8.0 * d[a] ** 2  # block Hamiltonians; vector in and out
    return {"flops": flops, "bytes": nbytes}


def work(case):
    kind = case["kind"]
    if kind == "apply":
        return _heff_work(case)
    if kind == "solve":  # five matvecs and the two eigenvector checks
        w = _heff_work(case)
        return {"flops": 7 * w["flops"], "bytes": w["bytes"]}
    b = _bond(case, 1)
    d = dict(zip(b.angm, b.dim))
    ops = [(a, c) for a in d for c in d if abs(a - 2) <= c <= a + 2 and (a + c) % 2 == 0]
    op_bytes = sum(8.0 * d[a] * d[c] for a, c in ops)
    if kind == "combine":
        return {"flops": (2.0 * case["nops"] - 1) * op_bytes / 8, "bytes": (case["nops"] + 1) * op_bytes}
    mps = [(a, c) for a in d for c in d if abs(a - c) == 1]
    mps_bytes = sum(8.0 * d[a] * d[c] for a, c in mps)
    if kind == "env":
        n = case["nops"]
        flops = 0.0
        for a, a2 in ops:
            for c in d:
                if abs(a - c) == 1:
                    flops += n * 2.0 * d[a] * d[a2] * d[c]
                    for c2 in d:
                        if abs(a2 - c2) == 1 and abs(c - c2) <= 2 <= c + c2:
                            flops += n * 2.0 * d[a2] * d[c] * d[c2]
        for a, c in mps:  # block Hamiltonian: X^T U, then T^T V; the pairs share their T
            flops += 2.0 * d[a] * d[a] * d[c] + 2.0 * d[a] * d[c] * d[c]
        return {"flops": flops, "bytes": 2 * n * op_bytes + mps_bytes}
    enl = dict(zip(_fuse(b).angm, _fuse(b).dim))
    vec = sum(8.0 * m * m for m in enl.values())
    if kind == "input":
        return {"flops": sum(2.0 * enl[c] ** 2 * d[c] for c in d if c in enl), "bytes": 2 * mps_bytes + vec}
    # a dense singular value decomposition with both factors: about 22 n^3
    return {"flops": sum(22.0 * m ** 3 for m in enl.values()), "bytes": vec + 2 * mps_bytes}


# ------------------------------------------------------------------ exact
_CG = {}


def _cg(j1, j2, j3):
    """Clebsch-Gordan coefficients by Racah's formula, [m1, m2, m3] ascending (spins as 2j)."""
    if (j1, j2, j3) in _CG:
        return _CG[(j1, j2, j3)]
    f = math.factorial
    out = np.zeros((j1 + 1, j2 + 1, j3 + 1))
    pre = (j3 + 1) * f((j3 + j1 - j2) // 2) * f((j3 - j1 + j2) // 2) * f((j1 + j2 - j3) // 2) / f((j1 + j2 + j3) // 2 + 1)
    for i in range(j1 + 1):
        for j in range(j2 + 1):
            m1, m2 = 2 * i - j1, 2 * j - j2
            m3 = m1 + m2
            if abs(m3) > j3:
                continue
            tot = 0
            for k in range((j1 + j2 + j3) // 2 + 1):
                den = [k, (j1 + j2 - j3) // 2 - k, (j1 - m1) // 2 - k, (j2 + m2) // 2 - k, (j3 - j2 + m1) // 2 + k, (j3 - j1 - m2) // 2 + k]
                if min(den) >= 0:
                    tot += (-1) ** k / math.prod(f(v) for v in den)
            sq = math.prod(f(v) for v in ((j3 + m3) // 2, (j3 - m3) // 2, (j1 + m1) // 2, (j1 - m1) // 2, (j2 + m2) // 2, (j2 - m2) // 2))
            out[i, j, (m3 + j3) // 2] = math.sqrt(pre) * math.sqrt(sq) * tot
    _CG[(j1, j2, j3)] = out
    return out


def _ratio(t, ref):
    pos = np.unravel_index(np.argmax(np.abs(ref)), ref.shape)
    return float(t[pos] / ref[pos])


def _heff_exact(psi, terms, hl, hr):
    """x -> H x as dense products per sector; the recoupling factor of a
    spin-1 block (j, 2, j') is sqrt((j' + 1) / (j + 1)) in doubled spins."""
    pblk, _ = _blocks(psi)
    oblk, _ = _blocks(terms[0][0])
    hblk, _ = _blocks(hl[0])

    def apply(x):
        y = torch.zeros_like(x)
        for key, blk in pblk.items():
            p, out = _view(x, blk), _view(y, blk)
            out += hl[2] * (_view(hl[1], hblk[key]).t() @ p)
            out += hr[2] * (p @ _view(hr[1], hblk[key]))
        for (_, xl, _, xr, coef) in terms:
            for (a, s, c), blk in oblk.items():
                if (c, c) in pblk:
                    f = coef * math.sqrt((c + 1) / (a + 1))
                    out = _view(y, pblk[(c, c)])
                    out += f * (_view(xl, blk).t() @ (_view(x, pblk[(a, a)]) @ _view(xr, blk)))
        return y

    return apply


def _lanczos_exact(apply, x, mlanc=5):
    """Lanczos with full reorthogonalisation, the ground vector of the
    tridiagonal matrix formed at step mlanc (or at step 4 if converged)."""
    def ground(al, be):
        w, z = np.linalg.eigh(np.diag(al) + np.diag(be, 1) + np.diag(be, -1))
        v = z[:, 0]
        first = v[np.argmax(np.abs(v) > 1e-4 * np.abs(v).max())]
        return float(w[0]), v if first > 0 else -v

    ff, al, be, n = [x / x.norm()], [], [], 0
    for m in range(1, mlanc + 1):
        w = apply(ff[m - 1])
        n += 1
        al.append(float(ff[m - 1] @ w))
        if m == mlanc:
            break
        w = w - al[-1] * ff[m - 1]
        if m >= 2:
            w = w - be[-1] * ff[m - 2]
            for v in ff:
                w = w - float(w @ v) * v
        be.append(float(w.norm()))
        ff.append(w / be[-1])
        if m >= 2 and m % 4 == 0:
            e, z = ground(al, be[:-1])
            v = sum(float(z[k]) * ff[k] for k in range(m))
            v = v / v.norm()
            hv = apply(v)
            n += 1
            if abs(abs(float(hv @ v) / float(hv.norm())) - 1) < 1e-8:
                return e, n, v
    e, z = ground(al, be)
    v = sum(float(z[k]) * ff[k] for k in range(mlanc))
    return e, n + 1, v / v.norm()


def _env_exact(case, rnd):
    flag, n = case["flag"], case["nops"]
    uu, xu, op, ops, hs, xh = _env_parts(case, rnd)
    ublk, _ = _blocks(uu)
    oblk, _ = _blocks(op)
    hblk, _ = _blocks(hs)
    U = {((k[0], k[2]) if flag == 0 else (k[1], k[2])): _mat(xu, b, flag) for k, b in ublk.items()}
    new = uu.bonds[2]
    angm = new.angm
    tri = lambda a, s, c: abs(a - s) <= c <= a + s and (a + s + c) % 2 == 0  # noqa: E731

    def site(i, j):  # C(i, 1/2, j) with the physical leg second (left) or first (right), as [i, q, j]
        return _cg(i, 1, j) if flag == 0 else _cg(1, i, j).transpose(1, 0, 2)

    def pack(get, three):
        parts = []
        for idx in range(len(angm) ** 2):
            c, c2 = angm[idx % len(angm)], angm[idx // len(angm)]
            if (tri(c, 2, c2) if three else c == c2):
                m = get(c, c2)
                if m is not None:
                    parts.append(m.t().reshape(-1))
        return torch.cat(parts) if parts else torch.zeros(1, dtype=torch.float64, device=rnd.dev)

    carry, onsite, pairup = {}, {}, {}
    for (a, s, a2) in oblk:
        for c in angm:
            for c2 in angm:
                if (a, c) in U and (a2, c2) in U:
                    if tri(c, 2, c2):
                        t = np.einsum("iqj,imk,kql->jml", site(a, c), _cg(a, 2, a2), site(a2, c2), optimize=True)
                        carry[(a, a2, c, c2)] = _ratio(t, _cg(c, 2, c2))
                    if c == c2:
                        # C(1/2, 1, 1/2) joined with the spin-1 singlet (-1)^r / sqrt(3) on [r, 2 - r], times sqrt(3)
                        w = _cg(1, 2, 1)[:, ::-1, :] * np.array([1.0, -1.0, 1.0])[None, :, None]
                        t = np.einsum("iqj,ink,qnp,kpl->jl", site(a, c), _cg(a, 2, a2), w, site(a2, c), optimize=True)
                        pairup[(a, a2, c)] = _ratio(t, np.eye(c + 1))
    for c in angm:
        for c2 in angm:
            if tri(c, 2, c2):
                for a in uu.bonds[flag].angm:
                    if (a, c) in U and (a, c2) in U:
                        t = np.einsum("iqj,qmp,ipl->jml", site(a, c), _cg(1, 2, 1), site(a, c2), optimize=True)
                        onsite[(a, c, c2)] = _ratio(t, _cg(c, 2, c2))
    out = []
    tol = 1e-8
    for x in ops:
        def moved(c, c2):
            got = None
            for (a, s, a2), blk in oblk.items():
                f = carry.get((a, a2, c, c2), 0.0)
                if abs(f) >= tol:
                    m = f * (U[(a, c)].t() @ (_view(x, blk) @ U[(a2, c2)]))
                    got = m if got is None else got + m
            return got
        out.append(pack(moved, True))

    def placed(c, c2):
        got = None
        for a in uu.bonds[flag].angm:
            f = onsite.get((a, c, c2), 0.0)
            if abs(f) >= tol:
                m = math.sqrt(0.75) * f * (U[(a, c)].t() @ U[(a, c2)])
                got = m if got is None else got + m
        return got
    out.append(pack(placed, True))

    def block(c, c2):
        got = None
        for (a, _), blk in hblk.items():
            if (a, c) in U:
                m = U[(a, c)].t() @ (_view(xh, blk) @ U[(a, c)])
                got = m if got is None else got + m
        for t in range(min(n, 3)):
            for (a, s, a2), blk in oblk.items():
                f = pairup.get((a, a2, c), 0.0)
                if abs(f) >= tol:
                    m = -(0.5 + t) * math.sqrt(0.75) * f * (U[(a, c)].t() @ (_view(ops[t], blk) @ U[(a2, c)]))
                    got = m if got is None else got + m
        return got
    out.append(pack(block, False))
    return out


def _svd_exact(case, rnd):
    psi, x = _svd_vector(case, rnd)
    pblk, _ = _blocks(psi)
    b = _bond(case, 1)
    dec = {}
    for (j, _), blk in pblk.items():
        u, s, vt = torch.linalg.svd(_view(x, blk).cpu())
        u, s, v = u.flip(1), s.flip(0), vt.t().flip(1)  # ascending
        first = (v.abs() > 1e-4 * v.abs().max(0).values).to(torch.int8).argmax(0)
        sign = torch.sign(v[first, torch.arange(v.shape[1])])
        dec[j] = (u * sign, s, v * sign)
    every = sorted(((float(v), j) for j, (_, s, _) in dec.items() for v in s), reverse=True)
    kept = {}
    for _, j in every[: case["D"]]:
        kept[j] = kept.get(j, 0) + 1
    w = np.concatenate([dec[j][1][len(dec[j][1]) - kept.get(j, 0):].numpy() for j in sorted(dec)] +
                       [dec[j][1][: len(dec[j][1]) - kept.get(j, 0)].numpy() for j in sorted(dec)])
    new = sorted(kept)
    start = {}  # first row of (bond sector, centre sector) in the fused sector
    fill = {}
    for a, d in zip(b.angm, b.dim):
        for c in (a - 1, a + 1):
            if c >= 0:
                start[(a, c)] = fill.get(c, 0)
                fill[c] = fill.get(c, 0) + d
    sides = []
    for side in (0, 1):
        parts = []
        for j in new:
            u, s, v = dec[j]
            m = (u * s if side == 0 else v)[:, u.shape[1] - kept[j]:]
            for a, d in zip(b.angm, b.dim):
                if abs(a - j) == 1:
                    parts.append(m[start[(a, j)]: start[(a, j)] + d].t().reshape(-1))
        sides.append(torch.cat(parts))
    return {"bond": np.array([new, [kept[j] for j in new]]), "tu": sides[0], "tv": sides[1], "w": w}


def _input_exact(case, rnd):
    (sl, xl), (sr, xr) = _mps_pair(case, rnd)
    lblk, _ = _blocks(sl)
    rblk, _ = _blocks(sr)
    b = _bond(case, 1)
    enl = _fuse(b)
    parts = []
    for c in enl.angm:
        left = [_mat(xl, lblk[(a, 1, c)], 0) for a in b.angm if (a, 1, c) in lblk]
        right = [_mat(xr, rblk[(1, a, c)], 1) for a in b.angm if (1, a, c) in rblk]
        n = dict(zip(enl.angm, enl.dim))[c]
        if left and right:
            m = torch.cat(left) @ torch.cat(right).t()
        else:
            m = torch.zeros(n, n, dtype=torch.float64, device=rnd.dev)
        parts.append(m.t().reshape(-1))
    return torch.cat(parts)


def exact(case, seed):
    rnd = _Random(seed)
    kind = case["kind"]
    if kind in ("apply", "solve"):
        psi, x, terms, hl, hr = _prepare_heff(case, rnd)
        h = _heff_exact(psi, terms, hl, hr)
        if kind == "apply":
            return h(x)
        e, n, v = _lanczos_exact(h, x)
        return {"energy": e, "matvecs": n, "psi": v}
    if kind == "env":
        return _env_exact(case, rnd)
    if kind == "svd":
        return _svd_exact(case, rnd)
    if kind == "input":
        return _input_exact(case, rnd)
    st = prepare(case, seed)
    return sum(c * x for c, (_, x) in zip(st["coefs"], st["ops"]))
