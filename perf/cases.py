"""The work that a user of chainamps_b200 has it do, as cases that can be timed.

Every case goes through the public classes of the package.  The kinds:

* ``matvec``    H_eff . theta on device vectors (``TwoVertexComponents.multiply_device``),
                the operation that an eigensolver repeats;
* ``callback``  the same on host vectors (``multiply``), as ARPACK's reverse
                communication calls it, with pinned workd slices;
* ``eigs``      the ground state of one window with its vector on the host
                (``HED``), the reference's ``TwoVertexComponents::HED`` seam;
* ``step``      a whole iDMRG growth step (``iDMRG.grow``): environment update,
                operator build, prediction, eigensolve, truncated block SVD;
* ``gradient``  dE/dJ_perp of a window (``adjoint``), the backward direction.

and the models, each with the charge structure that decides the block sizes:

* ``xxz``      spin-1/2 XXZ chain, one site per vertex, total Sz: tiny blocks;
* ``ladder``   four coupled Heisenberg chains, 16 states per vertex, total Sz:
               many ragged sectors, the folded contraction order;
* ``ising``    coupled transverse-field Ising chains cut to 64 states per
               vertex, Z2 parity: two large sectors, the canonical order;
* ``sectors``  40 bond sectors with left / right dimensions drawn
               log-uniformly, dense complex MPO of bond dimension 16.

Precisions are those of the C ABI: FP64, split TF32, split BF16.
"""
import functools

import numpy as np
import torch

import chainamps_b200 as ca
from chainamps_b200 import capi, models

PRECISION = {"fp64": capi.CMPS_FP64, "tf32": capi.CMPS_SPLIT_TF32, "bf16": capi.CMPS_SPLIT_BF16}


def listed():
    return [
        # plain iDMRG on the XXZ chain: a matvec of a few microseconds' worth of
        # work, where launches and latency count
        dict(name="matvec_xxz_100_fp64", kind="matvec", model="xxz", chi=100, precision="fp64"),
        # the ladder at the bond dimension of its runs, in the plain and in the
        # mixed-precision form that its eigensolver uses
        dict(name="matvec_ladder_512_fp64", kind="matvec", model="ladder", chi=512, width=3.5, precision="fp64"),
        dict(name="matvec_ladder_512_bf16", kind="matvec", model="ladder", chi=512, width=3.5, precision="bf16"),
        # an odd bond dimension on the way up, in the other split form
        dict(name="matvec_ladder_201_tf32", kind="matvec", model="ladder", chi=201, width=3.0, precision="tf32"),
        # coupled Ising chains, plain and mixed
        dict(name="matvec_ising_64_fp64", kind="matvec", model="ising", chi=64, precision="fp64"),
        dict(name="matvec_ising_128_bf16", kind="matvec", model="ising", chi=128, precision="bf16"),
        # charge sectors of very uneven sizes, nothing a multiple of a tile
        dict(name="matvec_sectors_96_fp64", kind="matvec", model="sectors", chi=96, precision="fp64"),
        # an ARPACK driver's MV callback on its own host arrays
        dict(name="callback_ladder_256_bf16", kind="callback", model="ladder", chi=256, width=3.5, precision="bf16"),
        # one window's ground state handed back to a host program
        dict(name="eigs_xxz_100_fp64", kind="eigs", model="xxz", chi=100, precision="fp64"),
        # the steady state of a growth run: the ladder and the Ising chains in
        # the mixed form
        dict(name="step_ladder_512_bf16", kind="step", model="ladder", chi=512, precision="bf16"),
        dict(name="step_ising_64_bf16", kind="step", model="ising", chi=64, precision="bf16"),
        # the gradient with respect to the interchain coupling
        dict(name="gradient_ladder_128", kind="gradient", model="ladder", chi=128, width=3.5, precision="fp64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    kind = rng.choice(["matvec"] * 5 + ["callback", "eigs", "step", "gradient"])
    any_precision = rng.choice(["fp64", "fp64", "bf16", "bf16", "tf32"])
    mixed = rng.choice(["fp64", "bf16"])
    if kind == "matvec":
        model = rng.choice(["xxz", "ladder", "ladder", "ising", "ising", "sectors"])
        hi = {"xxz": (16, 256), "ladder": (32, 512), "ising": (8, 128), "sectors": (16, 96)}[model]
        case = dict(kind=kind, model=model, chi=_log_int(rng, *hi), precision=any_precision)
    elif kind == "callback":
        case = dict(kind=kind, model="ladder", chi=_log_int(rng, 32, 384), precision=mixed)
    elif kind == "eigs":
        case = dict(kind=kind, model="xxz", chi=_log_int(rng, 24, 160), precision=mixed)
    elif kind == "step":
        model = rng.choice(["ladder", "ising"])
        hi = {("ladder", "bf16"): (64, 320), ("ladder", "fp64"): (64, 256), ("ising", "bf16"): (16, 56),
              ("ising", "fp64"): (16, 32)}[model, mixed]
        case = dict(kind=kind, model=model, chi=_log_int(rng, *hi), precision=mixed)
    else:
        case = dict(kind=kind, model="ladder", chi=_log_int(rng, 32, 160), precision="fp64")
    if case["model"] == "ladder" and kind != "step":
        case["width"] = round(rng.uniform(2.5, 5.0), 2)
    return case


# ---- models and inputs ------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _context():
    return ca.Context(0)


@functools.lru_cache(maxsize=None)
def _stream():
    return torch.cuda.Stream()


@functools.lru_cache(maxsize=None)
def _ising_vertex():
    """The 12-site periodic chain at g = 1.2 cut to its 64 lowest states."""
    return models.ising_chain_vertex(12, 1.2, 64)


def _mpo(model, coupling, seed=0):
    """(rules, charges, W, bq): the vertex model's MPO with its interchain
    (or rung, or z) coupling."""
    if model == "xxz":
        return models.xxz_model(1.0, coupling, 0.0)
    if model == "ladder":
        return models.ladder_model(4, 1.0, coupling)
    if model == "ising":
        ch, ops, H, _, _ = _ising_vertex()
        W, bq = models.general_hmpo(ch, (2,), H, ops, [(f"X{i}", f"X{i}", coupling) for i in range(12)])
        return (2,), ch, W, bq
    rng = np.random.default_rng([seed, 1])
    d, D = 4, 16
    W = (rng.standard_normal((d, D, d, D)) + 1j * rng.standard_normal((d, D, d, D))) / np.sqrt(2)
    return (0,), np.zeros((d, 1), np.int64), W, np.zeros((D, 1), np.int64)


COUPLING = {"xxz": 1.0, "ladder": 0.5, "ising": 0.05, "sectors": 0.0}


def _bonds(case):
    """Charges of the left and the right bond."""
    chi = case["chi"]
    if case["model"] == "ising":
        b = (np.arange(chi) % 2).reshape(-1, 1).astype(np.int64)
        return b, b
    if case["model"] == "sectors":
        rng = np.random.default_rng(20261203)
        dims = np.round(np.exp(rng.uniform(np.log(8), np.log(chi), (2, 40)))).astype(int)
        left, right = (np.repeat(np.arange(40), n).reshape(-1, 1).astype(np.int64) for n in dims)
        return left, right
    width = case.get("width", 1.7 if case["model"] == "xxz" else 3.5)
    b = models.gaussian_bond(chi, step=2, width=width)
    return b, b


def _sectors(bond):
    keys = sorted({int(q) for q in bond[:, 0]})
    return {q: np.nonzero(bond[:, 0] == q)[0] for q in keys}


def _to_env(blocks, bond, bq, right):
    """Sector blocks {(b, q): (rows a', columns a)} of an environment, q the
    charge of a, as the reference's 6-index tensor (CSC, column b + D a)."""
    chi, D = bond.shape[0], bq.shape[0]
    sec = _sectors(bond)
    count = np.zeros(chi * D, np.int64)
    for (b, q), (rows, _) in blocks.items():
        count[b + D * sec[q]] = rows.size
    colptr = np.concatenate([[0], np.cumsum(count)])
    rowind = np.zeros(colptr[-1], np.int64)
    vals = np.zeros(colptr[-1], np.complex128)
    for (b, q), (rows, v) in blocks.items():
        at = colptr[b + D * sec[q]][:, None] + np.arange(rows.size)[None, :]
        rowind[at] = rows[None, :]
        vals[at] = v.T
    I, z = ca.MPXIndexSpec, np.zeros((1, bond.shape[1]), np.int64)
    if right:
        idx = [I(False, False, bond), I(True, False, z), I(True, False, bq), I(False, False, z), I(True, False, bond),
               I(False, False, z)]
    else:
        idx = [I(False, False, z), I(True, False, bond), I(True, False, z), I(False, False, bq), I(True, False, z),
               I(False, False, bond)]
    return ca.MPXTensor(idx, 2 if right else 3, chi, D * chi, colptr, rowind, vals)


def _partner(q, mod, sec):
    q = q % mod if mod else q
    return q if q in sec else None


def _random_blocks(rng, bond, bq, mod, used):
    """Complex Gaussian blocks on every charge-consistent (b, sector)."""
    sec, out = _sectors(bond), {}
    for b in used:
        for q, cols in sec.items():
            p = _partner(int(bq[b, 0]) + q, mod, sec)
            if p is not None:
                s = (sec[p].size, cols.size)
                out[b, q] = (sec[p], (rng.standard_normal(s) + 1j * rng.standard_normal(s)) / np.sqrt(2))
    return out


def _hermitian_blocks(rng, bond, bq, used, identity, energy):
    """Blocks of a Hermitian H_eff: the identity on slot `identity`, block
    energies growing like an entanglement spectrum on slot `energy`, and on
    the coupling slots random boundary operators of norm about 0.3, conjugate
    slots (opposite charge, mirrored inside their coupling) adjoint to each
    other."""
    sec, chi, out = _sectors(bond), bond.shape[0], {}
    level = np.log1p(rng.permutation(chi)).astype(np.complex128)
    for q, e in sec.items():
        out[identity, q] = (e, np.eye(e.size, dtype=np.complex128))
        out[energy, q] = (e, np.diag(level[e]))
    slots = [b for b in used if b not in (identity, energy)]
    invol = [b for b in slots if bq[b, 0] == 0]
    n = int(bq.shape[0] - 2) // 3  # slots per coupling of the three couplings
    for b in slots:
        base = 1 + (b - 1) // n * n
        mirror = b if b in invol else next(c for c in range(base, base + n) if bq[c, 0] == -bq[b, 0])
        for q, cols in sec.items():
            p = int(bq[b, 0]) + q
            if p not in sec or (b, q) in out:
                continue
            s = (sec[p].size, cols.size)
            v = (rng.standard_normal(s) + 1j * rng.standard_normal(s)) * (0.15 / np.sqrt(max(s)))
            v = 0.5 * (v + v.conj().T) if b == mirror else v
            out[b, q] = (sec[p], v)
            if b != mirror and mirror in slots:
                out[mirror, p] = (cols, v.conj().T)
    return out


def _window(case, seed):
    """Everything that defines one H_eff: model arrays and the blocks of both
    environments.  A window whose ground state is asked for is Hermitian."""
    model = case["model"]
    rng = np.random.default_rng([seed, 2])
    rules, ch, W, bq = _mpo(model, COUPLING[model], seed)
    used_l = sorted({int(b) for b in np.nonzero(np.any(W != 0, axis=(0, 2, 3)))[0]})
    used_r = sorted({int(b) for b in np.nonzero(np.any(W != 0, axis=(0, 1, 2)))[0]})
    left, right = _bonds(case)
    if case["kind"] == "eigs":
        D = bq.shape[0]
        lb = _hermitian_blocks(rng, left, bq, used_l, D - 1, 0)
        rb = _hermitian_blocks(rng, right, bq, used_r, 0, D - 1)
    else:
        lb = _random_blocks(rng, left, bq, rules[0], used_l)
        rb = _random_blocks(rng, right, bq, rules[0], used_r)
    return dict(rules=rules, ch=ch, W=W, bq=bq, left=left, right=right, lb=lb, rb=rb)


def _operator(case, w):
    return ca.TwoVertexComponents(_context(), w["rules"], _to_env(w["lb"], w["left"], w["bq"], False),
                                  models.mpo_tensor(w["ch"], w["W"], w["bq"]),
                                  _to_env(w["rb"], w["right"], w["bq"], True), precision=PRECISION[case["precision"]])


def _vector(n, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    return torch.randn(n, dtype=torch.complex128, device="cuda", generator=g)


def _derivative(case):
    """dW/dJ: the MPO is linear in its coupling."""
    rules, ch, a, bq = _mpo(case["model"], 1.0)
    return ch, a - _mpo(case["model"], 0.0)[2], bq


# growth steps before the timed one: the bond dimension reaches chi, and the
# environments are those of a chain of a few vertices
GROWN = {"ladder": 3, "ising": 2}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        u = np.random.default_rng([seed, 3]).uniform(-0.1, 0.1)
        rules, ch, W, bq = _mpo(case["model"], COUPLING[case["model"]] * (1.0 + u))
        run_ = ca.iDMRG(_context(), rules, models.mpo_tensor(ch, W, bq), precision=PRECISION[case["precision"]],
                        tol=1e-12)
        for _ in range(GROWN[case["model"]]):
            run_.grow(case["chi"], 1e-14)
        # the driver's buffer for the kept values: the cap may be exceeded by a
        # multiplet of equal values
        return dict(kind=kind, chi=case["chi"], run=run_, values=np.zeros(2 * case["chi"] + 64))
    w = _window(case, seed)
    h = _operator(case, w)
    s = dict(kind=kind, h=h)
    if kind == "matvec":
        s["x"] = _vector(h.n, seed)
        s["y"] = torch.empty_like(s["x"])
        s["stream"] = _stream().cuda_stream
    elif kind == "callback":
        s["x"] = _vector(h.n, seed).cpu().pin_memory().numpy()
        s["y"] = torch.empty(h.n, dtype=torch.complex128).pin_memory().numpy()
    elif kind == "gradient":
        h.set_theta(_vector(h.n, seed).cpu().numpy())
        s["dW"] = models.mpo_tensor(*_derivative(case))
    torch.cuda.synchronize()
    return s


def run(state):
    kind = state["kind"]
    if kind == "matvec":
        state["h"].multiply_device(state["x"].data_ptr(), state["y"].data_ptr(), state["stream"])
        return state["y"]
    if kind == "callback":
        return state["h"].multiply(state["x"], out=state["y"])
    if kind == "eigs":
        energy, vector, _ = state["h"].HED(tol=1e-13)
        return {"energy": energy, "vector": vector}
    if kind == "step":
        row = state["run"].grow(state["chi"], 1e-14)
        state["values"][row["chi"]:] = 0.0
        state["values"][:row["chi"]] = state["run"].values()
        return {"energy": float(row["energy"]), "entropy": float(row["entropy"]), "chi": int(row["chi"]),
                "values": state["values"].copy()}
    return state["h"].adjoint(state["dW"])


# ---- what a pass cannot do without ------------------------------------------

def _count(rules, ch, W, bq, left, right):
    """(vector length, floating-point operations of one H_eff . theta applied
    one index at a time over non-zero blocks, entries of both environments)."""
    mod = rules[0]
    red = (lambda q: q % mod) if mod else (lambda q: q)
    L = {q: v.size for q, v in _sectors(left).items()}
    R = {q: v.size for q, v in _sectors(right).items()}
    sig = [int(q) for q in ch[:, 0]]
    cls = {q: sig.count(q) for q in set(sig)}
    b_q = [int(q) for q in bq[:, 0]]
    nz = np.argwhere(W != 0)
    bl, br = sorted(set(nz[:, 1].tolist())), sorted(set(nz[:, 3].tolist()))
    # non-zero MPO entries by (slot of the contracted side, charge of the contracted state)
    w1, w2 = {}, {}
    for _, b0, s, _ in nz.tolist():
        w1[b0, sig[s]] = w1.get((b0, sig[s]), 0) + 1
        w2[b0, sig[s]] = w2.get((b0, sig[s]), 0) + 1
    ms = {red(s + q) for s in cls for q in L} & {red(q - s) for s in cls for q in R}
    rows = {m: sum(n * L.get(red(m - s), 0) for s, n in cls.items()) for m in ms}
    cols = {m: sum(n * R.get(red(m + s), 0) for s, n in cls.items()) for m in ms}
    f = 0.0
    for m in ms:
        for s, n in cls.items():
            a0, a2 = L.get(red(m - s), 0), R.get(red(m + s), 0)
            for b in bl:
                f += 8.0 * n * L.get(red(m - s + b_q[b]), 0) * a0 * cols[m]
                f += 8.0 * w1.get((b, s), 0) * L.get(red(m - s + b_q[b]), 0) * cols[m] * (a0 > 0)
                f += 8.0 * w2.get((b, s), 0) * rows.get(red(m + b_q[b]), 0) * a2
            for b in br:
                f += 8.0 * n * rows[m] * a2 * R.get(red(m + s + b_q[b]), 0)
    env = sum(L[q] * L.get(red(q + b_q[b]), 0) for q in L for b in bl)
    env += sum(R[q] * R.get(red(q + b_q[b]), 0) for q in R for b in br)
    return sum(rows[m] * cols[m] for m in ms), f, env


def work(case):
    """One pass over the input vector and the environments and one over the
    output; the operations of the contraction one index at a time.  A solve
    and a step are counted with 30 applications, what a Krylov space needs
    from a good start vector, and a gradient with two."""
    rules, ch, W, bq = _mpo(case["model"], COUPLING[case["model"]])
    n, f, env = _count(rules, ch, W, bq, *_bonds(case))
    if case["kind"] in ("eigs", "step"):
        return {"bytes": 16.0 * env + 30 * 32.0 * n, "flops": 30 * f}
    if case["kind"] == "gradient":
        return {"bytes": 16.0 * (env + n), "flops": 2 * f}
    return {"bytes": 16.0 * env + 32.0 * n, "flops": f}


# ---- the same in 64 bits, dense ---------------------------------------------

class _Dense:
    """H_eff of a window on dense tensors [a2][s2][a0][s1] in torch."""

    def __init__(self, w):
        D, mod = w["bq"].shape[0], w["rules"][0]
        to = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
        self.env = []
        for blocks, bond in ((w["lb"], w["left"]), (w["rb"], w["right"])):
            sec, e = _sectors(bond), {}
            for (b, q), (rows, v) in blocks.items():
                m = e.setdefault(b, np.zeros((bond.shape[0],) * 2, np.complex128))
                m[np.ix_(rows, sec[q])] = v
            self.env.append({b: to(m) for b, m in e.items()})
        self.W = self.pieces(w["W"])
        red = (lambda q: q % mod) if mod else (lambda q: q)
        s = w["ch"][:, 0]
        row = red(w["left"][:, 0][:, None] + s[None, :])               # a0, s1
        col = red(w["right"][:, 0][:, None] - s[None, :])              # a2, s2
        self.mask = to(col[:, :, None, None] == row[None, None, :, :])
        self.D = D

    @staticmethod
    def pieces(W):
        bs = {(int(a), int(b)) for a, b in np.argwhere(np.any(W != 0, axis=(0, 2)))}
        return {k: torch.as_tensor(np.ascontiguousarray(W[:, k[0], :, k[1]]), device="cuda") for k in sorted(bs)}

    def __call__(self, x, W1=None, W2=None):
        W1, W2 = W1 or self.W, W2 or self.W
        L, R = self.env
        t = torch.zeros(self.mask.shape, dtype=torch.complex128, device="cuda")
        t[self.mask] = x
        n2, d, n0, _ = t.shape
        Y = {}
        for b0, l in L.items():
            if not any(k[0] == b0 for k in W1):
                continue
            X = torch.matmul(l, t.view(n2 * d, n0, d))
            for (p, b1), w in W1.items():
                if p == b0 and any(k[0] == b1 for k in W2):
                    y = torch.matmul(X, w.T)
                    Y[b1] = Y[b1].add_(y) if b1 in Y else y
            del X
        out = torch.zeros_like(t).view(n2, -1)
        for b2, r in R.items():
            Z = None
            for (b1, p), w in W2.items():
                if p == b2 and b1 in Y:
                    z = torch.matmul(w, Y[b1].view(n2, d, n0 * d))
                    Z = z if Z is None else Z.add_(z)
            if Z is not None:
                out += torch.matmul(r, Z.view(n2, -1))
        return out.view(t.shape)[self.mask]


def _lowest(apply, n, steps=60, rounds=40):
    """Lowest eigenpair by restarted Lanczos with full re-orthogonalisation."""
    x = _vector(n, 1)
    for _ in range(rounds):
        V = torch.zeros((steps, n), dtype=torch.complex128, device="cuda")
        T = np.zeros((steps, steps))
        V[0] = x / x.norm()
        k = steps
        for j in range(steps):
            r = apply(V[j])
            for _ in range(2):
                c = V[:j + 1].conj() @ r
                r = r - V[:j + 1].T @ c
                T[j, j] += float(c[j].real)
            b = float(r.norm())
            if j + 1 == steps or b < 1e-13:
                k = j + 1
                break
            T[j, j + 1] = T[j + 1, j] = b
            V[j + 1] = r / b
        e, u = np.linalg.eigh(T[:k, :k])
        x = V[:k].T @ torch.as_tensor(u[:, 0], dtype=torch.complex128, device="cuda")
        x /= x.norm()
        if float((apply(x) - e[0] * x).norm()) < 1e-13 * max(1.0, abs(e[0])):
            break
    top = x[int(x.abs().argmax())]
    return float(e[0]), x * (top.conj() / top.abs())


def exact(case, seed):
    if case["kind"] == "step":
        return None  # a growth run of several vertices, by another code
    w = _window(case, seed)
    h = _Dense(w)
    n = int(h.mask.sum())
    if case["kind"] == "eigs":
        energy, vector = _lowest(h, n)
        return {"energy": energy, "vector": vector}
    x = _vector(n, seed)
    if case["kind"] == "gradient":
        d = _Dense.pieces(_derivative(case)[1])
        dx = h(x, W1=d) + h(x, W2=d)
        return float((torch.vdot(x, dx) / torch.vdot(x, x)).real)
    return h(x)
