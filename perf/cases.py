"""Performance cases of the tensor backend: what is timed, on which inputs, and what it should give.

Every case goes through an entry point that a program calls: ITensor contraction, permute, sums, svd
and factorize of the Python mirror, dmrg and dmrg_batched, and the two-site H_eff matvec and
eigensolver of the C ABI (include/itg.h).  Sizes run from the few-microsecond contractions of a
chain's ends to the chi = 1024 update of the bulk.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "itensorsgpu.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import itg  # noqa: E402

_PREC = {"fp64": 0, "split": 1}


def listed():
    return [
        # one site tensor times its neighbour near the end of a chain or in a small run: launch latency
        dict(name="contract-fp64-16", kind="contract", precision="fp64", cplx=False, a=16, k=16, b=16, s=2, lead=False),
        # ComplexF64 site tensors (time evolution, complex Hamiltonians), ragged, contracted index leading
        dict(name="contract-c64-150", kind="contract", precision="fp64", cplx=True, a=150, k=131, b=143, s=2, lead=True),
        # H_eff matvec of a plain FP64 run at a moderate, odd bond dimension
        dict(name="heff-fp64-181", kind="heff", precision="fp64", chiL=181, chiR=167, d=2, w=5),
        # H_eff matvec of a cutoff-limited run (N = 100 Heisenberg at 1e-12 reaches 182-189) in the split form
        dict(name="heff-split-189", kind="heff", precision="split", chiL=189, chiR=182, d=2, w=5),
        # the headline matvec
        dict(name="heff-split-1024", kind="heff", precision="split", chiL=1024, chiR=1024, d=2, w=5),
        # one bond's eigensolve as dmrg calls it: Davidson, subspace 3, 2 restarts
        dict(name="eigsolve-split-384", kind="eigsolve", precision="split", chiL=384, chiR=377, d=2, w=5),
        # bond split of the cutoff-limited run, rectangular, truncated by its cutoff
        dict(name="factorize-378", kind="factorize", m=378, n=366, keep=186, by="cutoff", ortho="right"),
        # bond split at chi = 1024: 2048 x 2048 kept at maxdim
        dict(name="factorize-2048", kind="factorize", m=2048, n=2048, keep=1024, by="maxdim", ortho="left"),
        # FP64 SVD of a small rectangular matrix with truncation
        dict(name="svd-fp64-150", kind="svd", m=150, n=120, keep=64),
        # a large rank-4 tensor brought into another index order (HBM-bound), odd sizes
        dict(name="permute-rank4", kind="permute", d0=129, d1=250, d2=64, d3=63, order=3, add=False),
        # a whole small run: critical-type transverse-field chain, FP64
        dict(name="dmrg-n20", kind="dmrg", N=20, maxdim=24, sweeps=2, seed=11),
        # many small disordered chains in lockstep, each with its own bond dimension
        dict(name="batched-16x10", kind="batched", count=16, N=10, maxdim=24, sweeps=2),
    ]


def _logint(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["contract", "contract", "heff", "heff", "eigsolve", "factorize", "factorize", "svd",
                       "permute", "permute", "dmrg", "batched"])
    if kind == "contract":
        p = rng.choice(["fp64", "split"])
        hi = 320 if p == "fp64" else 700
        return dict(kind=kind, precision=p, cplx=rng.random() < 0.3, a=_logint(rng, 8, hi), k=_logint(rng, 8, hi),
                    b=_logint(rng, 8, hi), s=rng.choice([2, 2, 3]), lead=rng.random() < 0.5)
    if kind in ("heff", "eigsolve"):
        p = rng.choice(["fp64", "split", "split"])
        hi = {"heff": {"fp64": 256, "split": 1024}, "eigsolve": {"fp64": 128, "split": 640}}[kind][p]
        x = _logint(rng, 24, hi)
        y = max(16, min(hi, int(x * rng.uniform(0.8, 1.2))))
        return dict(kind=kind, precision=p, chiL=x, chiR=y, d=rng.choice([2, 2, 3]) if x < 200 else 2,
                    w=rng.choice([3, 5]))
    if kind == "factorize":
        m = _logint(rng, 64, 1700)
        n = max(48, min(1700, int(m * rng.uniform(0.75, 1.3)))) if rng.random() < 0.7 else m
        return dict(kind=kind, m=m, n=n, keep=max(8, int(min(m, n) * rng.uniform(0.35, 0.6))),
                    by=rng.choice(["maxdim", "cutoff"]), ortho=rng.choice(["left", "right"]))
    if kind == "svd":
        m = _logint(rng, 24, 360)
        n = max(16, min(360, int(m * rng.uniform(0.6, 1.4))))
        return dict(kind=kind, m=m, n=n, keep=max(4, int(min(m, n) * rng.uniform(0.3, 0.7))))
    if kind == "permute":
        return dict(kind=kind, d0=_logint(rng, 16, 150), d1=_logint(rng, 16, 250), d2=_logint(rng, 2, 64),
                    d3=_logint(rng, 16, 64), order=rng.randrange(len(_ORDERS)), add=rng.random() < 0.4)
    if kind == "dmrg":
        return dict(kind=kind, N=rng.randrange(8, 21), maxdim=rng.randrange(8, 25), sweeps=rng.choice([1, 2]),
                    seed=rng.randrange(1000))
    return dict(kind="batched", count=rng.randrange(4, 17), N=rng.randrange(6, 11), maxdim=rng.randrange(8, 25),
                sweeps=rng.choice([1, 2]))


# index orders of the rank-4 permutations and sums
_ORDERS = [(1, 0, 2, 3), (0, 2, 1, 3), (2, 3, 0, 1), (3, 2, 1, 0), (1, 2, 3, 0), (0, 3, 2, 1)]


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape, cplx=False):
    dt = torch.complex128 if cplx else torch.float64
    return torch.randn(*shape, dtype=dt, device="cuda", generator=g)


def _tensor(data, *inds):
    return itg.ITensor(itg.Dense(data), inds)


def _contract_dims(c):
    """Dims of A and B, storage order; the bond k leads in both or trails in A."""
    a, k, b, s = c["a"], c["k"], c["b"], c["s"]
    return ((k, s, a) if c["lead"] else (a, s, k)), (k, s, b)


def _contract_data(c, seed):
    g = _gen(seed)
    dA, dB = _contract_dims(c)
    return [_randn(g, math.prod(d), cplx=c["cplx"]) for d in (dA, dB)]


def _heff_data(c, seed):
    """L, R, W1, W2, psi as flat column-major data, N(0,1); symmetric for the eigensolve.
    The torch views list the dims slowest first."""
    g = _gen(seed)
    x, y, d, w = c["chiL"], c["chiR"], c["d"], c["w"]
    L, R = _randn(g, x, w, x), _randn(g, y, w, y)
    W1, W2 = _randn(g, w, d, d, w), _randn(g, w, d, d, w)
    psi = _randn(g, y, d, d, x)
    if c["kind"] == "eigsolve":
        # a Hermitian operator whose spectrum has a separated lower end, as a gapped chain's has
        L, R = L + L.transpose(0, 2), R + R.transpose(0, 2)
        W1, W2 = W1 + W1.transpose(1, 2), W2 + W2.transpose(1, 2)
    return [t.contiguous().view(-1) for t in (L, W1, W2, R, psi)]


def _spectrum(r, keep):
    """Schmidt values of a bond: exponential decay to 3e-4 at the last kept one, a multiplet gap, then a
    decaying tail of values to be discarded."""
    j = np.arange(r)
    s = np.exp(-8.1 * j / keep)
    s[keep:] = 0.25 * 3e-4 * np.exp(-8.1 * (j[keep:] - keep) / keep)
    return s / np.sqrt((s * s).sum())


def _matrix(c, seed):
    """An m x n matrix with that spectrum between random bases (a two-site tensor), torch (n, m) = column-major."""
    g = _gen(seed)
    m, n = c["m"], c["n"]
    r = min(m, n)
    U, _ = torch.linalg.qr(_randn(g, m, r))
    V, _ = torch.linalg.qr(_randn(g, n, r))
    s = torch.from_numpy(_spectrum(r, c["keep"])).cuda()
    return ((V * s) @ U.T).contiguous()


def _trunc(c):
    if c.get("by", "maxdim") == "maxdim":
        return dict(maxdim=c["keep"], cutoff=0.0)
    p = _spectrum(min(c["m"], c["n"]), c["keep"]) ** 2
    lost = p[c["keep"]:].sum()
    return dict(cutoff=float(math.sqrt(lost * (lost + p[c["keep"] - 1]))))


def _permute_dims(c):
    return (c["d0"], c["d1"], c["d2"], c["d3"])


def _permute_data(c, seed):
    g = _gen(seed)
    n = math.prod(_permute_dims(c))
    return [_randn(g, n) for _ in range(2 if c["add"] else 1)]


def prepare(case, seed):
    c = case
    st = dict(c)
    if c["kind"] == "contract":
        A, B = _contract_data(c, seed)
        k, s, a, s2, b = (itg.Index(x) for x in (c["k"], c["s"], c["a"], c["s"], c["b"]))
        st["A"] = _tensor(A, *((k, s, a) if c["lead"] else (a, s, k)))
        st["B"] = _tensor(B, k, s2, b)
    elif c["kind"] in ("heff", "eigsolve"):
        L, W1, W2, R, psi = _heff_data(c, seed)
        st.update(L=L, W1=W1, W2=W2, R=R, psi=psi, out=torch.empty_like(psi), h=itg.handle(0))
    elif c["kind"] in ("factorize", "svd"):
        i, j = itg.Index(c["m"]), itg.Index(c["n"])
        st["A"] = _tensor(_matrix(c, seed).view(-1), i, j)
        st["i"], st["trunc"] = i, _trunc(c)
    elif c["kind"] == "permute":
        data = _permute_data(c, seed)
        inds = [itg.Index(x) for x in _permute_dims(c)]
        st["order"] = [inds[q] for q in _ORDERS[c["order"]]]
        st["A"] = _tensor(data[0], *inds)
        if c["add"]:
            st["B"] = _tensor(data[1], *st["order"])
    elif c["kind"] == "dmrg":
        rng = np.random.default_rng(seed)
        sites = itg.siteinds("S=1/2", c["N"])
        st["H"] = itg.cuMPO(itg.tfim_mpo(sites, h=float(rng.uniform(0.55, 0.7))))
        st["psi"] = itg.randomCuMPS(sites, min(8, c["maxdim"]), seed=1000 * c["seed"] + int(seed) % 1000 + 1)
        st["sweeps"] = itg.Sweeps(c["sweeps"], maxdim=[min(12, c["maxdim"]), c["maxdim"]], cutoff=[1e-10])
    else:
        rng = np.random.default_rng(seed)
        st["H"], st["psi"], st["md"] = [], [], []
        for q in range(c["count"]):
            sites = itg.siteinds("S=1/2", c["N"])
            J = rng.uniform(0.5, 1.5, c["N"] - 1)
            D = rng.uniform(0.3, 1.7, c["N"] - 1)
            st["H"].append(itg.cuMPO(itg.xxz_mpo(sites, J=J, Delta=D, h=0.25)))
            md = max(6, c["maxdim"] - 4 * (q % 4))
            st["md"].append([min(md, 8), md])
            st["psi"].append(itg.randomCuMPS(sites, min(6, md), seed=int(rng.integers(1, 1 << 30))))
    return st


# --------------------------------------------------------------------- run
def _p(t):
    return C.c_void_p(t.data_ptr())


def _dense_state(psi):
    """The state vector of a small MPS: the product of its site tensors."""
    t = psi[0]
    for j in range(1, len(psi)):
        # the sites so far as one index: a tensor has at most 16
        t = _tensor(t.store.data, itg.Index(itg.dim(t.inds[:-1])), t.inds[-1]) * psi[j]
    return t.store.data


def run(st):
    kind = st["kind"]
    if kind == "contract":
        return itg.contract(st["A"], st["B"], precision=_PREC[st["precision"]]).store.data
    if kind in ("heff", "eigsolve"):
        h = st["h"]
        dims = [C.c_int64(x) for x in (st["chiL"], st["chiR"], st["d"], st["w"], st["w"], st["w"])]
        ops = [_p(st[x]) for x in ("L", "W1", "W2", "R")]
        if kind == "heff":
            h.call("itg_heff2_apply", *dims, *ops, _p(st["psi"]), _p(st["out"]), _PREC[st["precision"]])
            return st["out"]
        x = st["out"]
        x.copy_(st["psi"])
        e, nmv = C.c_double(), C.c_int()
        h.call("itg_davidson_heff2", *dims, *ops, _p(x), 3, 2, C.c_double(1e-14), _PREC[st["precision"]], C.byref(e),
               C.byref(nmv))
        return {"energy": e.value, "psi": x, "matvecs": nmv.value}
    if kind == "factorize":
        # the bond split of a sweep: the factors, the two-site tensor that the next step forms from them, and the
        # overlap of the orthonormal one (its environment)
        L, R, spec = itg.factorize(st["A"], st["i"], ortho=st["ortho"], precision="split", **st["trunc"])
        Q = L if st["ortho"] == "left" else R
        q = next(x for x in Q.inds if x in L.inds and x in R.inds)
        gram = itg.contract(Q, Q.replaceinds([q], [q.prime()]), precision=_PREC["split"])
        phi = itg.contract(L, R, precision=_PREC["split"])
        return {"phi": phi.store.data, "gram": gram.store.data, "eigs": spec.eigs}
    if kind == "svd":
        U, S, V, spec = itg.svd(st["A"], st["i"], **st["trunc"])
        return {"A": (U * S * V).store.data, "S": S.store.data}
    if kind == "permute":
        if st["add"]:
            return (st["B"] + st["A"]).store.data
        return itg.permute(st["A"], *st["order"]).store.data
    if kind == "dmrg":
        e, psi = itg.dmrg(st["H"], st["psi"], st["sweeps"])
        return {"energy": e, "state": _dense_state(psi)}
    e, psis, _ = itg.dmrg_batched(st["H"], st["psi"], st["sweeps"], st["md"], 1e-10)
    return {"energies": e, "states": [_dense_state(p) for p in psis]}


# -------------------------------------------------------------------- work
def work(case):
    c = case
    k = c["kind"]
    if k == "contract":
        f = 4 if c["cplx"] else 1
        dA, dB = _contract_dims(c)
        e = 16 if c["cplx"] else 8
        out = c["s"] ** 2 * c["a"] * c["b"]
        return {"bytes": e * (math.prod(dA) + math.prod(dB) + out), "flops": f * 2 * out * c["k"]}
    if k in ("heff", "eigsolve"):
        x, y, d, w = c["chiL"], c["chiR"], c["d"], c["w"]
        env, n = w * (x * x + y * y), d * d * x * y
        flops = 2 * n * w * (x + y) + 2 * x * y * (2 * w * w * d ** 3)
        if k == "heff":
            return {"bytes": 8 * (env + 2 * n + 2 * w * w * d * d), "flops": flops}
        return {"bytes": 8 * (env + 2 * n), "flops": 5 * flops}
    if k in ("factorize", "svd"):
        m, n = max(c["m"], c["n"]), min(c["m"], c["n"])
        # QR, singular values and one set of vectors, the projection
        return {"bytes": 8 * (m * n + c["keep"] * (m + n)),
                "flops": 2 * m * n * n + 8 * n ** 3 + 2 * m * n * c["keep"]}
    if k == "permute":
        return {"bytes": 8 * (3 if c["add"] else 2) * math.prod(_permute_dims(c)), "flops": 0}
    # whole runs: the matvecs (five an eigensolve) and the splits of the bonds at the run's bond dimension
    w = 3 if k == "dmrg" else 5
    count = 1 if k == "dmrg" else c["count"]
    flops = byts = 0
    for b in range(c["N"] - 1):
        x, y = (min(c["maxdim"], 2 ** q, 2 ** (c["N"] - q)) for q in (b, b + 2))
        n = 4 * x * y
        m, r = 2 * max(x, y), 2 * min(x, y)
        flops += 5 * 2 * n * w * (x + y) + 2 * m * r * r + 8 * r ** 3
        byts += 8 * (w * (x * x + y * y) + 2 * n)
    return {"bytes": 2 * c["sweeps"] * count * byts, "flops": 2 * c["sweeps"] * count * flops}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    c = case
    k = c["kind"]
    if k == "contract":
        A, B = _contract_data(c, seed)
        dA, dB = _contract_dims(c)
        A, B = A.view(dA[::-1]), B.view(dB[::-1])   # slowest index first
        # out (a, s, s2, b) in storage order: leading-bond A keeps (s, a)
        out = torch.einsum("atk,buk->buat" if c["lead"] else "kta,buk->buta", A, B)
        return out.contiguous().view(-1)
    if k == "heff":
        L, W1, W2, R, psi = _heff_data(c, seed)
        x, y, d, w = c["chiL"], c["chiR"], c["d"], c["w"]
        L, R = L.view(x, w, x), R.view(y, w, y)                 # [a', w, a]
        W1, W2 = W1.view(w, d, d, w), W2.view(w, d, d, w)       # [x, s, s', w]
        psi = psi.view(y, d, d, x)                              # [b, s2, s1, a]
        t = torch.einsum("pwa,btsa->pwbts", L, psi)
        t = torch.einsum("pwbts,xsuw->pbtxu", t, W1)
        t = torch.einsum("pbtxu,ytvx->pbuvy", t, W2)
        return torch.einsum("pbuvy,qyb->qvup", t, R).contiguous().view(-1)
    if k in ("factorize", "svd"):
        A = _matrix(c, seed)  # (n, m), the transposed matrix
        U, s, Vh = torch.linalg.svd(A, full_matrices=False)
        q = c["keep"]
        kept = ((U[:, :q] * s[:q]) @ Vh[:q]).contiguous().view(-1)
        if k == "svd":
            return {"A": kept, "S": s[:q]}
        return {"phi": kept, "gram": torch.eye(q, dtype=torch.float64, device="cuda").view(-1), "eigs": s[:q] ** 2}
    if k == "permute":
        data = _permute_data(c, seed)
        dims = _permute_dims(c)
        order = _ORDERS[c["order"]]
        # torch axis of storage mode q is 3 - q
        t = data[0].view(dims[::-1]).permute([3 - q for q in order[::-1]]).contiguous().view(-1)
        return t + data[1] if c["add"] else t
    return None
