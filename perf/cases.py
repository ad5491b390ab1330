"""The work that users of this package give the GPU, as cases whose time can be measured.

Whole calls (a solve, a served batch, a product rounded back to low rank) return dense tensors, which
do not depend on the gauge of the TT cores; the building blocks (the local product of the AMEn sweep
on each engine, the interface updates of both sweep directions, the SVD of a supercore) go through
``torchtt_gb300.ops``. Sizes are those of the repository's workloads (``torchtt_gb300/workloads.py``)
and tests: modes of 12 to 64, operator ranks 2 (Kronecker sum), 3 (with a potential) and 7 (with a
dense perturbation), solution ranks up to the 160 to 175 of the parametric-diffusion systems.
"""
import math

import torch

from torchtt_gb300 import TT, amen_solve, ops
from torchtt_gb300 import workloads as W
from torchtt_gb300.serving import Server

DEV = "cuda"
F64 = torch.float64
ENGINES = {"tc": ops.ENGINE_TC, "df": ops.ENGINE_DF, "fp32": ops.ENGINE_FP32}


def listed():
    return [
        # the smallest whole solve: the random system of the solver tests, direct local solves;
        # launches and host synchronisations are all there is
        dict(name="solve_random_4x5x6", kind="solve", op="random", d=3, n=5, rank=2, eps=1e-10,
             precision="fp64"),
        # an ordinary plain solve with the default settings' eps (the d = 5, n = 12 Laplacian)
        dict(name="solve_laplace_d5_n12", kind="solve", op="laplace", d=5, n=12, rank=3, eps=1e-10,
             precision="fp64"),
        # a solve of the mixed path: an anisotropic Laplacian as in the serving trace
        dict(name="solve_mixed_d4_n32", kind="solve", op="laplace", d=4, n=32, rank=6, eps=1e-10,
             precision="mixed"),
        # requests served at once, more than there are slots
        dict(name="serve_6_d4_n16", kind="serve", requests=6, slots=4, d=4, n=16, rank=5, eps=1e-10,
             precision="mixed"),
        # the local product of an early sweep (d = 8, n = 16 Laplacian): latency
        dict(name="product_small_r4_n16", kind="product", op="laplace", r=4, n=16, R=4,
             engine="fp64"),
        # the plain path's local product at the ranks of the parametric-diffusion systems
        dict(name="product_r161_n32_R157", kind="product", op="laplace", r=161, n=32, R=157,
             engine="fp64"),
        # the true residual of the mixed path at the d = 20, n = 64 workload's ranks
        dict(name="product_df_r88_n64_R79", kind="product", op="potential", r=88, n=64, R=79,
             engine="df"),
        # the operator of the mixed path's inner GMRES, tensor cores, ragged ranks
        dict(name="product_tc_r61_n64_R67", kind="product", op="potential", r=61, n=64, R=67,
             engine="tc"),
        # the forward sweep's interface of an operator with a dense perturbation (rounding stress)
        dict(name="interface_fwd_dense_r64_n32", kind="interface", op="dense", r=64, n=32, R=60,
             direction="fwd"),
        # the backward sweep's interface of a Kronecker sum, ordinary odd ranks
        dict(name="interface_bck_r37_n32_R53", kind="interface", op="laplace", r=37, n=32, R=53,
             direction="bck"),
        # the truncation of a supercore
        dict(name="svd_r80_n64_R77", kind="svd", r=80, n=64, R=77, decay=4.0),
        # an operator applied to a TT and the product rounded back
        dict(name="apply_round_d4_n32_r24", kind="round", op="laplace", d=4, n=32, rank=24,
             eps=1e-10),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["product", "product", "product", "interface", "interface", "svd", "round",
                       "solve", "solve", "serve"])
    if kind == "product":
        return dict(kind=kind, op=rng.choice(["laplace", "potential", "potential", "dense"]),
                    r=_log_int(rng, 2, 128), n=_log_int(rng, 12, 64), R=_log_int(rng, 2, 96),
                    engine=rng.choice(["fp64", "fp64", "df", "tc", "fp32"]))
    if kind == "interface":
        return dict(kind=kind, op=rng.choice(["laplace", "potential", "dense"]),
                    r=_log_int(rng, 2, 96), n=_log_int(rng, 12, 64), R=_log_int(rng, 2, 96),
                    direction=rng.choice(["fwd", "bck"]))
    if kind == "svd":
        return dict(kind=kind, r=_log_int(rng, 2, 80), n=_log_int(rng, 12, 64),
                    R=_log_int(rng, 4, 80), decay=round(rng.uniform(2.0, 4.0), 2))
    if kind == "round":
        return dict(kind=kind, op=rng.choice(["laplace", "potential"]), d=rng.randint(3, 4),
                    n=_log_int(rng, 12, 32), rank=_log_int(rng, 2, 20), eps=1e-10)
    if kind == "serve":
        return dict(kind=kind, requests=rng.randint(2, 6), slots=rng.randint(2, 4), d=rng.randint(3, 4),
                    n=_log_int(rng, 8, 16), rank=rng.randint(1, 5), eps=1e-10,
                    precision=rng.choice(["mixed", "fp64"]))
    return dict(kind=kind, op="laplace", d=rng.randint(3, 4), n=_log_int(rng, 8, 32),
                rank=rng.randint(1, 6), eps=1e-10, precision=rng.choice(["fp64", "mixed"]))


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------

def _tt(cores):
    return TT([c.to(DEV) for c in cores])


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _coeffs(seed, d):
    """Per-mode coefficients U[0.1, 10] of the serving trace."""
    g = torch.Generator().manual_seed(int(seed) * 104729 + 5)
    return (0.1 + 9.9 * torch.rand(d, generator=g, dtype=F64)).tolist()


def _system(case, seed):
    """Operator and right-hand side of a solve, as CPU cores."""
    d, n, r = case["d"], case["n"], case["rank"]
    if case.get("op") == "random":
        w = W.small_random_system(seed=seed, N=(n - 1, n, n + 1))
        return w["A"], w["b"]
    return (W.laplace_ttm(d, n, coeffs=_coeffs(seed, d)),
            W.random_tt([n] * d, [1] + [r] * (d - 1) + [1], seed))


def _operator_core(op, n, seed):
    """A middle core of the operator: Kronecker sum (rank 2), with a potential (rank 3), or with a
    dense perturbation (rank 7)."""
    if op == "laplace":
        return W.laplace_ttm(3, n, coeffs=_coeffs(seed, 3))[1].to(DEV)
    if op == "potential":
        return W.laplace_potential_ttm(3, n)[1].to(DEV)
    return W.laplace_lowrank_spd_ttm(3, n, seed)[1].to(DEV)


def _orthogonal(r, g):
    return torch.linalg.qr(torch.randn(r, r, generator=g, dtype=F64, device=DEV))[0]


def _interface(op, r, n, left, g):
    """An interface r x s x r as a sweep has it: the identity where no term of the sum has been
    applied, an SPD matrix with the spread of a projected Laplacian where one has, near-constant SPD
    or random blocks for the potential and the perturbation; of unit norm."""
    s = {"laplace": 2, "potential": 3, "dense": 7}[op]
    phi = torch.empty(r, s, r, dtype=F64, device=DEV)
    eye = torch.eye(r, dtype=F64, device=DEV)
    for k in range(s):
        q = _orthogonal(r, g)
        u = torch.rand(r, generator=g, dtype=F64, device=DEV)
        if k == (1 if left else 0):
            m = (q * (30.0 + 4.0 * (n + 1) ** 2 * u)) @ q.T
        elif k < 2:
            m = eye
        elif op == "potential" or k == s - 1:
            m = (q * (0.5 + u)) @ q.T
        else:
            m = torch.randn(r, r, generator=g, dtype=F64, device=DEV)
        phi[:, k] = m
    return phi / torch.linalg.vector_norm(phi)


def _core(r, n, R, g):
    """A supercore: entries that fall off along both ranks, of unit norm."""
    x = torch.randn(r, n, R, generator=g, dtype=F64, device=DEV)
    x = x * torch.logspace(0, -3, r, dtype=F64, device=DEV)[:, None, None]
    x = x * torch.logspace(0, -3, R, dtype=F64, device=DEV)
    return x / torch.linalg.vector_norm(x)


def _left_orthogonal(r, n, R, g):
    """A core with orthonormal columns (r n >= R) or rows."""
    x = torch.randn(r * n, R, generator=g, dtype=F64, device=DEV)
    q = torch.linalg.qr(x)[0] if r * n >= R else torch.linalg.qr(x.T)[0].T
    return q.reshape(r, n, R).contiguous()


def _supercore(case, seed):
    """An (r n) x R unfolding whose singular values fall off geometrically by `decay` decades."""
    g = _gen(seed)
    rows, cols = case["r"] * case["n"], case["R"]
    k = min(rows, cols)
    u = torch.linalg.qr(torch.randn(rows, k, generator=g, dtype=F64, device=DEV))[0]
    v = torch.linalg.qr(torch.randn(cols, k, generator=g, dtype=F64, device=DEV))[0]
    s = torch.logspace(0, -case["decay"], k, dtype=F64, device=DEV)
    return ((u * s) @ v.T).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        A, b = _system(case, seed)
        return dict(case=case, A=_tt(A), b=_tt(b))
    if kind == "serve":
        pairs = [_system(case, seed * 64 + i) for i in range(case["requests"])]
        return dict(case=case, systems=[(_tt(A), _tt(b)) for A, b in pairs],
                    server=Server(slots=case["slots"]))
    if kind == "product":
        g = _gen(seed)
        r, n, R = case["r"], case["n"], case["R"]
        return dict(case=case, phi_l=_interface(case["op"], r, n, True, g),
                    phi_r=_interface(case["op"], R, n, False, g),
                    A=_operator_core(case["op"], n, seed), x=_core(r, n, R, g))
    if kind == "interface":
        g = _gen(seed)
        r, n, R = case["r"], case["n"], case["R"]
        fwd = case["direction"] == "fwd"
        # the enriched core of a sweep can have no more columns than rows
        x = _left_orthogonal(r, n, R, g) if fwd else \
            _left_orthogonal(R, n, r, g).permute(2, 1, 0).contiguous()
        return dict(case=case, phi=_interface(case["op"], r if fwd else R, n, fwd, g),
                    A=_operator_core(case["op"], n, seed), x=x)
    if kind == "svd":
        return dict(case=case, m=_supercore(case, seed))
    d, n, r = case["d"], case["n"], case["rank"]
    A = W.laplace_ttm(d, n) if case["op"] == "laplace" else W.laplace_potential_ttm(d, n)
    return dict(case=case, A=_tt(A), x=_tt(W.random_tt([n] * d, [1] + [r] * (d - 1) + [1], seed)))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        return amen_solve(state["A"], state["b"], eps=case["eps"], precision=case["precision"]).full()
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(A, b, eps=case["eps"], precision=case["precision"])
               for A, b in state["systems"]]
        return [srv.result(i)[0].full() for i in ids]
    if kind == "product":
        if case["engine"] == "fp64":
            return ops.local_product(state["phi_r"], state["phi_l"], state["A"], state["x"])
        return ops.local_product_lowp(state["phi_r"], state["phi_l"], state["A"], state["x"],
                                      engine=ENGINES[case["engine"]])
    if kind == "interface":
        update = ops.compute_phi_fwd_A if case["direction"] == "fwd" else ops.compute_phi_bck_A
        return update(state["phi"], state["x"], state["A"], state["x"])
    if kind == "svd":
        # the signs of a pair of singular vectors are free: those with a positive column sum
        u, s, vh = ops.svd(state["m"])
        sign = torch.sign(u.sum(dim=0))
        return u * sign, s, vh * sign[:, None]
    return (state["A"] @ state["x"]).round(case["eps"]).full()


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without, and its results from plain torch in 64 bits
# ------------------------------------------------------------------------------------------------

def _nnz(op, n):
    """Nonzeros of a middle operator core: identities, tridiagonal blocks and diagonals."""
    if op == "dense":
        return 16 * n * n + 6 * n
    return 2 * n + (3 * n - 2) + (n if op == "potential" else 0)


def work(case):
    kind = case["kind"]
    if kind in ("solve", "serve"):
        # one local product per core at the rank of the right-hand side, and the dense result
        d, n, r = case["d"], case["n"], case["rank"]
        m = case.get("requests", 1)
        full = float(n) ** d
        return {"bytes": 8.0 * m * (full + d * (2 * n * n * 2 + r * n * r)),
                "flops": m * (d * 2.0 * r * n * r * 4 * r + 2.0 * full * r)}
    if kind == "round":
        d, n = case["d"], case["n"]
        s = 2 if case["op"] == "laplace" else 3
        full, q = float(n) ** d, s * case["rank"]
        return {"bytes": 8.0 * (full + d * (s * n * n * s + case["rank"] ** 2 * n)),
                "flops": 2.0 * full * min(q, n) + d * 6.0 * q * n * q * min(q, n)}
    r, n, R = case["r"], case["n"], case["R"]
    if kind == "svd":
        a, b = max(r * n, R), min(r * n, R)
        return {"bytes": 8.0 * (2 * a * b + b + b * b), "flops": 6.0 * a * b * b + 20.0 * b ** 3}
    s = {"laplace": 2, "potential": 3, "dense": 7}[case["op"]]
    nnz = _nnz(case["op"], n)
    core, phi_l, phi_r = r * n * R, r * s * r, R * s * R
    flops = 2.0 * (core * r * s + nnz * r * R + core * R * s)
    # input and output cores of a product; one core and two interfaces of an update
    moved = 2 * core if kind == "product" else core
    return {"bytes": 8.0 * (moved + phi_l + phi_r + nnz), "flops": flops}


def _dense_solve(case, seed):
    """The exact solution: by the eigenvectors of the 1-D operators, or a dense solve."""
    A, b = _system(case, seed)
    A, b = [c.to(DEV) for c in A], [c.to(DEV) for c in b]
    rhs = _full(b)
    if case.get("op") == "random":
        m = A[0][0]
        for c in A[1:]:
            k = m.shape[0] * c.shape[1]
            m = torch.einsum("abs,smnS->ambnS", m, c).reshape(k, k, c.shape[3])
        return torch.linalg.solve(m[..., 0], rhs.reshape(-1)).reshape(rhs.shape)
    d, n = case["d"], case["n"]
    lam, q = torch.linalg.eigh(torch.as_tensor(W.laplace_1d(n), dtype=F64, device=DEV))
    total = torch.zeros([1] * d, dtype=F64, device=DEV)
    for k, c in enumerate(_coeffs(seed, d)):
        total = total + (c * lam).reshape([-1 if i == k else 1 for i in range(d)])

    def rotate(t, m):
        for _ in range(d):   # the first mode each time, moved to the end
            t = torch.tensordot(t, m, dims=([0], [0]))
        return t

    return rotate(rotate(rhs, q) / total, q.T.contiguous())


def _full(cores):
    t = cores[0][0]
    for c in cores[1:]:
        t = torch.tensordot(t, c, dims=([t.dim() - 1], [0]))
    return t[..., 0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        return _dense_solve(case, seed)
    if kind == "serve":
        return [_dense_solve(case, seed * 64 + i) for i in range(case["requests"])]
    st = prepare(case, seed)
    if kind == "product":
        w = torch.einsum("lsr,rnR->lsnR", st["phi_l"], st["x"])
        w = torch.einsum("smnS,lsnR->lmSR", st["A"], w)
        return torch.einsum("lmSR,LSR->lmL", w, st["phi_r"])
    if kind == "interface":
        x = st["x"]
        if case["direction"] == "fwd":
            t = torch.einsum("lsr,lML->srML", st["phi"], x)
            t = torch.einsum("srML,sMNS->rLNS", t, st["A"])
            return torch.einsum("rLNS,rNR->LSR", t, x)
        t = torch.einsum("LSR,lML->lMSR", st["phi"], x)
        t = torch.einsum("lMSR,sMNS->lsNR", t, st["A"])
        return torch.einsum("lsNR,rNR->lsr", t, x)
    if kind == "svd":
        u, s, vh = torch.linalg.svd(st["m"], full_matrices=False)
        sign = torch.sign(u.sum(dim=0))
        return u * sign, s, vh * sign[:, None]
    t = _full(st["x"].cores)
    total = torch.zeros_like(t)
    d, n = case["d"], case["n"]

    def on_mode(v, m, k):
        return torch.movedim(torch.tensordot(m, v, dims=([1], [k])), 0, k)

    lap = torch.as_tensor(W.laplace_1d(n), dtype=F64, device=DEV)
    for k in range(d):
        total = total + on_mode(t, lap, k)
    if case["op"] == "potential":
        p = torch.as_tensor(W.potential_1d(n), dtype=F64, device=DEV)
        for k in range(d):
            t = on_mode(t, p, k)
        total = total + t
    return total
