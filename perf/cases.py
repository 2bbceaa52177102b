"""The work that users of this framework have it do, as cases to be timed.

Each case calls the public Python API on host arrays, as a program that replaces
the Julia package would: the C ABI takes host pointers, so the copies in and out
belong to a pass.

Kinds:
  trg          ln Z per site of the 2D Ising model and its β-derivative (the
               README's and the user guide's example), bond dimension χ, niter
               coarse-graining steps
  mag          magnetisation of the Ising model by CTMRG from a random
               environment (src/exampletensors.jl:57-69)
  energy       iPEPS energy of the Heisenberg model on the plain FP64 path, with
               the gradient of the unrolled CTMRG when ``grad``: one evaluation
               of a variational optimisation
  mixed        the same evaluation on the mixed path (TF32X3 ladder, subspace
               solver, implicit adjoint)
  expectation  energy of a given environment: a measurement after CTMRG
  contract     one pairwise tensor contraction (the last one of CTMRG's corner
               growth), the role OMEinsum plays
  mlp          loss gradient of the warm-start network on one mini-batch
"""
from __future__ import annotations

import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

F64 = torch.float64


def _package():
    """The package directory of this tree (its name has a dot, so it is loaded by path)."""
    if "tnad_gb300" not in sys.modules:
        pkg = Path("tensornetworkad.jl_gb300").resolve()
        spec = importlib.util.spec_from_file_location("tnad_gb300", pkg / "__init__.py",
                                                      submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["tnad_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["tnad_gb300"]


# ---------------------------------------------------------------- the cases


def listed():
    return [
        # the user guide's example: the smallest call, all latency
        {"name": "trg_chi5_n5", "kind": "trg", "chi": 5, "niter": 5},
        # an odd bond dimension, 121×121 splits
        {"name": "trg_chi11_n8", "kind": "trg", "chi": 11, "niter": 8},
        # the README's bond dimension (400×400 splits), as many steps as reach them four times
        {"name": "trg_chi20_n7", "kind": "trg", "chi": 20, "niter": 7},
        # an order parameter at one temperature of a scan
        {"name": "mag_chi16", "kind": "mag", "chi": 16, "tol": 1e-6, "maxit": 100},
        # one optimisation step's evaluation on the README's model: D = 2, χ = 20 (80×80 corner)
        {"name": "energy_grad_D2_chi20", "kind": "energy", "D": 2, "chi": 20, "recipe": "uniform", "tol": 1e-10,
         "maxit": 100, "grad": True},
        # D = 3, χ = 36 (324×324 corner)
        {"name": "energy_grad_D3_chi36", "kind": "energy", "D": 3, "chi": 36, "recipe": "uniform", "tol": 1e-10,
         "maxit": 100, "grad": True},
        # the largest plain-path evaluation: D = 4, χ = 64 (1024×1024 corner), a few CTMRG steps
        {"name": "energy_grad_D4_chi64", "kind": "energy", "D": 4, "chi": 64, "recipe": "normal", "tol": 1e-7,
         "maxit": 5, "grad": True},
        # the mixed path where it is meant to be used: a line-search energy at D = 4, χ = 64
        {"name": "mixed_energy_D4_chi64", "kind": "mixed", "D": 4, "chi": 64, "recipe": "near_bench", "tol": 1e-9,
         "maxit": 400, "grad": False},
        # the mixed path with its implicit adjoint, D = 3, χ = 36
        {"name": "mixed_grad_D3_chi36", "kind": "mixed", "D": 3, "chi": 36, "recipe": "uniform", "tol": 1e-12,
         "maxit": 200, "grad": True},
        # a measurement on a converged environment
        {"name": "expectation_D4_chi64", "kind": "expectation", "D": 4, "chi": 64},
        # corner growth at an odd χ as one library call
        {"name": "contract_d9_chi41", "kind": "contract", "D": 3, "chi": 41},
        # training the warm-start network: forward and backward on one mini-batch
        {"name": "mlp_grad_D2_chi16", "kind": "mlp", "D": 2, "chi": 16, "batch": 128},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trg", "trg", "mag", "energy", "energy", "energy", "mixed", "expectation", "contract", "mlp"])
    if kind == "trg":
        return {"kind": kind, "chi": rng.randint(4, 19), "niter": rng.randint(3, 7)}
    if kind == "mag":
        return {"kind": kind, "chi": rng.randint(3, 32), "tol": 1e-6, "maxit": rng.randint(40, 100)}
    if kind == "energy":
        D = rng.choice([2, 2, 3, 3, 4])
        recipe = rng.choice(["uniform", "normal"])
        chi = {2: rng.randint(8, 60), 3: rng.randint(10, 45), 4: rng.randint(17, 52)}[D]
        maxit = {2: rng.randint(10, 30), 3: rng.randint(6, 12), 4: rng.randint(3, 6)}[D]
        return {"kind": kind, "D": D, "chi": chi, "recipe": recipe, "tol": 1e-10, "maxit": maxit,
                "grad": rng.random() < 0.7}
    if kind == "mixed":
        D = rng.choice([2, 3, 4])
        chi = {2: rng.randint(12, 60), 3: rng.randint(12, 60), 4: rng.randint(24, 63)}[D]
        return {"kind": kind, "D": D, "chi": chi, "recipe": "uniform" if D < 4 else "near_bench",
                "tol": 10.0 ** -rng.uniform(8.5, 9.5), "maxit": 400, "grad": False}
    if kind == "expectation":
        return {"kind": kind, "D": rng.choice([2, 3, 4]), "chi": _log_int(rng, 7, 63)}
    if kind == "contract":
        return {"kind": kind, "D": rng.choice([2, 3, 4]), "chi": _log_int(rng, 9, 63)}
    D = rng.choice([2, 3])
    return {"kind": kind, "D": D, "chi": rng.randint(8, 24) if D == 2 else rng.randint(9, 20),
            "batch": _log_int(rng, 24, 200)}


# ---------------------------------------------------------------- inputs


def _site(case, seed):
    """Site tensor D×D×D×D×2: the benchmark's recipes, or (near_bench) a tensor in the
    neighbourhood of the D = 4 benchmark tensor, as a line search visits it."""
    D, rng = case["D"], np.random.default_rng(seed)
    shape = (D, D, D, D, 2)
    if case["recipe"] == "uniform":
        A = rng.random(shape)
    elif case["recipe"] == "normal":
        A = rng.standard_normal(shape)
        A = A / np.abs(A).max()
    else:
        A = np.random.default_rng(0).standard_normal(shape)
        A = A / np.abs(A).max()
        A = A + 0.01 * rng.standard_normal(shape)
    return np.asfortranarray(A)


def _beta(case, seed):
    lo, hi = (0.3, 0.6) if case["kind"] == "trg" else (0.46, 0.8)
    return float(np.random.default_rng(seed).uniform(lo, hi))


def _environment(case, seed):
    """A symmetric normalised environment and the double layer of a random site tensor."""
    D, chi = case["D"], case["chi"]
    d, rng = D * D, np.random.default_rng(seed)
    Cm, Tm = rng.standard_normal((chi, chi)), rng.standard_normal((chi, d, chi))
    Cm, Tm = Cm + Cm.T, Tm + Tm.transpose(2, 1, 0)
    A = rng.random((D, D, D, D, 2))
    ap = np.einsum("abcdx,ijkly->aibjckdlxy", A, A).transpose(1, 0, 3, 2, 5, 4, 7, 6, 8, 9).reshape(d, d, d, d, 2, 2)
    f = np.asfortranarray
    return f(Cm / np.linalg.norm(Cm)), f(Tm / np.linalg.norm(Tm)), f(ap), f(np.einsum("abcdxx->abcd", ap))


def _contraction(case, seed):
    d, chi, rng = case["D"] ** 2, case["chi"], np.random.default_rng(seed)
    return (np.asfortranarray(rng.standard_normal((chi, d, d, chi))),
            np.asfortranarray(rng.standard_normal((d, d, d, d))))


WIDTH = 512


def _mlp_sizes(case):
    D, chi = case["D"], case["chi"]
    return 2 * D ** 4, chi + chi * D * D * chi


def _mlp_inputs(case, seed):
    n_in, n_out = _mlp_sizes(case)
    rng = np.random.default_rng(seed)

    def layer(rows, cols):
        return (rng.standard_normal((rows, cols)) * math.sqrt(2.0 / cols)).astype(np.float32)

    W = [layer(WIDTH, n_in), layer(WIDTH, WIDTH), layer(n_out, WIDTH)]
    b = [(0.01 * rng.standard_normal(w.shape[0])).astype(np.float32) for w in W]
    X = np.asfortranarray(rng.standard_normal((n_in, case["batch"])).astype(np.float32))
    Y = np.asfortranarray(rng.standard_normal((n_out, case["batch"])).astype(np.float32))
    return W, b, X, Y


def prepare(case, seed):
    tn = _package()
    kind = case["kind"]
    st = {"tn": tn, "case": case}
    if kind == "trg":
        st["beta"] = _beta(case, seed)
    elif kind == "mag":
        st["beta"], st["seed"] = _beta(case, seed), seed
    elif kind in ("energy", "mixed"):
        st["h"] = tn.hamiltonian(tn.Heisenberg())
        st["ipeps"] = tn.SquareIPEPS(_site(case, seed))
    elif kind == "expectation":
        Cm, Tm, ap, bulk = _environment(case, seed)
        st["h"], st["ap"] = tn.hamiltonian(tn.Heisenberg()), ap
        st["rt"] = tn.SquareCTMRGRuntime(bulk, Cm, Tm)
    elif kind == "contract":
        st["x"], st["a"] = _contraction(case, seed)
    else:
        # the package by name: its submodule `learned` is loaded on first use
        learned = importlib.import_module("tnad_gb300.learned")
        W, b, st["X"], st["Y"] = _mlp_inputs(case, seed)
        st["net"] = learned.WarmStartNet(case["D"], 2, case["chi"], width=WIDTH, seed=1)
        st["net"].set_params(np.concatenate([x for w, v in zip(W, b) for x in (w.ravel(order="F"), v)]))
    return st


# ---------------------------------------------------------------- one pass


def run(st):
    tn, case, kind = st["tn"], st["case"], st["case"]["kind"]
    if kind == "trg":
        return tn.trg_beta(st["beta"], case["chi"], case["niter"])
    if kind == "mag":
        return tn.magnetisation(tn.Ising(), st["beta"], case["chi"], rng=np.random.default_rng(st["seed"]),
                                tol=case["tol"], maxit=case["maxit"])
    if kind in ("energy", "mixed"):
        # an optimisation that wants 1e-9 gradients asks the adjoint for them
        opts = tn.mixed_opts(fp_tol=1e-11) if kind == "mixed" else None
        args = (st["h"], st["ipeps"], case["chi"], case["tol"], case["maxit"])
        return tn.energy_and_gradient(*args, opts=opts) if case["grad"] else tn.energy(*args, opts=opts)
    if kind == "expectation":
        return tn.expectationvalue(st["h"], st["ap"], st["rt"])
    if kind == "contract":
        return tn.contract("ibcl,jkcb->ijlk", st["x"], st["a"])
    return st["net"].gradient(st["X"], st["Y"])


# ---------------------------------------------------------------- the work a pass cannot do without


def _ctmrg_step_flops(d, chi, full):
    """Corner growth and projection at the pairwise order, and the decomposition of the
    χd×χd corner (9n³ for all of it, a few products with χ columns for the leading part)."""
    n = chi * d
    grow = 2.0 * (chi ** 3 * d + chi ** 3 * d * d + chi * chi * d ** 4)
    proj = 2.0 * (n * n * chi + n * chi * chi + 2 * chi ** 3 * d * d + chi * chi * d ** 4)
    return grow + proj + (9.0 * n ** 3 if full else 8.0 * n * n * chi)


def work(case):
    kind, chi = case["kind"], case["chi"]
    if kind == "trg":
        flops, k = 0.0, 2
        for _ in range(case["niter"]):
            n = k * k
            k2 = min(chi, n)
            flops += 2 * 21.0 * n ** 3  # two full SVDs
            flops += 2.0 * (2 * k ** 2 * k * k2 ** 2 + k2 ** 4 * k * k)  # the four-tensor contraction
            flops += 2 * 8.0 * n ** 3 + 4.0 * k2 ** 4 * k * k  # its pullback and the SVD adjoints
            k = k2
        return {"bytes": 8 * 32, "flops": flops}
    if kind == "mag":
        return {"bytes": 8.0 * (16 + 2 * (chi * chi + 2 * chi * chi)), "flops": 30 * _ctmrg_step_flops(2, chi, True)}
    D = case["D"]
    d, nA = D * D, 2 * D ** 4
    if kind == "energy":
        steps = min(case["maxit"] + 1, 6 if case["recipe"] == "uniform" else 20)
        f = steps * _ctmrg_step_flops(d, chi, True)
        n = chi * d
        if case["grad"]:
            f += steps * (2 * _ctmrg_step_flops(d, chi, False) + 8.0 * n * n * chi)
        return {"bytes": 8.0 * (nA + 16 + (nA if case["grad"] else 1)), "flops": f}
    if kind == "mixed":
        n = chi * d
        f = (8 if case["recipe"] == "uniform" else 40) * _ctmrg_step_flops(d, chi, False)
        if case["grad"]:
            f += 9.0 * n ** 3 + 10 * 2 * _ctmrg_step_flops(d, chi, False)
        return {"bytes": 8.0 * (nA + 16 + (nA if case["grad"] else 1)), "flops": f}
    if kind == "expectation":
        f = 2.0 * (2 * chi ** 3 * d + chi ** 3 * d * d + chi * chi * d ** 4 * 4 + 4 * chi ** 3 * d * d +
                   16 * chi * chi * d)
        return {"bytes": 8.0 * (chi * chi * (1 + d) + 4 * d ** 4 + 16), "flops": f}
    if kind == "contract":
        return {"bytes": 8.0 * (2 * chi * chi * d * d + d ** 4), "flops": 2.0 * chi * chi * d ** 4}
    n_in, n_out = _mlp_sizes(case)
    params, B = WIDTH * (n_in + WIDTH + n_out) + 2 * WIDTH + n_out, case["batch"]
    return {"bytes": 4.0 * (2 * params + B * (n_in + n_out)), "flops": 6.0 * params * B}


# ---------------------------------------------------------------- the same in 64 bits, by plain torch


class _Svd(torch.autograd.Function):
    """Thin real SVD (U, S, V) of a square matrix; adjoint with F = d/(d² + 1e-40)."""

    @staticmethod
    def forward(ctx, A):
        U, S, Vh = torch.linalg.svd(A, full_matrices=False)
        V = Vh.T.contiguous()
        ctx.save_for_backward(U, S, V)
        return U, S, V

    @staticmethod
    def backward(ctx, dU, dS, dV):
        U, S, V = ctx.saved_tensors
        gap = (S * S)[None, :] - (S * S)[:, None]
        F = gap / (gap * gap + 1e-40)
        J, K = F * (U.T @ dU), F * (V.T @ dV)
        return U @ ((J + J.T) * S[None, :] + S[:, None] * (K + K.T) + torch.diag(dS)) @ V.T


def _cm(x, shape):
    """Column-major reshape."""
    r = x.permute(*reversed(range(x.ndim))).reshape(tuple(reversed(shape)))
    return r.permute(*reversed(range(len(shape))))


def _ising(beta, diag):
    cb, sb = torch.sqrt(torch.cosh(beta)), torch.sqrt(torch.sinh(beta))
    q = torch.stack([torch.stack([cb + sb, cb - sb]), torch.stack([cb - sb, cb + sb])]) / math.sqrt(2)
    t = torch.zeros(2, 2, 2, 2, dtype=F64)
    t[0, 0, 0, 0], t[1, 1, 1, 1] = diag
    return torch.einsum("abcd,ai,bj,ck,dl->ijkl", t, q, q, q, q)


def _exact_trg(beta, chi, niter):
    b = torch.tensor(beta, dtype=F64, requires_grad=True)
    a, ln = _ising(b, (1.0, 1.0)), torch.zeros((), dtype=F64)

    def split(t):
        d1, d2, d3, d4 = t.shape
        u, s, v = _Svd.apply(_cm(t, (d1 * d2, d3 * d4)))
        k = min(int((s > 1e-16).sum()) + 1, chi, s.numel())
        r = torch.sqrt(s[:k])
        return _cm(u[:, :k] * r, (d1, d2, k)), _cm(v[:, :k].T * r[:, None], (k, d3, d4))

    for n in range(niter):
        top = a.abs().max()
        a, ln = a / top, ln + 2.0 ** -n * torch.log(top)
        dr, ul = split(torch.einsum("urdl->drul", a))
        ld, ru = split(torch.einsum("urdl->ldru", a))
        a = torch.einsum("nuor,doln->urdl", torch.einsum("npu,por->nuor", dr, ld),
                         torch.einsum("dom,lmn->doln", ul, ru))
    ln = ln + torch.log(torch.einsum("ijij->", a)) / 2.0 ** niter
    (g,) = torch.autograd.grad(ln, b)
    return float(ln.detach()), float(g)


def _ctmrg(a, C, T, tol, maxit):
    chi, d = C.shape[0], a.shape[0]
    old, k = None, 0
    while True:
        cp = torch.einsum("ibcl,jkcb->ijlk", torch.einsum("ibd,dcl->ibcl", torch.einsum("ad,iba->ibd", C, T), T), a)
        M = _cm(cp, (chi * d, chi * d))
        u, s, _ = _Svd.apply(M + M.T)
        z = _cm(u[:, :chi], (chi, d, chi))
        C = torch.einsum("icd,cdj->ij", torch.einsum("abcd,abi->icd", cp, z), z)
        T = torch.einsum("dijc,dck->ijk", torch.einsum("edbi,bjce->dijc", torch.einsum("aed,abi->edbi", T, z), a), z)
        C, T = C + C.T, T + T.permute(2, 1, 0)
        C, T = C / torch.linalg.vector_norm(C), T / torch.linalg.vector_norm(T)
        vals, k = (s / s[0]).detach(), k + 1
        if k > maxit or (old is not None and float(torch.linalg.vector_norm(vals - old)) <= tol):
            return C, T
        old = vals


def _heisenberg():
    x, y, z = np.array([[0, 1.0], [1, 0]]), np.array([[0, -1.0], [1, 0]]), np.diag([1.0, -1.0])
    h = np.einsum("ij,kl->ijkl", z, z) - np.einsum("ij,kl->ijkl", x, x) + np.einsum("ij,kl->ijkl", y, y)
    return torch.as_tensor(np.einsum("ijcd,kc,ld->ijkl", h, x, x) / 2)


def _expectation(ap, C, T):
    ap = ap / torch.linalg.vector_norm(ap)
    w = torch.einsum("icb,bde->icde", torch.einsum("ab,ica->icb", C, T), T)
    v = torch.einsum("icde,cjfdlm->iejflm", w, ap)
    el = torch.einsum("iejflm,efk->ijklm", v, torch.einsum("eg,gfk->efk", C, T))
    G = torch.einsum("abcij,abckl->ijkl", el, el)
    return (G * _heisenberg()).sum() / torch.einsum("aabb->", G)


def _exact_energy(A0, chi, tol, maxit, grad):
    x = torch.tensor(np.ascontiguousarray(A0), requires_grad=grad)
    A = x
    for p in ((0, 3, 2, 1, 4), (2, 1, 0, 3, 4), (1, 0, 3, 2, 4), (3, 2, 1, 0, 4)):
        A = A + A.permute(*p)
    A = A / torch.linalg.vector_norm(A)
    d = A.shape[0] ** 2
    ap = _cm(torch.einsum("abcdx,ijkly->aibjckdlxy", A, A), (d, d, d, d, 2, 2))
    a = torch.einsum("ijklaa->ijkl", ap)
    C, T, m = torch.zeros(chi, chi, dtype=F64), torch.zeros(chi, d, chi, dtype=F64), min(d, chi)
    C[:m, :m] = a.detach().sum(dim=(2, 3))[:m, :m]
    T[:m, :, :m] = a.detach().sum(dim=3)[:m, :, :m]
    E = _expectation(ap, *_ctmrg(a, C, T, tol, maxit))
    if not grad:
        return float(E.detach())
    (g,) = torch.autograd.grad(E, x)
    return float(E.detach()), np.asfortranarray(g.numpy())


def exact(case, seed):
    kind = case["kind"]
    if kind == "trg":
        return _exact_trg(_beta(case, seed), case["chi"], case["niter"])
    if kind == "mag":
        beta, chi = torch.tensor(_beta(case, seed), dtype=F64), case["chi"]
        rng = np.random.default_rng(seed)
        C, T = torch.as_tensor(rng.standard_normal((chi, chi))), torch.as_tensor(rng.standard_normal((chi, 2, chi)))
        a = _ising(beta, (1.0, 1.0))
        C, T = _ctmrg(a, C + C.T, T + T.permute(2, 1, 0), case["tol"], case["maxit"])
        env = torch.einsum("alc,ckd,bjd,bia->ijkl", torch.einsum("ia,ajb,bk->ijk", C, T, C), T,
                           torch.einsum("ia,ajb,bk->ijk", C, T, C), T)
        return abs(float((env * _ising(beta, (1.0, -1.0))).sum() / (env * a).sum()))
    if kind in ("energy", "mixed"):
        tol = min(case["tol"], 1e-10) if kind == "mixed" else case["tol"]
        with torch.set_grad_enabled(case["grad"]):
            return _exact_energy(_site(case, seed), case["chi"], tol, case["maxit"], case["grad"])
    if kind == "expectation":
        Cm, Tm, ap, _ = (torch.as_tensor(np.ascontiguousarray(x)) for x in _environment(case, seed))
        return float(_expectation(ap, Cm, Tm))
    if kind == "contract":
        x, a = (torch.as_tensor(np.ascontiguousarray(v)) for v in _contraction(case, seed))
        return np.asfortranarray(torch.einsum("ibcl,jkcb->ijlk", x, a).numpy())
    W, b, X, Y = _mlp_inputs(case, seed)
    p = [torch.tensor(np.ascontiguousarray(v), dtype=F64, requires_grad=True) for w, v0 in zip(W, b) for v in (w, v0)]
    hcur = torch.as_tensor(X.astype(np.float64))
    for q in range(3):
        hcur = p[2 * q] @ hcur + p[2 * q + 1][:, None]
        hcur = torch.relu(hcur) if q < 2 else hcur
    loss = torch.mean((hcur - torch.as_tensor(Y.astype(np.float64))) ** 2)
    gs = torch.autograd.grad(loss, p)
    return float(loss.detach()), np.concatenate([g.numpy().ravel(order="F") for g in gs])
