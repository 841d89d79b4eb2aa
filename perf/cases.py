"""The work that users of this framework have it do, as timed cases.

`listed()` are the cases that are quoted, `draw` gives more of the same ranges.
`prepare` makes what a program holds before the call (an initialised solver, a
mesh on the host, a training set), `run` is one pass through the public entry
points, `work` the bytes and operations a pass cannot do without, and `exact`
the values of `run` in plain 64-bit numpy where such values exist.

Five kinds of call:

solve     `Solver.solve()` on an initialised handle: begin_solve (which
          refactors), `iters` ADMM iterations, positions out.
batch     the same on several uneven meshes of their own materials in one handle.
whole     `solve_bar`: a mesh on the host in, create, initialize, solve, positions out.
gradient  the element-level entry points of a caller that drives its own
          iteration: the global gradient at given positions, then A^-1 of it.
train     the prox network's trainer: a gradient, then one epoch, blob out.

The iteration counts end before elements of the meshes start to pass through
a vanishing stretch, where the energy follows the last bit of the positions.
"""
import math

import numpy as np
import torch

from wrapd_b200 import bars, prox_net
from wrapd_b200.solver import Solver, solve_bar

YOUNGS, POISSON = 1e5, 0.45


def listed():
    return [
        # the smallest mesh that the repository measures: iterations of some
        # hundred microseconds, launches and host round trips
        dict(name="solve_8x8x32", kind="solve", na=8, nb=8, nl=32, twist=180.0, bend=0.0, noise=0.02, iters=30,
             rw_every=0, history=6, mode="fp64"),
        # uneven sizes at the reference's own settings (history 6, reweighting
        # by the weight ratio, which is looked at in every iteration)
        dict(name="solve_13x11x37", kind="solve", na=13, nb=11, nl=37, twist=150.0, bend=0.0, noise=0.02, iters=20,
             rw_every=0, history=6, mode="fp64"),
        # the optional line search of the global step
        dict(name="solve_line_search_16x16x64", kind="solve", na=16, nb=16, nl=64, twist=180.0, bend=0.0, noise=0.01,
             iters=20, rw_every=10, history=5, mode="line_search"),
        # rotation-unaware ADMM: one linear solve per iteration
        dict(name="solve_unaware_20x18x50", kind="solve", na=20, nb=18, nl=50, twist=90.0, bend=0.0, noise=0.01,
             iters=20, rw_every=0, history=6, mode="unaware"),
        # the ARAP model, rotation-aware, fixed weights
        dict(name="solve_arap_24x24x48", kind="solve", na=24, nb=24, nl=48, twist=90.0, bend=0.0, noise=0.01,
             iters=20, rw_every=0, history=6, mode="arap"),
        # the benchmark's bar and settings
        dict(name="solve_32x32x128_bent", kind="solve", na=32, nb=32, nl=128, twist=360.0, bend=90.0, noise=0.01,
             iters=10, rw_every=10, history=5, mode="fp64"),
        # FP32 local steps, warm-started by the shipped network where stretches are stale
        dict(name="solve_32x32x128_network", kind="solve", na=32, nb=32, nl=128, twist=180.0, bend=0.0, noise=0.02,
             iters=20, rw_every=10, history=5, mode="network"),
        # the largest bar, reweight and refactor every 20 iterations
        dict(name="solve_64x64x160", kind="solve", na=64, nb=64, nl=160, twist=180.0, bend=0.0, noise=0.005, iters=20,
             rw_every=20, history=5, mode="fp64"),
        # many uneven meshes at once, FP32 local steps
        dict(name="batch_16_bars", kind="batch", count=16, iters=20, rw_every=10, history=5, mode="mixed"),
        # a new mesh from host memory to positions: symbolic analysis, uploads, solve
        dict(name="whole_16x16x64", kind="whole", na=16, nb=16, nl=64, twist=180.0, bend=0.0, noise=0.01, iters=20,
             rw_every=10, history=5, mode="fp64"),
        # element-level entry points with host arrays in and out
        dict(name="gradient_24x24x48", kind="gradient", na=24, nb=24, nl=48, twist=120.0, bend=0.0, noise=0.02),
        # training, at the trainer's default batch
        dict(name="train_262144", kind="train", samples=262144, batch=4096),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "batch", "whole", "gradient", "train"])
    if kind == "train":
        return dict(kind=kind, samples=_log_uniform(rng, 5000, 262144), batch=rng.choice([1000, 2048, 4096, 8192]))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 24), iters=rng.randint(5, 20), rw_every=rng.choice([0, 5, 10]),
                    history=rng.randint(3, 8), mode=rng.choice(["fp64", "mixed"]))
    na = _log_uniform(rng, 4, 40 if kind == "solve" else 24)
    nb = max(3, int(round(na * rng.uniform(0.6, 1.4))))
    c = dict(kind=kind, na=na, nb=nb, nl=int(round(max(na, nb) * rng.uniform(1.5, 4.0))),
             twist=round(rng.uniform(30.0, 180.0), 1), bend=0.0, noise=0.01)
    if kind == "gradient":
        return c
    c.update(iters=rng.randint(5, 20), rw_every=rng.choice([0, 5, 10]), history=rng.randint(3, 8), mode="fp64")
    if kind == "solve":
        c["mode"] = rng.choice(["fp64", "fp64", "mixed", "network", "line_search", "unaware", "arap"])
        if c["mode"] in ("unaware", "arap"):
            c["twist"] = round(rng.uniform(30.0, 90.0), 1)
    return c


# Settings of a mode.  tol = 0: a pass is a fixed number of iterations.
# rw_delay = 0: the weights come from the Hessian's eigenvalue from the first
# solve on, as they do past the first iterations of a long run.
_MODES = {
    "fp64": {},
    "mixed": dict(precision="mixed"),
    "network": dict(precision="mixed", prox_mode=2),
    "line_search": dict(global_ls=1),
    "unaware": dict(rot_aware=0),
    "arap": dict(model=1, reweighting=0),
}


def _settings(case):
    return dict(youngs=YOUNGS, poisson=POISSON, max_iters=case["iters"], tol=0.0, rw_delay=0,
                rw_every=case["rw_every"], lbfgs_m=case["history"], **_MODES[case["mode"]])


def _bar(case, seed):
    return bars.make_bar(case["na"], case["nb"], case["nl"], twist_deg=case["twist"], bend_deg=case["bend"],
                         noise=case["noise"], seed=seed)


def _batch(case, seed):
    """Uneven bars with their own materials, noise and twist from the seed."""
    sizes = bars.uniform01(77, 3 * case["count"]).reshape(-1, 3)
    own = bars.uniform01(seed, 3 * case["count"]).reshape(-1, 3)
    out = []
    for i, (s, u) in enumerate(zip(sizes, own)):
        na, nb, nl = 4 + int(13 * s[0]), 4 + int(13 * s[1]), 16 + int(49 * s[2])
        bar = bars.make_bar(na, nb, nl, twist_deg=30.0 + 150.0 * u[0], noise=0.02, seed=seed + i)
        out.append((bar, 10.0 ** (4.0 + 2.0 * u[1]), 0.35 + 0.1 * u[2]))
    return out


def _pairs(case, seed):
    """Prox inputs and targets of the shape that harvesting gives."""
    rng = np.random.default_rng(seed)
    n = case["samples"]
    mu, lam = prox_net.lame(YOUNGS, POISSON)
    sig = np.sort(rng.uniform(0.5, 1.5, (n, 3)), axis=1)[:, ::-1].copy()
    X = prox_net.features(sig, 10.0 ** rng.uniform(3.0, 6.0, n), mu, lam)
    T = (sig + 0.1 * (1.0 - sig) + 0.01 * rng.standard_normal(sig.shape)).astype(np.float32)
    return X, T


def _free(bar):
    return np.setdiff1d(np.arange(bar.n_verts), bar.pins)


def _gradient_input(case, seed):
    """The bar and the free positions at which the gradient is wanted: a step
    away from those at which the dual variables were set."""
    bar = _bar(case, seed)
    free = _free(bar)
    rng = np.random.default_rng(seed + 1)
    return bar, bar.init[free] + 0.01 * bar.h * rng.standard_normal((free.size, 3))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        X, T = _pairs(case, seed)
        return dict(case=case, X=X, T=T, blob=prox_net.init_blob(X, T, seed))
    if kind == "whole":
        return dict(case=case, bar=_bar(case, seed))
    if kind == "gradient":
        bar, x = _gradient_input(case, seed)
        s = Solver(youngs=YOUNGS, poisson=POISSON, reweighting=0)
        s.add_tetmesh(bar.rest, bar.init, bar.tets, pins=bar.pins)
        s.initialize()
        s.begin_solve()
        return dict(case=case, solver=s, x=x)
    s = Solver(**_settings(case))
    if kind == "batch":
        for bar, youngs, poisson in _batch(case, seed):
            s.add_tetmesh(bar.rest, bar.init, bar.tets, pins=bar.pins, youngs=youngs, poisson=poisson)
    else:
        bar = _bar(case, seed)
        s.add_tetmesh(bar.rest, bar.init, bar.tets, pins=bar.pins)
    if case["mode"] == "network":
        s.set_prox_net(prox_net.load_default())
    s.initialize()
    return dict(case=case, solver=s)


def _solved(s, x):
    return dict(x=x, objectives=s.log("objectives"), inner_iters=s.log("inner_iters").astype(np.int64),
                reweighted=s.log("reweighted").astype(np.int64))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("solve", "batch"):
        s = state["solver"]
        return _solved(s, s.solve())
    if kind == "whole":
        s, x = solve_bar(state["bar"], **_settings(case))
        out = _solved(s, x)
        s.close()
        return out
    if kind == "gradient":
        s = state["solver"]
        value, grad = s.global_grad(state["x"])
        return dict(value=value, grad=grad, step=s.solve_A(grad))
    tr = prox_net.Trainer(state["blob"])
    tr.set_data(state["X"], state["T"])
    loss, grad = tr.grad(0, min(case["batch"], case["samples"]))
    losses = tr.train(epochs=1, batch=case["batch"], lr=1e-3, lr_end=1e-4, seed=7)
    blob = tr.blob()
    tr.close()
    return dict(loss=loss, grad=grad, losses=losses, blob=blob)


# ---- what a pass cannot do without ------------------------------------------------
# Per element and iteration, FP64 state read once and written once: the local
# step 432 bytes; a gradient 18 of state, 12 of Di, 12 of gradient rows, 3 + 9
# of the stretches and the symmetric part, w2, vol and the indexes: 464 bytes.
# The factor of an n_a x n_b cross-section holds about 13 s values per free
# vertex (s = sqrt((n_a + 1)(n_b + 1)), from the dissection of the bars above) and
# costs about 13 s^3 operations per free vertex; a solve reads it twice.
_LOCAL_BYTES, _GRAD_BYTES, _ELEM_FLOPS = 432, 464, 4000


def _mesh_work(na, nb, nl, case):
    ne, nf = 6 * na * nb * nl, (na + 1) * (nb + 1) * (nl - 1)
    s = math.sqrt((na + 1) * (nb + 1))
    nnz, factor = 13.0 * s * nf, 13.0 * s ** 3 * nf
    it = case["iters"]
    factors = 0 if case["mode"] == "arap" else 1 + (it // case["rw_every"] if case["rw_every"] else 0)
    grads = 1 + (1 if case["mode"] == "unaware" else 2) * it
    per_solve = 16.0 * nnz + (2 * 8 * case["history"] + 6) * 24.0 * nf
    return dict(bytes=it * (_LOCAL_BYTES * ne + per_solve) + grads * _GRAD_BYTES * ne + factors * 16.0 * nnz,
                flops=it * (_ELEM_FLOPS * ne + 12.0 * nnz) + factors * factor)


def work(case):
    kind = case["kind"]
    if kind == "train":
        n, per = case["samples"], 2 * (5 * 64 + 64 * 64 + 64 * 3)
        steps = -(-n // case["batch"])
        return dict(bytes=2.0 * 32 * n + 8.0 * n + steps * 7 * 4.0 * prox_net.N_BLOB, flops=3.0 * per * n)
    if kind == "gradient":
        ne, nf = 6 * case["na"] * case["nb"] * case["nl"], (case["na"] + 1) * (case["nb"] + 1) * (case["nl"] - 1)
        nnz = 13.0 * math.sqrt((case["na"] + 1) * (case["nb"] + 1)) * nf
        return dict(bytes=_GRAD_BYTES * ne + 16.0 * nnz + 4 * 24.0 * nf, flops=1000.0 * ne + 12.0 * nnz)
    if kind == "batch":
        every = [_mesh_work(*bar.dims, case) for bar, _, _ in _batch(case, 0)]
        return {k: sum(w[k] for w in every) for k in ("bytes", "flops")}
    w = _mesh_work(case["na"], case["nb"], case["nl"], case)
    if kind == "whole":
        w["flops"] += 13.0 * ((case["na"] + 1) * (case["nb"] + 1)) ** 1.5 * (case["na"] + 1) * (case["nb"] + 1) * case["nl"]
    return w


# ---- the values in plain 64-bit arithmetic ------------------------------------------
def exact(case, seed):
    if case["kind"] == "gradient":
        return _exact_gradient(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    return None   # a trajectory of iterations, whose stopping rules are part of it


def _exact_gradient(case, seed):
    bar, x = _gradient_input(case, seed)
    free = _free(bar)
    mu, lam = prox_net.lame(YOUNGS, POISSON)
    P = bar.rest[bar.tets]
    Dm = np.stack([P[:, 1] - P[:, 0], P[:, 2] - P[:, 0], P[:, 3] - P[:, 0]], axis=2)
    w2 = (2.0066 * mu + 1.0122 * lam) * np.linalg.det(Dm) / 6.0
    S = np.array([[-1.0, -1.0, -1.0], [1.0, 0.0, 0.0], [0.0, 1.0, 0.0], [0.0, 0.0, 1.0]])
    Di = S @ np.linalg.inv(Dm)                                   # (n, 4, 3)

    def sym(xyz):
        F = np.swapaxes(xyz[bar.tets], 1, 2) @ Di                # (n, 3, 3)
        U, s, Vt = np.linalg.svd(F)
        V = np.swapaxes(Vt, 1, 2)
        for M in (U, V):                                          # reflections negate the last stretch
            r = np.linalg.det(M) < 0.0
            M[r, :, 2] *= -1.0
            s[r, 2] *= -1.0
        return F, U, s, V, (V * s[:, None, :]) @ np.swapaxes(V, 1, 2)

    P0 = sym(bar.init)[4]
    at = bar.init.copy()
    at[free] = x
    F, U, s, V, Sx = sym(at)
    value = float(np.sum(0.5 * w2 * np.sum((Sx - P0) ** 2, axis=(1, 2))))
    # d/dF of |sym(F) - P|^2 / 2 is F - U diag(s) (K + K^T) V^T, K = (V^T P V) / (s_i + s_j)
    Q = np.swapaxes(V, 1, 2) @ P0 @ V
    K = Q / (s[:, :, None] + s[:, None, :])
    M = F - (U * s[:, None, :]) @ (K + np.swapaxes(K, 1, 2)) @ np.swapaxes(V, 1, 2)
    ge = w2[:, None, None] * (Di @ np.swapaxes(M, 1, 2))          # (n, 4, 3)
    g = np.zeros((bar.n_verts, 3))
    np.add.at(g, bar.tets.ravel(), ge.reshape(-1, 3))
    # A = sum of w2 Di Di^T over the free vertices; A y = g by conjugate gradients, restarted
    idx = -np.ones(bar.n_verts, dtype=np.int64)
    idx[free] = np.arange(free.size)
    fi = idx[bar.tets]
    Ke = w2[:, None, None] * (Di @ np.swapaxes(Di, 1, 2))
    rows, cols = np.repeat(fi, 4, axis=1).ravel(), np.tile(fi, (1, 4)).ravel()
    keep = (rows >= 0) & (cols >= 0)
    A = torch.sparse_coo_tensor(np.stack([rows[keep], cols[keep]]), torch.from_numpy(Ke.ravel()[keep]),
                                (free.size, free.size)).coalesce().to_sparse_csr()
    diag = np.bincount(rows[keep & (rows == cols)], weights=Ke.ravel()[keep & (rows == cols)], minlength=free.size)
    inv = torch.from_numpy(1.0 / diag)[:, None]
    b = torch.from_numpy(g[free])
    y = torch.zeros_like(b)
    for _ in range(3):
        r = b - A @ y
        z = inv * r
        p, rz, d = z.clone(), (r * z).sum(0), torch.zeros_like(b)
        stop = 1e-12 * r.norm()
        for _ in range(3000):
            Ap = A @ p
            a = rz / (p * Ap).sum(0).clamp_min(1e-300)
            d += a * p
            r -= a * Ap
            if r.norm() <= stop:
                break
            z = inv * r
            rz, old = (r * z).sum(0), rz
            p = z + (rz / old.clamp_min(1e-300)) * p
        y += d
    return dict(value=value, grad=g[free], step=y.numpy())


def _exact_train(case, seed):
    """The network's loss and gradient in 64 bits; an epoch of updates has no such value."""
    X, T = _pairs(case, seed)
    blob = torch.from_numpy(prox_net.init_blob(X, T, seed).astype(np.float64))
    n = min(case["batch"], case["samples"])
    x, t = torch.from_numpy(X[:n].astype(np.float64)), torch.from_numpy(T[:n].astype(np.float64))
    w = blob[16:].clone().requires_grad_(True)
    w1, b1, w2, b2, w3, b3 = torch.split(w, [320, 64, 4096, 64, 192, 3])
    h = torch.nn.functional.gelu(((x - blob[0:5]) * blob[5:10]) @ w1.view(64, 5).T + b1, approximate="tanh")
    h = torch.nn.functional.gelu(h @ w2.view(64, 64).T + b2, approximate="tanh")
    y = h @ w3.view(3, 64).T + b3
    loss = ((y - (t - x[:, :3]) / blob[10:13]) ** 2).mean()
    loss.backward()
    return dict(loss=loss.item(), grad=w.grad.numpy(), losses=None, blob=None)
