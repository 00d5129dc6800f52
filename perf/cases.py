"""The work whose speed this framework is measured by, as its users call it.

A case is a dict of plain values whose "kind" names the public call it makes:

* "conj_grad": Session.conj_grad on host vectors -- the reference's own call;
* "solve": Session.power_iterate on a resident matrix, in each solver mode;
* "batch": Batch.solve on many independent systems of uneven size;
* "train": Gnn.loss_grad, the forward and backward pass of the network;
* "mg": Mg.run, the multigrid benchmark's timed region;
* "ft": Ft.run, the Fourier transform benchmark's timed region.

The matrices have the structure of the benchmark's generator: a sum of n
weighted outer products of random sparse vectors plus a shifted diagonal.  They
are made here on the GPU from the seed alone, and handed over as host CSR
arrays, as a user's program has them.

The Mg and Ft objects generate their own right-hand side and field.  What a
user does choose is the smoother and the grid's shape, so those come from the
seed here.  The EP and IS benchmarks take no input but their size, so no case
can give them other inputs for another seed; they are not listed.

Left out of the outputs: rnorm, p and q of a solve that has converged, because
they hold rounding noise of about 1e-15 that no two orders of summation share;
and iteration counts where a tolerance stops the solve, which a last-bit
difference may move by one.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "npb-gpu_b200"))
import npbcg  # noqa: E402

RCOND = 0.1
MODES = {"fp64": npbcg.MODE_FP64, "fp64_tol": npbcg.MODE_FP64_TOL, "mixed": npbcg.MODE_MIXED,
         "learned": npbcg.MODE_MIXED_LEARNED}
AXIS_ORDERS = [(0, 1, 2), (1, 2, 0), (2, 0, 1)]


def listed():
    return [
        # One call of the reference's conj_grad at its smallest class: launch latency and
        # host copies, as a program that keeps the reference's outer loop calls it.
        dict(name="conj_grad n1400", kind="conj_grad", n=1400, nonzer=7, shift=10.0),
        # The benchmark's class A, FP64, the reference algorithm: a matrix that fits in L2.
        dict(name="solve fp64 n14000", kind="solve", mode="fp64", n=14000, nonzer=11, shift=20.0, niter=15, tol=0.0),
        # Class B: the headline benchmark.
        dict(name="solve fp64 n75000", kind="solve", mode="fp64", n=75000, nonzer=13, shift=60.0, niter=75, tol=0.0),
        # Class C: the matrix is three times the L2.
        dict(name="solve fp64 n150000", kind="solve", mode="fp64", n=150000, nonzer=15, shift=110.0, niter=75, tol=0.0),
        # Class C with the mixed-precision solver, the fastest way to the same zeta.
        dict(name="solve mixed n150000", kind="solve", mode="mixed", n=150000, nonzer=15, shift=110.0, niter=75, tol=1e-12),
        # Class B with the learned preconditioner at its configuration's tolerance.
        dict(name="solve learned n75000", kind="solve", mode="learned", n=75000, nonzer=13, shift=60.0, niter=75, tol=1e-10),
        # Many small systems at once, sizes as in the uneven batch workload.
        dict(name="batch fp64 128", kind="batch", mode="fp64", systems=128, n_low=1400, n_high=20000, niter=15, tol=0.0),
        # One training step's loss and gradients on a class A sized matrix.
        dict(name="train n14000", kind="train", n=14000, nonzer=11, shift=20.0),
        # Multigrid on the smallest class's grid and on class C's.  (Fewer cycles than class C runs:
        # with the stronger smoother, 20 would bring the residual down to rounding noise.)
        dict(name="mg 32", kind="mg", lt=5, nit=4),
        dict(name="mg 512", kind="mg", lt=9, nit=6),
        # The Fourier transform at class W's and class B's shapes.
        dict(name="ft 128x128x32", kind="ft", nx=128, ny=128, nz=32, niter=6),
        dict(name="ft 512x256x256", kind="ft", nx=512, ny=256, nz=256, niter=20),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["conj_grad", "solve", "solve", "solve", "batch", "train", "mg", "ft"])
    nonzer = rng.randint(7, 15)
    if kind == "conj_grad":
        n = _log_int(rng, 1400, 75000)
        return dict(kind=kind, n=n, nonzer=nonzer, shift=10.0 + n / 1500.0)
    if kind == "solve":
        n, mode = _log_int(rng, 1400, 150000), rng.choice(sorted(MODES))
        tol = {"fp64": 0.0, "learned": 1e-10}.get(mode, rng.choice([1e-10, 1e-11, 1e-12]))
        return dict(kind=kind, mode=mode, n=n, nonzer=nonzer, shift=10.0 + n / 1500.0, niter=rng.randint(10, 75), tol=tol)
    if kind == "batch":
        mode = rng.choice(["fp64", "mixed"])
        return dict(kind=kind, mode=mode, systems=_log_int(rng, 8, 160), n_low=1400, n_high=_log_int(rng, 4000, 20000),
                    niter=rng.randint(5, 15), tol=1e-12 if mode == "mixed" else 0.0)
    if kind == "train":
        n = _log_int(rng, 3000, 40000)
        return dict(kind=kind, n=n, nonzer=rng.randint(7, 13), shift=10.0 + n / 1500.0)
    if kind == "mg":
        return dict(kind=kind, lt=rng.randint(4, 9), nit=rng.randint(2, 8))
    sides = [1 << rng.randint(5, 10) for _ in range(3)]
    while math.prod(sides) > 1 << 26 or sides[0] == sides[1] == sides[2]:
        sides = [1 << rng.randint(5, 10) for _ in range(3)]
    return dict(kind="ft", nx=sides[0], ny=sides[1], nz=sides[2], niter=rng.randint(3, 20))


# ------------------------------------------------------------------ the inputs
def _matrix(n, nonzer, shift, seed):
    """(rowstr, colidx, a) on the GPU: sum_i w_i v_i v_i^T + (rcond - shift) I, v_i with nonzer
    random entries in (0, 1) and 0.5 at i, w_i falling geometrically from 1 to rcond.  Products
    are whole multiples of 2^-48, so that their sum does not depend on its order."""
    g = torch.Generator("cuda").manual_seed(seed)
    pos = torch.randint(n, (n, nonzer), generator=g, device="cuda")
    val = torch.rand((n, nonzer), generator=g, device="cuda", dtype=torch.float64)
    own = torch.arange(n, device="cuda")[:, None]
    pos = torch.cat([pos, own], 1)
    val = torch.cat([val, torch.full((n, 1), 0.5, device="cuda", dtype=torch.float64)], 1)
    w = torch.pow(RCOND, own / n)[:, :, None]
    prod = torch.round(w * val[:, :, None] * val[:, None, :] * 2.0 ** 48).to(torch.int64).reshape(-1)
    key = (pos[:, :, None] * n + pos[:, None, :]).reshape(-1)
    del val, w
    key, inverse = torch.unique(key, return_inverse=True)
    a = torch.zeros(key.numel(), dtype=torch.int64, device="cuda").index_add_(0, inverse, prod).double() * 2.0 ** -48
    rows, cols = key // n, key % n
    a[rows == cols] += RCOND - shift
    rowstr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rowstr[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return rowstr.int(), cols.int(), a


def _to_host(matrix):
    return tuple(t.cpu().numpy() for t in matrix)


def _host_vector(n, seed):
    """A positive start vector as conj_grad gets it: n + 1 entries near one."""
    return 0.5 + np.random.RandomState(seed % (1 << 31)).random_sample(n + 1)


def _batch_specs(case, seed):
    """(n, nonzer, shift, seed) of each system: n log-uniform in the case's range, nonzer 7 to 13."""
    rng = np.random.RandomState(seed % (1 << 31))
    low, high = math.log(case["n_low"]), math.log(case["n_high"])
    sizes = np.exp(low + (high - low) * (np.arange(case["systems"]) + 0.5) / case["systems"]).round().astype(int)
    rng.shuffle(sizes)
    return [(int(n), int(rng.randint(7, 14)), 10.0 + n / 1000.0, int(rng.randint(1 << 30))) for n in sizes]


def _probes(n, seed):
    g = torch.Generator("cuda").manual_seed(seed + 1)
    return torch.randn((n, 32), generator=g, device="cuda").cpu().numpy()


def _ft_shape(case, seed):
    sides = (case["nx"], case["ny"], case["nz"])
    return tuple(sides[k] for k in AXIS_ORDERS[seed % 3])


def prepare(case, seed):
    kind, s = case["kind"], dict(case=case)
    if kind in ("conj_grad", "solve", "train"):
        csr = _to_host(_matrix(case["n"], case["nonzer"], case["shift"], seed))
    if kind == "conj_grad":
        s.update(session=npbcg.Session(*csr), x=_host_vector(case["n"], seed))
    elif kind == "solve":
        s["session"] = npbcg.Session(*csr)
        if case["mode"] == "learned":
            net = npbcg.Gnn()
            net.load()
            with net.graph(*csr) as graph:
                net.attach(graph, s["session"])
            net.close()
    elif kind == "batch":
        specs = _batch_specs(case, seed)
        s["batch"] = npbcg.Batch([_to_host(_matrix(*spec)) for spec in specs], [spec[2] for spec in specs])
    elif kind == "train":
        s["net"] = npbcg.Gnn()
        s["net"].load()
        s.update(graph=s["net"].graph(*csr), probes=_probes(case["n"], seed))
    elif kind == "mg":
        s["mg"] = npbcg.Mg(case["lt"], seed % 2)
    else:
        s["ft"] = npbcg.Ft(*_ft_shape(case, seed))
    return s


# ------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "conj_grad":
        z, _, _, r, _ = state["session"].conj_grad(state["x"])
        return dict(z=z, r=r)
    if kind == "solve":
        mode = MODES[case["mode"]]
        tol = {} if case["mode"] == "fp64" else dict(tol=case["tol"], cgitmax=100)
        got = state["session"].power_iterate(case["niter"], case["shift"], mode=mode, want_x=True, **tol)
        out = dict(zeta=got["zeta"], x=got["x"])
        if case["mode"] == "fp64":
            out["iters"] = got["iters"]
        return out
    if kind == "batch":
        tol = {} if case["mode"] == "fp64" else dict(tol=case["tol"], cgitmax=100)
        got = state["batch"].solve(niter=case["niter"], mode=MODES[case["mode"]], **tol)
        return dict(zeta=got["zeta"], status=got["status"])
    if kind == "train":
        loss, grad = state["net"].loss_grad(state["graph"], state["probes"])
        return dict(loss=np.array([loss], np.float32), grad=grad)
    if kind == "mg":
        got = state["mg"].run(case["nit"])
        return dict(norms=np.array([got["rnm2"], got["rnmu"]]))
    return dict(sums=np.array(state["ft"].run(case["niter"])["sums"]))


# ------------------------------------------------------------------ what a pass cannot do without
def _entries(n, nonzer):
    """Stored entries of a matrix: outer products of nonzer + 1 entries, their diagonals in common."""
    return n * ((nonzer + 1) ** 2 - nonzer)


def _solve_work(n, nnz, niter, mode, tol):
    """A step reads the matrix once for each of its products, and each product's vectors."""
    if mode == "fp64":
        products, value = 26, 8
    else:  # about one iteration for each digit and a half after the start on earlier iterates
        products, value = 2 + max(1.0, -math.log10(tol)) / 4, 8 if mode == "fp64_tol" else 4
    each = (value + 4) * nnz + 4 * (n + 1) + 16 * n
    return dict(bytes=niter * products * each, flops=niter * products * 2.0 * nnz)


def work(case):
    kind = case["kind"]
    if kind == "conj_grad":
        return _solve_work(case["n"], _entries(case["n"], case["nonzer"]), 1, "fp64", 0.0)
    if kind == "solve":
        return _solve_work(case["n"], _entries(case["n"], case["nonzer"]), case["niter"], case["mode"], case["tol"])
    if kind == "batch":
        low, high = case["n_low"], case["n_high"]
        n = (high - low) / math.log(high / low) * case["systems"]
        return _solve_work(n, n * 112.0, case["niter"], case["mode"], case["tol"])
    if kind == "train":
        # the scaled matrix in FP32 with its columns, and 32 channels a row, once for each of the
        # three layers and the three products with probes, forward and backward
        n, nnz = case["n"], _entries(case["n"], case["nonzer"])
        return dict(bytes=12 * (8.0 * nnz + 2 * 128.0 * n), flops=12 * 64.0 * nnz)
    if kind == "mg":
        # a cycle on the finest grid reads u and v and writes u, then reads u and v and writes r;
        # the coarser grids add a seventh
        points = 8.0 ** case["lt"] * 8 / 7
        return dict(bytes=case["nit"] * 6 * 8 * points, flops=case["nit"] * 58 * points)
    # the transform of a field beyond the caches takes two passes over it
    points = case["nx"] * case["ny"] * case["nz"]
    return dict(bytes=(case["niter"] + 1) * 64.0 * points, flops=(case["niter"] + 1) * 5.0 * points * math.log2(points))


def tolerance(case):
    """About four times what each call is off its 64-bit value, or by the solver's own tolerance."""
    kind = case["kind"]
    if kind in ("solve", "batch") and case["tol"]:
        return dict(rel=20 * case["tol"])  # seen: 2 tol
    if kind == "batch":
        return dict(rel=2.5e-11)  # seen: 6.4e-12; some of the systems are indefinite
    if kind == "train":
        return dict(rel=1.5e-5)  # seen: 3.5e-6
    if kind == "mg":  # rounding of the right-hand side's size, while a cycle takes the residual down up to five-fold
        return dict(rel=4e-15 * 5 ** case["nit"])
    return dict(rel=1e-13)  # seen: 4e-16; sums of up to 75000 terms in another order


# ------------------------------------------------------------------ the same in 64 bits
def _csr(matrix):
    rowstr, cols, a = matrix
    n = rowstr.numel() - 1
    return torch.sparse_csr_tensor(rowstr, cols, a, size=(n, n))


def _cg(A, x, steps=None):
    """conj_grad from z = 0: a fixed number of steps, or until the residual is rounding."""
    z, r, p = torch.zeros_like(x), x.clone(), x.clone()
    rho = first = torch.dot(r, r)
    for k in range(steps or 200):
        q = A @ p
        alpha = rho / torch.dot(p, q)
        z, r = z + alpha * p, r - alpha * q
        last, rho = rho, torch.dot(r, r)
        if not steps and float(rho) < 1e-30 * float(first):
            break
        p = r + (rho / last) * p
    return z


def _power(A, n, shift, niter, steps):
    x, zeta = torch.ones(n, dtype=torch.float64, device="cuda"), []
    for _ in range(niter):
        z = _cg(A, x, steps)
        zeta.append(shift + 1.0 / torch.dot(x, z))
        x = z / z.norm()
    return torch.stack(zeta), x


def _exact_train(case, seed):
    n = case["n"]
    rowstr, cols, a = _matrix(n, case["nonzer"], case["shift"], seed)
    cols = cols.long()
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), torch.diff(rowstr.long()))
    flat = np.fromfile(os.path.join(ROOT, "npb-gpu_b200", "npbcg", "lp_weights.f32"), dtype="<f4")
    flat = torch.from_numpy(flat.astype(np.float64)).cuda().requires_grad_(True)
    sizes = [(4, 32), (32,)] + [(32, 32), (32, 32), (32,)] * 3 + [(32,), (1,), (32,), (1,)]
    parts = [p.reshape(s) for p, s in zip(torch.split(flat, [math.prod(s) for s in sizes]), sizes)]
    diagonal = rows == cols
    delta = (-a[diagonal]).mean()
    ahat = -a / delta
    off, low = ~diagonal, cols < rows
    ro, co, ao, rl, cl, al = rows[off], cols[off], ahat[off], rows[low], cols[low], ahat[low]
    spread = lambda src: torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, ro, src)  # noqa: E731
    degree = spread(torch.ones_like(ao))
    features = torch.stack([ahat[diagonal], spread(ao.abs()), spread(ao), degree / degree.mean().clamp(min=1.0)], 1)

    def product(r, c, v, X):  # rows r of the result gather rows c of X, in slabs that fit the memory
        out = torch.zeros_like(X)
        for k in range(0, r.numel(), 1 << 21):
            at = slice(k, k + (1 << 21))
            out = out.index_add(0, r[at], v[at, None] * X[c[at]])
        return out

    h = torch.relu(features @ parts[0] + parts[1])
    for l in range(3):
        own, message, bias = parts[2 + 3 * l: 5 + 3 * l]
        h = torch.relu(h @ own + product(ro, co, ao, h @ message) + bias)
    w_d, c_d, w_e, c_e = parts[11:]
    gdiag = torch.nn.functional.softplus(h @ w_d + c_d)
    goff = al * ((h[rl] * h[cl]) @ w_e + c_e)
    R = torch.from_numpy(_probes(n, seed)).cuda().double()
    T = product(rl, cl, goff, R) + gdiag[:, None] * R
    U = product(cl, rl, goff, T) + gdiag[:, None] * T
    W = product(ro, co, ao, U) + ahat[diagonal][:, None] * U - R
    loss = ((W * W).sum(0) / (R * R).sum(0)).mean()
    loss.backward()
    return dict(loss=loss.detach()[None], grad=flat.grad)


def _lcg(count, first=0):
    """Draws first + 1 to first + count of the benchmark's stream, as whole numbers below 2^46."""
    mask, mult = (1 << 46) - 1, pow(5, 13)
    x = torch.empty(count, dtype=torch.int64, device="cuda")
    x[0] = 314159265 * pow(mult, first + 1, 1 << 46) & mask
    have = 1
    while have < count:
        more = min(have, count - have)
        x[have: have + more] = x[:more] * pow(mult, have, 1 << 46) & mask
        have += more
    return x


def _exact_mg(case, smoother):
    lt, side = case["lt"], 1 << case["lt"]
    draws = _lcg(side ** 3)
    v = torch.zeros(side ** 3, dtype=torch.float64, device="cuda")
    v[torch.topk(draws, 10).indices], v[torch.topk(draws, 10, largest=False).indices] = 1.0, -1.0
    v = v.reshape(side, side, side)
    del draws
    c0, c1, c2 = (-3 / 17, 1 / 33, -1 / 61) if smoother else (-3 / 8, 1 / 32, -1 / 64)
    both = lambda g, axis: torch.roll(g, 1, axis) + torch.roll(g, -1, axis)  # noqa: E731

    def resid(u, rhs):
        x, y = both(u, 2), both(u, 1)
        xy = both(x, 1)
        return rhs + 8 / 3 * u - (xy + both(x + y, 0)) / 6 - both(xy, 0) / 12

    def smooth(r, u):
        x, y = both(r, 2), both(r, 1)
        return u + c0 * r + c1 * (x + y + both(r, 0)) + c2 * (both(x, 1) + both(x + y, 0))

    def restrict(r):
        for axis in range(3):
            r = (r + 0.5 * both(r, axis)).index_select(axis, torch.arange(1, r.shape[axis], 2, device="cuda"))
        return 0.5 * r

    def prolong(z):
        for axis in range(3):
            z = torch.stack([0.5 * (z + torch.roll(z, 1, axis)), z], axis + 1).flatten(axis, axis + 1)
        return z

    u, r = torch.zeros_like(v), v
    for _ in range(case["nit"]):
        rs = {lt: r}
        for k in range(lt, 1, -1):
            rs[k - 1] = restrict(rs[k])
        z = smooth(rs[1], torch.zeros_like(rs[1]))
        for k in range(2, lt):
            z = prolong(z)
            z = smooth(resid(z, rs[k]), z)
        u = u + prolong(z)
        u = smooth(resid(u, v), u)
        r = resid(u, v)
    return dict(norms=torch.stack([r.square().mean().sqrt(), r.abs().max()]))


def _exact_ft(case, shape):
    nx, ny, nz = shape
    points = nx * ny * nz
    field = (_lcg(2 * points).double() * 2.0 ** -46).reshape(nz, ny, nx, 2)
    spectrum = torch.fft.ifftn(torch.view_as_complex(field)) * points
    del field
    k = [((torch.arange(s, device="cuda", dtype=torch.float64) + s // 2) % s - s // 2) ** 2 for s in shape]
    k2 = k[2][:, None, None] + k[1][:, None] + k[0]
    j = torch.arange(1, 1025, device="cuda")
    sums = []
    for t in range(1, case["niter"] + 1):
        u = torch.fft.fftn(spectrum * torch.exp(-4e-6 * math.pi ** 2 * t * k2))
        total = u[5 * j % nz, 3 * j % ny, j % nx].sum() / points
        sums.append(torch.view_as_real(total))
        del u
    return dict(sums=torch.stack(sums))


def exact(case, seed):
    kind = case["kind"]
    if kind == "conj_grad":
        A = _csr(_matrix(case["n"], case["nonzer"], case["shift"], seed))
        z = _cg(A, torch.from_numpy(_host_vector(case["n"], seed)[:-1]).cuda(), 25)
        # the call's arrays have one entry more than the system, which the products leave alone
        last = torch.from_numpy(_host_vector(case["n"], seed)[-1:]).cuda()
        return dict(z=torch.cat([z, z.new_zeros(1)]), r=torch.cat([A @ z, last]))
    if kind == "solve":
        A = _csr(_matrix(case["n"], case["nonzer"], case["shift"], seed))
        zeta, x = _power(A, case["n"], case["shift"], case["niter"], 25 if case["mode"] == "fp64" else None)
        out = dict(zeta=zeta, x=x)
        if case["mode"] == "fp64":
            out["iters"] = np.full(case["niter"], 25, np.int32)
        return out
    if kind == "batch":
        zeta = [_power(_csr(_matrix(*spec)), spec[0], spec[2], case["niter"], 25)[0][-1] for spec in _batch_specs(case, seed)]
        return dict(zeta=torch.stack(zeta), status=None)
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "mg":
        return _exact_mg(case, seed % 2)
    return _exact_ft(case, _ft_shape(case, seed))
