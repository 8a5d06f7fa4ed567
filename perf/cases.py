"""The timed workloads of this library: what a user's program calls, over the sizes, dimensions, densities and
options it is called with.  `listed()` gives the standing ones, `draw(rng)` another of the same ranges; `prepare` builds what
the program has in hand before the call, `run` makes ONE pass through the public API, `work` counts what the pass cannot do
without, `tolerance` says how far another correct implementation may be, and `exact` computes the same outputs in 64 bits by
plain torch (a cell is cut by brute force: every edge is the interval of a line left by all the other half-spaces).

A case is a dict of plain values:
  what   "diagram"  one query of a PowerDiagram: `query` measures / moments / hessian / vjp / linear
         "solve"    OtProblem.solve, the damped Newton on the weights, from scratch
         "w2"       w2_batch and its backward on CUDA tensors
         "fit"      weights_batch and its backward (the implicit function theorem)
         "serve"    a slice of the serving stream through the Server
  d, n   dimension and number of seeds; `batch` problems ("w2", "fit") or requests ("serve")
  target "uniform" (the unit box), "gauss" (4 gaussians on it), "image" (16 gaussians on `res` x `res` pixels)
  spread the seeds' weights are uniform in [0, spread] ("diagram"; 0: none, Voronoi)
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "sdot-ffi_b200") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "sdot-ffi_b200"))

import sdot  # noqa: E402
from sdot import Iterative, OtProblem, SumOfDiracs, SumOfGaussians, Tuning  # noqa: E402

RTOL = 1e-8                     # the masses' relative tolerance of the solves, the benchmark's


def _case(name, what, d, n, target="uniform", query="", batch=1, res=0, spread=0.0):
    return dict(name=name, what=what, d=d, n=n, target=target, query=query, batch=batch, res=res, spread=spread)


def listed():
    return [
        # the smallest call: a thousand seeds, where latency and launches count
        _case("solve 2D 1000", "solve", 2, 1000),
        # the ordinary solves of the serving stream (n in [1e3, 2e5], both dimensions, both targets), odd sizes
        _case("solve 2D 100003", "solve", 2, 100003),
        _case("solve 2D gauss 20011", "solve", 2, 20011, "gauss"),
        _case("solve 3D 20000", "solve", 3, 20000),
        _case("solve 3D gauss 3001", "solve", 3, 3001, "gauss"),
        # the transport onto an image (blurred continuation)
        _case("solve 2D image 10000", "solve", 2, 10000, "image", res=128),
        # one diagram: every cell's area of a million seeds; volumes, centroids and costs under gaussians; the Newton
        # Hessian of a weighted diagram
        _case("measures 2D 1e6", "diagram", 2, 1000000, query="measures"),
        _case("moments 3D gauss 50021", "diagram", 3, 50021, "gauss", "moments"),
        _case("hessian 3D 1e5", "diagram", 3, 100000, query="hessian", spread=1e-4),
        # training on W2: 32 point clouds, the cost's gradient; and the fitted weights' gradient of one larger cloud
        _case("w2 32 x 2D 500", "w2", 2, 500, batch=32),
        _case("fit 2 x 2D 7919", "fit", 2, 7919, batch=2),
        # a slice of the serving stream: 8 requests of both dimensions and targets
        _case("serve 8", "serve", 0, 8000, "mixed", batch=8),
    ]


def _size(rng, lo, hi):
    """log-uniform in [lo, hi], mostly odd"""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | 1))


def draw(rng):
    what = rng.choice(["diagram", "diagram", "solve", "solve", "w2", "fit", "serve"])
    d = rng.choice([2, 3])
    if what == "diagram":
        query = rng.choice(["measures", "moments", "hessian", "vjp", "linear"])
        target = "uniform" if query in ("vjp", "linear") else rng.choice(["uniform", "gauss"] + (["image"] if d == 2 else []))
        top = 100000 if query == "linear" else (50000 if d == 3 and target == "gauss" else (1000000 if d == 2 else 200000))
        n = _size(rng, 1000, top)
        # (weights of up to a fifth of the spacing squared: most cells keep their seed)
        return _case("drawn", what, d, n, target, query, res=128 if target == "image" else 0,
                     spread=rng.choice([0.0, 0.2 * n ** (-2.0 / d)]))
    if what == "solve":
        target = rng.choice(["uniform", "gauss", "image"] if d == 2 else ["uniform", "gauss"])
        top = {("uniform", 2): 100000, ("uniform", 3): 20000, ("gauss", 2): 20000, ("gauss", 3): 3000, ("image", 2): 10000}[target, d]
        return _case("drawn", what, d, _size(rng, 1000, top), target, res=128 if target == "image" else 0)
    if what == "w2":
        return _case("drawn", what, d, _size(rng, 100, 1000 if d == 2 else 500), batch=rng.randrange(2, 33))
    if what == "fit":
        return _case("drawn", what, d, _size(rng, 500, 8000 if d == 2 else 3000), batch=rng.randrange(1, 3))
    return _case("drawn", what, 0, _size(rng, 2000, 8000), "mixed", batch=rng.randrange(4, 9))


# ---- the inputs ---------------------------------------------------------------------------------------------------------
def _target(rng, kind, d, res=0):
    """(distribution, its gaussians or None)"""
    if kind == "gauss":
        c, s = rng.uniform(0.2, 0.8, size=(4, d)), rng.uniform(0.05, 0.15, size=4)
        return SumOfGaussians(c, s, np.full(4, 0.25), support_box=(np.zeros(d), np.ones(d))), (c, s, np.full(4, 0.25))
    if kind == "image":
        c, s, a = rng.uniform(size=(16, 2)), rng.uniform(0.02, 0.1, size=16), rng.uniform(0.5, 2.0, size=16)
        x = (np.arange(res) + 0.5) / res
        v = sum(a[k] * np.exp(-((x[:, None] - c[k, 0]) ** 2 + (x[None, :] - c[k, 1]) ** 2) / (2 * s[k] ** 2)) for k in range(16))
        return sdot.Image(v + 0.01 * v.max(), frame=np.full(2, 1.0 / res)), None
    return sdot.Box(nb_dims=d), None


def _settings(rtol=RTOL):
    return Iterative(tol=0.0, tuning=Tuning(mass_rtol=rtol))


def _inputs(case, seed):
    """the seed's arrays (numpy), the same for `prepare` and `exact`"""
    what, d, n, B = case["what"], case["d"], case["n"], case["batch"]
    rng = np.random.default_rng([seed, d, n, B])
    if what == "serve":
        # dimension 2 (70 %) or 3, n log-uniform in [1e3, case n], uniform or gaussian targets half and half
        reqs, sizes = [], np.random.default_rng([n, B])
        for k in range(B):
            dk = 2 if sizes.uniform() < 0.7 else 3
            gauss = sizes.uniform() < 0.5
            nk = int(round(math.exp(sizes.uniform(math.log(1e3), math.log(n if dk == 2 or not gauss else max(1000.0, n / 4))))))
            reqs.append((rng.uniform(size=(nk, dk)), _target(rng, "gauss" if gauss else "uniform", dk)[0]))
        return dict(reqs=reqs)
    if what in ("w2", "fit"):
        nu = rng.uniform(0.5, 1.5, size=(B, n))
        return dict(pos=rng.uniform(size=(B, n, d)), nu=nu / nu.sum(axis=1, keepdims=True), g=rng.normal(size=(B, n)))
    pos = rng.uniform(size=(n, d))
    w = rng.uniform(0, case["spread"], size=n) if case["spread"] else None
    target, gauss = _target(rng, case["target"], d, case["res"])
    return dict(pos=pos, w=w, target=target, gauss=gauss, g=rng.normal(size=n))


def prepare(case, seed):
    what, d = case["what"], case["d"]
    A = _inputs(case, seed)
    if what == "serve":
        return dict(what=what, reqs=A["reqs"], server=sdot_server())
    if what in ("w2", "fit"):
        pos = torch.from_numpy(A["pos"]).cuda().requires_grad_(True)
        nu = torch.from_numpy(A["nu"]).cuda().requires_grad_(True)
        return dict(what=what, pos=pos, nu=nu, g=torch.from_numpy(A["g"]).cuda())
    if what == "solve":
        return dict(what=what, source=SumOfDiracs(A["pos"]), target=A["target"])
    return dict(what=what, pd=sdot.PowerDiagram(A["pos"], A["w"], boundaries=sdot.box_half_spaces(np.zeros(d), np.ones(d)),
                                                distribution=None if case["target"] == "uniform" else A["target"]),
                query=case["query"], g=A["g"], rhs=A["g"] - A["g"].mean())


_SERVER = []


def sdot_server():
    """the program's server, started once"""
    if not _SERVER:
        from sdot.server import Server
        _SERVER.append(Server())
    return _SERVER[0]


# ---- one pass -----------------------------------------------------------------------------------------------------------
def run(state):
    what = state["what"]
    if what == "solve":
        plan = OtProblem(state["source"], state["target"]).solve(_settings())
        return plan.weights, plan.cell_masses, plan.barycenters, plan.cost
    if what == "diagram":
        pd, query = state["pd"], state["query"]
        if query == "measures":
            return pd.measures
        if query == "moments":
            return pd.barycenters_and_costs()
        if query == "hessian":
            return pd.hessian_rows()
        if query == "vjp":
            return pd.measures_vjp(state["g"])
        return pd.laplacian_solve(state["rhs"])
    if what == "serve":
        srv = state["server"]
        tickets = [srv.submit(pos, target, settings=_settings()) for pos, target in state["reqs"]]
        done = [srv.result(t) for t in tickets]
        return [(r["weights"], r["masses"], r["barycentres"], r["cost"]) for r in done]
    from sdot import torch_ops
    pos, nu = state["pos"], state["nu"]
    pos.grad = nu.grad = None
    if what == "w2":
        out = torch_ops.w2_batch(pos, nu)
        out.sum().backward()
    else:
        out = torch_ops.weights_batch(pos, nu)
        (out * state["g"]).sum().backward()
    return out.detach(), pos.grad, nu.grad


# ---- what a pass cannot do without --------------------------------------------------------------------------------------
def work(case):
    """each input read once and each output written once; the operations of building and integrating each cell ONCE (a
    Newton solve builds it tens of times), from the cell's average 6 edges (2D) or 16 faces, 27 vertices (3D)"""
    what, d, n, B = case["what"], case["d"], case["n"], case["batch"]
    cell = 6 * 45 if d == 2 else 16 * 10 + 27 * 60 + 81 * 40
    if case["target"] == "gauss":          # 4 gaussians, an edge's 8 quadrature points of an exponential and an error function
        cell += (6 if d == 2 else 81) * 4 * 8 * 60
    if what == "serve":
        n, B, d = 3 * n / 8, B, 2
        return {"bytes": B * n * 8.0 * (2 + 5), "flops": B * n * (0.7 * (6 * 45) + 0.3 * 5000 + 0.5 * 6 * 4 * 8 * 60)}
    if what == "solve":
        return {"bytes": n * 8.0 * (d + 1 + 2 + d), "flops": float(n * cell)}
    if what in ("w2", "fit"):
        return {"bytes": B * n * 8.0 * (2 * (d + 1) + 1), "flops": float(B * n * cell)}
    out = {"measures": 1, "moments": 2 + d, "hessian": 0.5 + 1.5 * (6 if d == 2 else 16), "vjp": 2 + d, "linear": 2}[case["query"]]
    return {"bytes": n * 8.0 * (d + 1 + out), "flops": float(n * cell)}


def tolerance(case):
    """64-bit sums of cells cut in 64 bits, and fixed points of a Newton stopped at 1e-8 on the masses"""
    what = case["what"]
    if what == "diagram":
        if case["query"] == "linear":
            return {"rel": 1e-8, "max": 1e-7}
        if case["target"] == "gauss" and case["query"] == "moments":     # (the centroid of a cell in the gaussians' far tail)
            return {"rel": 1e-9, "max": 1e-5}
        return {"rel": 1e-11, "max": 1e-8, "differ": 1e-6}
    if what == "w2":
        return {"rel": 1e-8, "max": 1e-6}
    if what == "fit":
        return {"rel": 1e-7, "max": 1e-5}
    return {"rel": 1e-6, "max": 1e-4}


# ---- the outputs in 64 bits by plain torch ----------------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _candidates(p, w, rows, K):
    """the K seeds whose bisectors are nearest each of the `rows` [m, K], and how far every other one's is at least [m]"""
    n, d = p.shape
    out = torch.empty(len(rows), K, dtype=torch.long, device=p.device)
    beyond = torch.empty(len(rows), dtype=p.dtype, device=p.device)

    def nearest(at, cand, ok, bound):
        i = rows[at]
        q = p[cand] - p[i, None]
        l2 = (q * q).sum(-1)
        s = torch.where(ok & (l2 > 0), (l2 + w[i, None] - w[cand]) / (2 * l2.sqrt()), torch.inf)
        s, k = torch.topk(s, K, dim=1, largest=False)
        out[at], beyond[at] = torch.gather(cand, 1, k), torch.minimum(s[:, -1], bound)

    if n <= 30000:
        every = torch.arange(n, device=p.device)
        for a in range(0, len(rows), 1024):
            at = slice(a, min(len(rows), a + 1024))
            cand = every.expand(at.stop - a, n)
            nearest(at, cand, torch.ones_like(cand, dtype=torch.bool), torch.full((at.stop - a,), torch.inf).to(p))
        return out, beyond
    g = max(1, int((n / 2) ** (1 / d)))              # a grid of two seeds a cell; the candidates of a window of its cells
    c = (p * g).long().clamp(0, g - 1)
    key = sum(c[:, a] * g ** a for a in range(d))
    count = torch.bincount(key, minlength=g ** d)
    order = torch.argsort(key, stable=True)
    first = torch.cumsum(count, 0) - count
    cap = int(count.max())
    table = torch.full((g ** d, cap), -1, dtype=torch.long, device=p.device)
    table[key[order], torch.arange(n, device=p.device) - first[key[order]]] = order
    r = 5 if d == 2 else 4
    D = r / g                                        # (a seed outside the window is at least this far)
    bound = (D * D + w - w.max()) / (2 * D)
    off = torch.cartesian_prod(*[torch.arange(-r, r + 1, device=p.device)] * d)
    step = max(1, int(1e8 / (len(off) * cap)))
    for a in range(0, len(rows), step):
        at = slice(a, min(len(rows), a + step))
        cc = c[rows[at], None] + off
        ok = ((cc >= 0) & (cc < g)).all(-1)
        k = sum(cc[..., b].clamp(0, g - 1) * g ** b for b in range(d))
        cand = torch.where(ok[..., None], table[k], -1).reshape(at.stop - a, -1)
        nearest(at, cand.clamp(min=0), cand >= 0, bound[rows[at]])
    return out, beyond


class _Cells:
    """every cell in the unit box: its facets (ids, distance of the seeds, measure, first moment about the seed [n, F]), its
    mass, first moment about the seed and int |x - p|^2.  `ok`: no seed left out could cut a cell"""

    def __init__(self, p, w, gauss=None):
        n, d = p.shape
        new = lambda *s: torch.zeros(n, *s, dtype=p.dtype, device=p.device)  # noqa: E731
        self.mass, self.first, self.cost = new(), new(d), new()
        F = 24 if d == 2 else 64
        self.ids, self.dist, self.meas, self.cen = new(F).long(), new(F) + 1, new(F), new(F, d)
        side = torch.cat([-torch.eye(d, dtype=p.dtype, device=p.device), torch.eye(d, dtype=p.dtype, device=p.device)])
        rows = torch.arange(n, device=p.device)
        for K in (24, 64, 200) if d == 2 else (40, 80, 240):       # the few cells that a wider ring could cut are done again
            K = min(K, n - 1)
            step = max(1, int(6e7 / (K + 2 * d) ** d))
            ids, beyond = _candidates(p, w, rows, K)
            left = []
            for a in range(0, len(rows), step):
                i = rows[a:a + step]
                nb = ids[a:a + step]
                q = p[nb] - p[i, None]
                ln = (q * q).sum(-1).sqrt()
                N = torch.cat([q / ln[..., None], side.expand(len(i), 2 * d, d)], 1)
                O = torch.cat([(ln * ln + w[i, None] - w[nb]) / (2 * ln), p[i], 1 - p[i]], 1)
                R, meas, cen, self.mass[i], self.first[i], self.cost[i] = self._two(N, O, p[i], gauss) if d == 2 else self._three(N, O)
                meas = meas[:, :K].clamp(min=0)
                top = torch.topk(meas, min(F, K), dim=1)[1]
                m = top.shape[1]
                self.ids[i, :m], self.dist[i, :m], self.meas[i, :m] = nb.gather(1, top), ln.gather(1, top), meas.gather(1, top)
                self.cen[i, :m] = cen.gather(1, top[..., None].expand(-1, -1, d))
                left.append(i[(R > beyond[a:a + step]) & (K < n - 1)])
            rows = torch.cat(left)
            if not len(rows):
                break
        self.ok = len(rows) == 0

    @staticmethod
    def _interval(a, b, skip):
        """{t : a t <= b} over the last axis"""
        eps = 1e-13
        t = b / a
        hi = torch.where((a > eps) & ~skip, t, torch.inf).min(-1)[0]
        lo = torch.where((a < -eps) & ~skip, t, -torch.inf).max(-1)[0]
        none = ((a.abs() <= eps) & ~skip & (b < 0)).any(-1)
        good = (hi > lo) & ~none & torch.isfinite(hi) & torch.isfinite(lo)
        return torch.where(good, lo, 0.0), torch.where(good, hi, 0.0)

    def _two(self, N, O, p, gauss):
        F = N.shape[1]
        T = torch.stack([-N[..., 1], N[..., 0]], -1)
        X = O[..., None] * N
        a = torch.einsum("ikc,ijc->ijk", N, T)
        b = O[:, None, :] - torch.einsum("ikc,ijc->ijk", N, X)
        lo, hi = self._interval(a, b, torch.eye(F, dtype=torch.bool, device=N.device)[None])
        A, B = X + lo[..., None] * T, X + hi[..., None] * T
        ln = hi - lo
        if gauss is None:
            c = O * ln / 2
            got = (ln, (A + B) / 2 * ln[..., None], c.sum(1), ((A + B) / 3 * c[..., None]).sum(1),
                   (((A * A).sum(-1) + (A * B).sum(-1) + (B * B).sum(-1)) / 6 * c).sum(1))
        else:
            # int rho = closed integral of G dy, G = int_{-inf}^x rho; the moments from x rho's and x^2 rho's own primitives
            gx, gw = (torch.from_numpy(v).to(N) for v in np.polynomial.legendre.leggauss(16))
            Y = (A[..., None, :] + (B - A)[..., None, :] * (0.5 + 0.5 * gx)[:, None])
            W = 0.5 * gw * ln[..., None]
            m = torch.zeros_like(W)
            fx, x2, rho = torch.zeros_like(W), torch.zeros_like(W), torch.zeros_like(W)
            for c, sg, mg in zip(*gauss):
                u = Y + p[:, None, None] - torch.from_numpy(c).to(N)
                e = mg / (2 * math.pi * sg * sg) * torch.exp(-(u * u).sum(-1) / (2 * sg * sg))
                G = 0.5 * mg / (sg * math.sqrt(2 * math.pi)) * torch.exp(-u[..., 1] ** 2 / (2 * sg * sg)) * torch.erfc(-u[..., 0] / (sg * math.sqrt(2)))
                cx = (Y - u)[..., 0]                 # the centre, seed frame
                m, rho = m + G, rho + e
                fx = fx + cx * G - sg * sg * e
                x2 = x2 + (cx * cx + sg * sg) * G - sg * sg * (Y[..., 0] + cx) * e
            dy = W * T[..., 1:2]
            got = ((W * rho).sum(-1), ((W * rho)[..., None] * Y).sum(-2), (m * dy).sum((1, 2)),
                   torch.stack([(fx * dy).sum((1, 2)), (Y[..., 1] * m * dy).sum((1, 2))], -1),
                   ((x2 + Y[..., 1] ** 2 * m) * dy).sum((1, 2)))
        return torch.where(ln > 0, torch.maximum((A * A).sum(-1), (B * B).sum(-1)), 0.0).max(1)[0].sqrt(), *got

    def _three(self, N, O):
        F = N.shape[1]
        eye = torch.eye(F, dtype=torch.bool, device=N.device)
        dot = torch.einsum("ijc,ikc->ijk", N, N)
        D = torch.cross(N[:, :, None].expand(-1, F, F, 3), N[:, None].expand(-1, F, F, 3), dim=-1)     # along the edge of faces j, k
        sn2 = (D * D).sum(-1).clamp(min=1e-300)
        al, be = (O[:, :, None] - dot * O[:, None, :]) / sn2, (O[:, None, :] - dot * O[:, :, None]) / sn2
        X = al[..., None] * N[:, :, None] + be[..., None] * N[:, None]
        a = torch.einsum("ilc,ijkc->ijkl", N, D)
        b = O[:, None, None, :] - torch.einsum("ilc,ijkc->ijkl", N, X)
        lo, hi = self._interval(a, b, eye[:, None, :] | eye[None, :, :])
        flat = eye[None] | (sn2 < 1e-20)
        lo, hi = torch.where(flat, 0.0, lo), torch.where(flat, 0.0, hi)
        A, B = X + lo[..., None] * D, X + hi[..., None] * D
        sn = sn2.sqrt()
        tri = (O[:, None, :] - dot * O[:, :, None]) / sn * (hi - lo) * sn / 2            # the triangle (foot of face j, edge jk)
        foot = (O[..., None] * N)[:, :, None]
        S = foot + A + B
        v = tri * O[:, :, None] / 3
        sq = (foot * foot).sum(-1) + (A * A).sum(-1) + (B * B).sum(-1) + (S * S).sum(-1)
        R = torch.where(hi > lo, torch.maximum((A * A).sum(-1), (B * B).sum(-1)), 0.0).amax((1, 2)).sqrt()
        return R, tri.sum(2), (tri[..., None] * S / 3).sum(2), v.sum((1, 2)), (v[..., None] * S / 4).sum((1, 2)), (v * sq / 20).sum((1, 2))

    def coef(self):
        """int_facet / 2 |p_i - p_j| [n, F]"""
        return self.meas / (2 * self.dist)

    def solve(self, rhs, tol=1e-14):
        """one solution of L x = rhs (of zero sum), by elimination or the conjugate gradient"""
        c = self.coef()
        dia = c.sum(1)
        n = len(dia)
        if n <= 4000:
            M = torch.diag(dia).scatter_add_(1, self.ids, -c) + dia.mean() / n
            return torch.linalg.solve((M + M.T) / 2, rhs - rhs.mean())
        apply = lambda x: dia * x - (c * x[self.ids]).sum(1)  # noqa: E731
        x, r = torch.zeros_like(rhs), rhs - rhs.mean()
        z = r / dia
        q, rz, stop = z.clone(), (r * z).sum(), tol * r.norm()
        for _ in range(20000):
            Aq = apply(q)
            al = rz / (q * Aq).sum()
            x, r = x + al * q, r - al * Aq
            if r.norm() <= stop:
                break
            z = r / dia
            rz, old = (r * z).sum(), rz
            q = z + rz / old * q
        return x


def _newton(p, nu):
    """the weights whose cells have the masses nu (gauge w[0] = 0): (w, its cells); None where a cell empties on the way"""
    w = torch.zeros_like(nu)
    C = _Cells(p, w)
    for _ in range(60):
        e = nu - C.mass
        if not C.ok or float((e.abs() / nu).max()) < 2e-13:
            break
        dw, t = C.solve(e), 1.0
        while t > 1e-3:
            N = _Cells(p, w + t * dw)
            if N.mass.min() > 0.1 * min(float(nu.min()), float(C.mass.min())) and (nu - N.mass).norm() < e.norm():
                break
            t /= 2
        if t <= 1e-3:                                # at the rounding of the masses
            break
        w, C = w + t * dw, N
    return (w - w[0], C) if C.ok and float(((nu - C.mass).abs() / nu).max()) < 1e-11 else (None, None)


def _vjp(C, g, p):
    """the adjoint of the masses: grad p [n, d], grad w [n]"""
    dg = g[:, None] - g[C.ids]
    return ((dg / C.dist)[..., None] * C.cen).sum(1), (C.coef() * dg).sum(1)


def exact(case, seed):
    what, d, n = case["what"], case["d"], case["n"]
    if what == "serve" or case["target"] == "image" or (case["target"] == "gauss" and (d == 3 or what == "solve")):
        return None
    if case["query"] == "hessian" or (what in ("solve", "w2", "fit") and n > (20000 if d == 2 else 3000)):
        return None                                  # (the order of a row's neighbours is the library's)
    A = _inputs(case, seed)
    dev = _dev()
    T = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(dev)  # noqa: E731
    if what in ("w2", "fit"):
        outs = []
        for b in range(case["batch"]):
            p, nu = T(A["pos"][b]), T(A["nu"][b])
            w, C = _newton(p, nu)
            if w is None:
                return None
            if what == "w2":
                outs.append((C.cost.sum(), -2 * C.first, w - w.mean()))
            else:
                g = T(A["g"][b])
                rhs = g.clone()
                rhs[0] -= g.sum()
                lam = C.solve(rhs)
                gp = -_vjp(C, lam, p)[0]
                outs.append((w, gp, lam - (nu * lam).sum()))
        return tuple(torch.stack(x) for x in zip(*outs))
    p = T(A["pos"])
    if what == "solve":
        w, C = _newton(p, torch.full((n,), 1.0 / n, dtype=torch.float64, device=dev))
        return None if w is None else (w, C.mass, p + C.first / C.mass[:, None], float(C.cost.sum()))
    C = _Cells(p, T(A["w"]) if A["w"] is not None else torch.zeros(n, dtype=torch.float64, device=dev), A["gauss"])
    if not C.ok:
        return None
    query = case["query"]
    if query == "measures":
        return C.mass.cpu()
    if query == "moments":
        m = C.mass[:, None]
        return C.mass, torch.where(m > 0, p + C.first / m, p), C.cost
    if query == "vjp":
        return _vjp(C, T(A["g"]), p)
    x = C.solve(T(A["g"] - A["g"].mean()))
    return x - x[0]
