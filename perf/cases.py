"""Timed workloads of the solver: what a program that switches to this library has it do.

Every case works on seeded arterial-capillary-venous networks of the kind
``blood_network_b200.network.vascular_network`` builds (two binary trees joined
by a capillary lattice, Poiseuille conductances, optionally a diffusive term on
30 % of the segments), generated here on the GPU so that large ones are quick
to make.  The trees' depth is round(log2(0.2 nodes)), the rule of the named
configurations and of ``network.batch_networks``.

Kinds (``path`` of a case):
  device     one solve with device-resident b and x on a kept hierarchy
  host       one solve with host b and x (the reference's own calling form)
  precond    one application of the AMG + IC(0) preconditioner (host vectors), for
             callers that run their own Krylov method
  oneshot    a new matrix on the device: hierarchy, one solve, release
  update     new values on a kept sparsity (host CSR), then a solve with host b and x
  block      many right-hand sides of one network, solved together
  segmented  many independent networks packed into one system
  gradient   pressures of a network as a function of its radii, and the gradient of
             a pressure misfit with respect to every log-radius (assembly, hierarchy,
             forward and adjoint solve)
"""
import ctypes as C
import math

import numpy as np
import torch

from blood_network_b200 import adjoint, amg
from blood_network_b200.network import D_DIFFUSION, MU_BLOOD, P_INLET, P_OUTLET

DEV = "cuda"


def _case(name, path, nodes, coarsening="pmis", theta=0.25, precision="fp64", stop="bnorm",
          tol=1e-8, diffusive=0.0, count=1):
    """count: columns of a block, networks of a segmented solve (nodes: the largest of them)."""
    c = dict(path=path, nodes=int(nodes), coarsening=coarsening, theta=theta,
             precision=precision, stop=stop, tol=tol, diffusive=diffusive, count=int(count))
    if name:
        c = dict(name=name, **c)
    return c


def listed():
    return [
        # one organ slice or a unit test: every cost is a launch or a latency
        _case("host 2k fp64", "host", 2_000),
        # the 20k-node configuration with the library's defaults, host arrays in and out:
        # how a program written for the reference calls it
        _case("host 20k fp64", "host", 20_000),
        # a user's own outer iteration applying the preconditioner
        _case("precond 75k fp64", "precond", 75_000),
        # a mid-size network, mixed precision, true-residual stop, HMIS as the large runs use it
        _case("device 300k mixed", "device", 300_000, "hmis", 0.5, "mixed", "relres", 1e-10,
              diffusive=0.3),
        # the 2M-node configuration, everything FP64
        _case("device 2m fp64", "device", 2_000_000),
        # the 4M-node configuration in FP64: HMIS, diffusive term
        _case("device 4m fp64", "device", 4_000_000, "hmis", 0.5, "fp64", "relres",
              diffusive=0.3),
        # the largest: the 20M-node configuration, mixed precision
        _case("device 20m mixed", "device", 20_000_000, "hmis", 0.5, "mixed", "relres",
              diffusive=0.3),
        # a network seen once (a reconstruction that changes its topology every time)
        _case("oneshot 1m fp64", "oneshot", 1_000_001, stop="relres"),
        # a vessel-adaptation step: same topology, new radii, host CSR
        _case("update 150k fp64", "update", 150_000),
        # boundary-pressure scenarios of one network
        _case("block 64 x 400k mixed", "block", 400_000, precision="mixed", stop="relres",
              tol=1e-10, count=64),
        # a cohort of networks of 5k-60k nodes in one call
        _case("segmented 64 x 60k mixed", "segmented", 60_000, precision="mixed",
              stop="relres", tol=1e-10, count=64),
        # fitting radii to measured pressures
        _case("gradient 500k fp64", "gradient", 500_000, stop="relres", tol=1e-12,
              diffusive=0.3),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["device", "device", "device", "host", "precond", "oneshot", "update",
                       "block", "segmented", "gradient"])
    coarsening, theta = rng.choice([("pmis", 0.25), ("hmis", 0.5), ("hmis", 0.25)])
    precision = rng.choice(["fp64", "mixed"])
    stop = rng.choice(["bnorm", "relres"])
    diffusive = rng.choice([0.0, 0.3])
    # mixed solves of small networks stop where x still follows FP32 rounding at 1e-8: the
    # tolerance there is one at which the system determines the result
    opt = dict(coarsening=coarsening, theta=theta, precision=precision, stop=stop,
               tol=1e-10 if precision == "mixed" else 1e-8, diffusive=diffusive)
    if path == "device":
        hi = 12_000_000 if precision == "mixed" else 8_000_000
        return _case("", path, _log_uniform(rng, 2_000, hi), **opt)
    if path in ("host", "precond"):
        return _case("", path, _log_uniform(rng, 1_500, 600_000), **opt)
    if path == "oneshot":
        return _case("", path, _log_uniform(rng, 3_000, 1_500_000), **opt)
    if path == "update":
        return _case("", path, _log_uniform(rng, 3_000, 600_000), **opt)
    if path == "block":
        k = rng.randint(2, 64)
        return _case("", path, _log_uniform(rng, 5_000, 25_000_000 // max(k, 16)), count=k, **opt)
    if path == "segmented":
        k = _log_uniform(rng, 4, 128)
        return _case("", path, _log_uniform(rng, 6_000, 80_000), count=k, **opt)
    return _case("", "gradient", _log_uniform(rng, 3_000, 600_000), "pmis", 0.25, "fp64",
                 "relres", 1e-12, diffusive)


# ------------------------------------------------------------------ networks
def _sizes(case):
    """Node counts of the case's networks (segmented: log-uniform below its largest)."""
    if case["path"] != "segmented":
        return [case["nodes"]]
    lo, hi, k = min(5_000, case["nodes"]), case["nodes"], case["count"]
    return [int(round(lo * (hi / lo) ** ((j + 0.5) / k))) for j in range(k)]


def _tree(depth, offset):
    child = torch.arange(1, (1 << depth) - 1, device=DEV)
    parent = (child - 1) // 2
    gen = torch.floor(torch.log2((child + 1).double())).long()
    return parent + offset, child + offset, gen


def _keep(edges, drop, gen):
    m = edges.numel()
    return edges[torch.randperm(m, generator=gen, device=DEV)[:m - int(drop * m)].sort().values]


def _network(nodes, gen, drop=0.25):
    """Segments (u, v), radius and length of one network; its node count; its two roots."""
    depth = max(4, int(round(math.log2(0.2 * nodes))))
    T = (1 << depth) - 1
    want = max(nodes - 2 * T, 8)
    side = max(2, int(round(want ** (1.0 / 3.0))))
    nz = max(2, -(-want // (side * side)))
    n_lat = side * side * nz
    lat0, ven0 = T, T + n_lat
    rand = lambda m: torch.rand(m, generator=gen, device=DEV, dtype=torch.float64)

    au, av, ag = _tree(depth, 0)
    vu, vv, vg = _tree(depth, ven0)
    r_tree = 1e-3 * torch.pow(torch.tensor(0.79, dtype=torch.float64, device=DEV),
                              (torch.cat([ag, vg]) - 1).double())
    r_tree = r_tree * (0.9 + 0.2 * rand(r_tree.numel()))
    hi = max(1e-3 * 0.79 ** (depth - 2), 3.0e-6 * 1.0001)

    n_leaf = 1 << (depth - 1)
    leaf = torch.arange(n_leaf, device=DEV)
    a_tgt = lat0 + (leaf * n_lat) // n_leaf
    v_tgt = lat0 + ((leaf * n_lat) // n_leaf + max(1, n_lat // (2 * n_leaf))) % n_lat
    a_leaf, v_leaf = T // 2 + leaf, ven0 + T // 2 + leaf

    idx = torch.arange(n_lat, device=DEV)
    x, y, z = idx % side, (idx // side) % side, idx // (side * side)
    ex, ey, ez = idx[x < side - 1], idx[y < side - 1], idx[z < nz - 1]
    # a fixed share of the y and z edges beside the backbone, so that sizes do not depend on
    # the seed
    ey = torch.cat([ey[z[ey] == 0], _keep(ey[z[ey] != 0], drop, gen)])
    ez = torch.cat([ez[x[ez] == 0], _keep(ez[x[ez] != 0], drop, gen)])
    cap_u = torch.cat([a_leaf, v_tgt, lat0 + ex, lat0 + ey, lat0 + ez])
    cap_v = torch.cat([a_tgt, v_leaf, lat0 + ex + 1, lat0 + ey + side, lat0 + ez + side * side])
    r_cap = torch.exp(math.log(3.0e-6) + (math.log(hi) - math.log(3.0e-6)) * rand(cap_u.numel()))

    u, v = torch.cat([au, vu, cap_u]), torch.cat([av, vv, cap_v])
    radius = torch.cat([r_tree, r_cap])
    length = 50e-6 + 450e-6 * rand(u.numel())
    return u, v, radius, length, 2 * T + n_lat, (0, ven0)


class _Vessels:
    """The segments of the case's network(s) and its Dirichlet nodes, on the GPU."""

    def __init__(self, case, seed):
        self.gen = torch.Generator(device=DEV)
        self.gen.manual_seed(seed)
        us, vs, rs, ls, bnd, start = [], [], [], [], [], 0
        self.seg_ptr = [0]
        for nodes in _sizes(case):
            u, v, r, l, n, roots = _network(nodes, self.gen)
            us.append(u + start)
            vs.append(v + start)
            rs.append(r)
            ls.append(l)
            bnd += [start + roots[0], start + roots[1]]
            start += n
            self.seg_ptr.append(self.seg_ptr[-1] + n - 2)
        u, v = torch.cat(us), torch.cat(vs)
        self.radius, self.length = torch.cat(rs), torch.cat(ls)
        self.mask = (torch.rand(u.numel(), generator=self.gen, device=DEV) < case["diffusive"]).double()
        self.g = self.conductance(self.radius)
        self.n_nodes, self.n = start, start - len(bnd)
        k = len(bnd) // 2
        p_in = P_INLET * (0.9 + 0.2 * torch.rand(k, generator=self.gen, device=DEV, dtype=torch.float64))
        p_out = P_OUTLET * (0.9 + 0.2 * torch.rand(k, generator=self.gen, device=DEV, dtype=torch.float64))
        self.bnd = torch.tensor(bnd, dtype=torch.int32, device=DEV)
        self.p_bnd = torch.stack([p_in, p_out], 1).reshape(-1).contiguous()
        self.u, self.v = u.to(torch.int32), v.to(torch.int32)

    def conductance(self, radius):
        g = math.pi * radius ** 4 / (8.0 * MU_BLOOD * self.length)
        return g + self.mask * (D_DIFFUSION * math.pi * radius ** 2 / self.length)

    def scenario(self, k):
        """Dirichlet pressures of k boundary scenarios (inlet 10-16 kPa, outlet 1-3 kPa)."""
        t = torch.rand(k, 2, generator=self.gen, device=DEV, dtype=torch.float64)
        return torch.stack([10e3 + 6e3 * t[:, 0], 1e3 + 2e3 * t[:, 1]], 1)

    def device_network(self):
        return adjoint.DeviceNetwork(self.n_nodes, self.u, self.v, self.bnd, self.p_bnd)


class _DeviceArray:
    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False),
                                         "version": 3, "strides": None}


def _assembled(net, g, p_bnd):
    """CSR and right-hand side of the pressure system (CUDA tensors)."""
    lib = amg.load_library()
    s = amg.NetworkSystem()
    torch.cuda.synchronize()
    rc = lib.amg_network_assemble_device(net.n_nodes, net.u.numel(), net.u.data_ptr(),
                                         net.v.data_ptr(), g.data_ptr(), net.bnd.numel(),
                                         net.bnd.data_ptr(), p_bnd.data_ptr(), C.byref(s))
    if rc != 0:
        raise amg.AMGError(rc, lib.amg_solver_last_error().decode())
    take = lambda ptr, n, t: torch.as_tensor(_DeviceArray(ptr, n, t), device=DEV).clone()
    out = (take(s.ia, s.n + 1, "<i4"), take(s.ja, s.nnz, "<i4"), take(s.val, s.nnz, "<f8"),
           take(s.rhs, s.n, "<f8"))
    torch.cuda.synchronize()
    lib.amg_network_system_free(C.byref(s))
    return out


def _options(case):
    return dict(threshold=case["theta"],
                coarsening=amg.COARSEN_HMIS if case["coarsening"] == "hmis" else amg.COARSEN_PMIS,
                precision=amg.PREC_MIXED if case["precision"] == "mixed" else amg.PREC_FP64,
                stop=amg.STOP_RELRES if case["stop"] == "relres" else amg.STOP_BNORM)


class _Handle:
    """A solver over device CSR (amg_solver_create_device), as a C or torch program holds it."""

    def __init__(self, ia, ja, val, case):
        self.lib = amg.load_library()
        o = amg.default_options(**_options(case))
        torch.cuda.synchronize()
        self.h = self.lib.amg_solver_create_device(ia.numel() - 1, ja.numel(), ia.data_ptr(),
                                                   ja.data_ptr(), val.data_ptr(), C.byref(o))
        if not self.h:
            raise amg.AMGError(self.lib.amg_solver_last_status(),
                               self.lib.amg_solver_last_error().decode())

    def close(self):
        if self.h:
            self.lib.amg_solver_free(self.h)
            self.h = None

    def __del__(self):
        self.close()

    def check(self, rc):
        if rc < 0:
            raise amg.AMGError(rc, self.lib.amg_solver_last_error().decode())

    def solve(self, b, tol):
        x = torch.zeros_like(b)
        torch.cuda.synchronize()
        self.check(self.lib.amg_solver_solve_device(self.h, b.data_ptr(), x.data_ptr(), tol, 500, 0))
        return x

    def solve_block(self, B, tol):
        X = torch.zeros_like(B)  # k x n: column-major n x k
        torch.cuda.synchronize()
        self.check(self.lib.amg_solver_solve_block_device(self.h, B.shape[0], B.data_ptr(),
                                                          X.data_ptr(), tol, 500, None, None))
        return X

    def solve_segmented(self, ptr, b, tol):
        x = torch.zeros_like(b)
        torch.cuda.synchronize()
        self.check(self.lib.amg_solver_solve_segmented_device(
            self.h, len(ptr) - 1, ptr.ctypes.data_as(C.c_void_p), b.data_ptr(), x.data_ptr(), tol,
            500, None, None))
        return x


def _observed(net, seed):
    """Measured pressures for the gradient case: 1 % of the interior nodes (seeded),
    a linear drop from inlet to outlet along the numbering with 10 % scatter."""
    m = max(4, net.n // 100)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed + 77)
    obs = torch.randperm(net.n, generator=gen, device=DEV)[:m]
    base = P_INLET + (P_OUTLET - P_INLET) * obs.double() / net.n
    noise = torch.rand(m, generator=gen, device=DEV, dtype=torch.float64)
    return obs, base * (0.9 + 0.2 * noise)


# ------------------------------------------------------------------ the passes
def prepare(case, seed):
    path = case["path"]
    net = _Vessels(case, seed)
    if path == "gradient":
        obs, target = _observed(net, seed)
        return dict(case=case, net=net.device_network(), length=net.length, mask=net.mask,
                    logr=torch.log(net.radius), obs=obs, target=target)
    ia, ja, val, rhs = _assembled(net, net.g, net.p_bnd)
    if path == "oneshot":
        return dict(case=case, csr=(ia, ja, val), b=rhs)
    if path in ("host", "precond", "update"):
        to = lambda t: t.cpu().numpy()
        s = amg.AMGSolver(ia.numel() - 1, to(ia), to(ja), to(val), **_options(case))
        st = dict(case=case, solver=s, b=to(rhs))
        if path == "precond":  # a residual-like vector
            st["b"] = st["b"].max() * np.random.default_rng(seed).standard_normal(net.n)
        if path == "update":  # radii a few per cent off, as after one adaptation step
            f = 0.97 + 0.06 * torch.rand(net.radius.numel(), generator=net.gen, device=DEV,
                                         dtype=torch.float64)
            ia, ja, val, rhs = _assembled(net, net.conductance(net.radius * f), net.p_bnd)
            st.update(csr=(to(ia), to(ja), to(val)), b=to(rhs))
        return st
    st = dict(case=case, solver=_Handle(ia, ja, val, case), b=rhs)
    if path == "block":  # the right-hand side is linear in the boundary pressures
        e = torch.eye(2, dtype=torch.float64, device=DEV)
        unit = torch.stack([_assembled(net, net.g, e[j].contiguous())[3] for j in range(2)])
        st["b"] = (net.scenario(case["count"]) @ unit).contiguous()
    if path == "segmented":
        st["ptr"] = np.array(net.seg_ptr, np.int32)
    return st


def run(state):
    case = state["case"]
    path, tol = case["path"], case["tol"]
    if path == "device":
        return state["solver"].solve(state["b"], tol)
    if path == "host":
        return state["solver"].solve(state["b"], tol=tol, maxiter=500)[0]
    if path == "precond":
        return state["solver"].precond(state["b"])
    if path == "update":
        state["solver"].update(*state["csr"])
        return state["solver"].solve(state["b"], tol=tol, maxiter=500)[0]
    if path == "block":
        return state["solver"].solve_block(state["b"], tol)
    if path == "segmented":
        return state["solver"].solve_segmented(state["ptr"], state["b"], tol)
    if path == "oneshot":
        h = _Handle(*state["csr"], case)
        x = h.solve(state["b"], tol)
        h.close()
        return x
    logr = state["logr"].detach().requires_grad_(True)
    g = adjoint.conductance(logr, state["length"], state["mask"])
    p = adjoint.network_pressure(g, state["net"], tol=tol)
    loss = ((p[state["obs"]] - state["target"]) ** 2).sum()
    loss.backward()
    return {"p": p.detach(), "grad": logr.grad}


# ------------------------------------------------------------------ work, exact
def _counts(case):
    """Interior nodes and segments over the case's networks."""
    n = m = 0
    for nodes in _sizes(case):
        depth = max(4, int(round(math.log2(0.2 * nodes))))
        T, leaf = (1 << depth) - 1, 1 << (depth - 1)
        want = max(nodes - 2 * T, 8)
        side = max(2, int(round(want ** (1.0 / 3.0))))
        nz = max(2, -(-want // (side * side)))
        n_lat = side * side * nz
        n += 2 * T + n_lat - 2
        x_edges, y_flat, y_rest = side * nz * (side - 1), side * (side - 1), side * (side - 1) * (nz - 1)
        z_flat, z_rest = side * (nz - 1), side * (side - 1) * (nz - 1)
        m += 2 * (T - 1) + 2 * leaf + x_edges + y_flat + z_flat
        m += y_rest - int(0.25 * y_rest) + z_rest - int(0.25 * z_rest)
    return n, m


def work(case):
    """The matrix (CSR, FP64) read once, every right-hand side read and every solution
    written once, a multiplication and an addition per entry and right-hand side."""
    n, m = _counts(case)
    k = case["count"] if case["path"] == "block" else 1
    nnz = n + 2 * m
    csr = 12 * nnz + 4 * n
    if case["path"] == "gradient":  # segments (ends, log-radius, length, mask) in; p, gradient out
        return {"bytes": 40 * m + 8 * n, "flops": 4 * nnz}
    return {"bytes": csr + 16 * n * k, "flops": 2 * nnz * k}


def _dense_solver(net, g, lo, hi, node_of):
    """x -> A^{-1} x in FP64 for the interior rows lo..hi of one network: dense Cholesky of
    the diagonally scaled matrix and two refinement steps."""
    n = hi - lo
    iu, iv = node_of[net.u.long()], node_of[net.v.long()]
    A = torch.zeros(n, n, dtype=torch.float64, device=DEV)
    d = torch.zeros(n, dtype=torch.float64, device=DEV)
    for a in (iu, iv):
        s = (a >= lo) & (a < hi)
        d.index_add_(0, a[s] - lo, g[s])
    s = (iu >= lo) & (iu < hi) & (iv >= 0)
    for a, b in ((iu, iv), (iv, iu)):
        A.index_put_((a[s] - lo, b[s] - lo), -g[s], accumulate=True)
    A.diagonal().add_(d)
    w = d.rsqrt()
    L = torch.linalg.cholesky(A * w[:, None] * w[None, :])
    solve = lambda r: w[:, None] * torch.cholesky_solve(w[:, None] * r, L)

    def apply(r):
        x = solve(r)
        for _ in range(2):
            x = x + solve(r - A @ x)
        return x
    return apply


def exact(case, seed):
    path = case["path"]
    if path == "precond":
        return None
    net = _Vessels(case, seed)
    rows = [b - a for a, b in zip(net.seg_ptr, net.seg_ptr[1:])]
    if sum(float(r) ** 3 for r in rows) > 3e13 or sum(rows) > 400_000:
        return None
    g, p_bnd = net.g, net.p_bnd
    node_of = torch.full((net.n_nodes,), -1, dtype=torch.long, device=DEV)
    inner = torch.ones(net.n_nodes, dtype=torch.bool, device=DEV)
    inner[net.bnd.long()] = False
    node_of[inner] = torch.arange(net.n, device=DEV)
    if path == "update":
        f = 0.97 + 0.06 * torch.rand(net.radius.numel(), generator=net.gen, device=DEV,
                                     dtype=torch.float64)
        g = net.conductance(net.radius * f)

    def rhs(p):
        P = torch.zeros(net.n_nodes, dtype=torch.float64, device=DEV)
        P[net.bnd.long()] = p
        out = torch.zeros(net.n, dtype=torch.float64, device=DEV)
        u, v = net.u.long(), net.v.long()
        for a, b in ((u, v), (v, u)):
            s = (node_of[a] >= 0) & (node_of[b] < 0)
            out.index_add_(0, node_of[a][s], g[s] * P[b][s])
        return out

    f = torch.stack([rhs(p) for p in net.scenario(case["count"])], 1) if path == "block" \
        else rhs(p_bnd)[:, None]
    x = torch.empty_like(f)
    for lo, hi in zip(net.seg_ptr, net.seg_ptr[1:]):
        solve = _dense_solver(net, g, lo, hi, node_of)
        x[lo:hi] = solve(f[lo:hi])
    if path == "block":
        return x.T.contiguous()
    x = x[:, 0].contiguous()
    if path != "gradient":
        return x
    obs, target = _observed(net, seed)
    back = torch.zeros(net.n, 1, dtype=torch.float64, device=DEV)
    back[obs, 0] = 2.0 * (x[obs] - target)
    lam = solve(back)[:, 0]
    full = lambda y, b: torch.zeros(net.n_nodes, dtype=torch.float64, device=DEV).masked_scatter_(
        inner, y).index_copy_(0, net.bnd.long(), b)
    P, Lam = full(x, p_bnd), full(lam, torch.zeros_like(p_bnd))
    u, v = net.u.long(), net.v.long()
    dg = -(Lam[u] - Lam[v]) * (P[u] - P[v])
    r, l = net.radius, net.length
    dr = (4.0 * math.pi * r ** 4 / (8.0 * MU_BLOOD * l)
          + net.mask * (2.0 * D_DIFFUSION * math.pi * r ** 2 / l))
    return {"p": x, "grad": dg * dr}
