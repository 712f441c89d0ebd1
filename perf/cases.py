"""Performance cases of the CVFEM engine, each one a call sequence that a
program using the library makes through its public entry points.

The cases cover what the engine is used for: SIMPLE outer iterations on hex8
meshes from a few thousand cells (launch latency) to two million (memory and
arithmetic), in both precisions, eager and as graphs, with the optional terms;
transient steps; the flow with the k-omega SST equations; a batch of
independent cavities; the tet4 conduction step; and the assembly entry points
that a host program drives itself.

A flow pass starts from given fields each time (a program that sweeps over
operating points or restarts), so every pass does the same work. Fields stay
on the device and are written on the flow's own stream. The FP64 form's fields
are returned as they are; the mixed form's carry single-precision fluxes and
are taken out as FP32, as a result file of such a run holds them.
"""
import math

import numpy as np
import torch

from openaccel_b200 import meshgen
from openaccel_b200 import runtime as rt

BENCH_TOL = dict(mom_rtol=0.1, mom_maxit=20, pc_rtol=1e-8)  # solver settings of the cavity example and bench


def listed():
    return [
        # a small study or a first try: launches and latency count
        dict(name="cavity_16_fp64", kind="flow", nx=16, ny=16, nz=16, perturb=0.2, mixed=False, graphs=2, hr=0,
             du_mode=0, tight=False, iters=5),
        # the 32^3 cavity with every setting at its default (eager, FP64, tight momentum tolerance)
        dict(name="cavity_32_defaults", kind="flow", nx=32, ny=32, nz=32, perturb=0.0, mixed=False, graphs=0, hr=0,
             du_mode=0, tight=True, iters=3),
        # odd sizes, high-resolution advection and SIMPLEC
        dict(name="box_61_hr_simplec", kind="flow", nx=61, ny=53, nz=47, perturb=0.2, mixed=False, graphs=2, hr=1,
             du_mode=1, tight=False, iters=3),
        # an ordinary production mesh, FP64
        dict(name="cavity_96_fp64", kind="flow", nx=96, ny=96, nz=96, perturb=0.2, mixed=False, graphs=2, hr=0,
             du_mode=0, tight=False, iters=3),
        # the largest: 2.1M cells, mixed form, each outer iteration one graph
        dict(name="cavity_128_mixed", kind="flow", nx=128, ny=128, nz=128, perturb=0.2, mixed=True, graphs=2, hr=0,
             du_mode=0, tight=False, iters=3),
        # transient run: two BDF2 steps of three coefficient iterations
        dict(name="transient_40_mixed", kind="transient", nx=40, ny=33, nz=29, perturb=0.2, mixed=True, graphs=2,
             steps=2, iters=3),
        # turbulent channel: outer iterations with the SST equations
        dict(name="channel_sst_mixed", kind="sst", nx=128, ny=48, nz=48, mixed=True, graphs=2, iters=2),
        # parameter study: independent cavities of uneven size as one batch
        dict(name="batch_16_mixed", kind="batch", count=16, nmin=16, nmax=40, mixed=True, graphs=2, iters=3),
        # tet4 conduction step, small and large
        dict(name="conduction_20_fp64", kind="conduction", n=20, mixed=False, graphs=0),
        dict(name="conduction_64_mixed", kind="conduction", n=64, mixed=True, graphs=1),
        # the assemblers called one by one by a host program that keeps its data on the device
        dict(name="operators_64_mixed", kind="operators", nx=64, ny=64, nz=64, star=0, mixed=True, shifted=1,
             copy=False),
        # assembled systems taken to the host, on a mesh that is not one block and with standard interpolation
        dict(name="systems_star_fp64", kind="operators", nx=10, ny=10, nz=12, star=5, mixed=False, shifted=0,
             copy=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    """nx >= ny, nz within a quarter of it, so the skewed cells stay valid."""
    nx = _log_int(rng, lo, hi)
    return dict(nx=nx, ny=max(4, int(nx * rng.uniform(0.75, 1.0))), nz=max(4, int(nx * rng.uniform(0.75, 1.0))))


def draw(rng):
    kind = rng.choice(["flow", "flow", "flow", "transient", "sst", "batch", "conduction", "operators"])
    mixed = rng.random() < 0.5
    if kind == "flow":
        return dict(kind=kind, **_box(rng, 12, 110 if mixed else 92), perturb=rng.choice([0.0, 0.1, 0.2]), mixed=mixed,
                    graphs=rng.choice([0, 1, 2, 2]), hr=rng.choice([0, 0, 1]), du_mode=rng.choice([0, 0, 1]),
                    tight=rng.random() < 0.3, iters=rng.randint(2, 4))
    if kind == "transient":
        return dict(kind=kind, **_box(rng, 12, 64), perturb=rng.choice([0.0, 0.2]), mixed=mixed,
                    graphs=rng.choice([0, 2]), steps=2, iters=rng.randint(2, 3))
    if kind == "sst":
        ny = _log_int(rng, 16, 56)
        return dict(kind=kind, nx=int(ny * rng.uniform(2.0, 2.6)), ny=ny, nz=max(8, int(ny * rng.uniform(0.8, 1.0))),
                    mixed=mixed, graphs=rng.choice([0, 2]), iters=2)
    if kind == "batch":
        lo = rng.randint(8, 20)
        return dict(kind=kind, count=rng.randint(4, 24), nmin=lo, nmax=lo + rng.randint(4, 20), mixed=mixed,
                    graphs=rng.choice([0, 2]), iters=rng.randint(2, 3))
    if kind == "conduction":
        return dict(kind=kind, n=_log_int(rng, 8, 60), mixed=mixed, graphs=rng.choice([0, 1]))
    star = rng.choice([0, 0, 0, 3, 5])
    sizes = dict(nx=(n := rng.randint(4, 12)), ny=n, nz=rng.randint(n // 2 + 1, n)) if star else _box(rng, 10, 72)
    return dict(kind=kind, **sizes, star=star, mixed=mixed, shifted=rng.choice([0, 1]),
                copy=sizes["nx"] <= 24 and rng.random() < 0.5)


# ---------------------------------------------------------------------------
# what a program has in hand before the call


def _seed(seed):
    return int(seed) % (1 << 31)


class _Raw:
    """A device array of the library, for torch to view; the view keeps the
    handle that owns the memory alive."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f8", data=(ptr, False), version=3)


def _field(flow, name):
    return torch.as_tensor(_Raw(flow, flow.device_ptr(name), flow._len(name)), device="cuda")


def _hex_mesh(c, seed):
    if c.get("star"):
        return meshgen.star_prism(c["star"], c["nx"], c["nz"], perturb=0.1, seed=_seed(seed))
    return meshgen.cavity((c["nx"], c["ny"], c["nz"]), perturb=c.get("perturb", 0.2), seed=_seed(seed))


def _channel_inputs(c, seed):
    m = meshgen.channel(c["nx"], c["ny"], c["nz"], ratio=1.05)
    r = np.random.default_rng(_seed(seed))
    k = 1e-3 * np.exp(0.2 * r.standard_normal(m.nn))
    w = 1e2 * np.exp(0.2 * r.standard_normal(m.nn))
    return m, meshgen.initial_velocity(m, sigma=0.1, seed=_seed(seed)), k, w


def _conduction_inputs(c, seed):
    m, gamma, src, _ = meshgen.conduction(c["n"], perturb=0.2, seed=_seed(seed))
    x = m.coords[:, 0]
    phi = x + 0.05 * np.random.default_rng(_seed(seed) + 1).standard_normal(m.nn) * x * (1.0 - x)
    return m, gamma, src, np.abs(phi)


def _pressure(m, seed):
    """A smooth nodal pressure with the lid's scale and a little noise."""
    x = m.coords
    noise = np.random.default_rng(_seed(seed) + 2).standard_normal(m.nn)
    return 0.1 * np.sin(3.0 * x[:, 0]) * np.cos(2.0 * x[:, 1] + x[:, 2]) + 0.002 * noise


def _settings(c):
    kw = dict(precision=rt.OA_PREC_MIXED if c["mixed"] else rt.OA_PREC_FP64)
    if c["kind"] == "operators":
        return rt.default_settings(u_shifted=c["shifted"], u_grad_shifted=c["shifted"], p_shifted=c["shifted"],
                                   p_grad_shifted=c["shifted"], **kw)
    kw.update(use_graphs=c["graphs"], hr=c.get("hr", 0), du_mode=c.get("du_mode", 0))
    if not c.get("tight"):
        kw.update(BENCH_TOL)
    if c["kind"] == "transient":
        kw.update(urf_u=1.0, urf_p=0.5)
    if c["kind"] == "batch":
        kw.update(ref_node=-1)
    return rt.default_settings(**kw)


def prepare(case, seed):
    c = dict(case)
    if c["kind"] == "conduction":
        m, gamma, src, phi = _conduction_inputs(c, seed)
        mesh = rt.Mesh(m)
        d = rt.Diffusion(mesh, rt.default_diffusion_settings(
            precision=rt.OA_PREC_MIXED if c["mixed"] else rt.OA_PREC_FP64, use_graphs=c["graphs"]))
        d.set_field("gamma", gamma)
        d.set_field("src", src)
        view = torch.as_tensor(_Raw(d, d.device_ptr("phi"), m.nn), device="cuda")
        return dict(case=c, mesh=mesh, diffusion=d, stream=torch.cuda.ExternalStream(d.stream_handle()), phi=view,
                    phi0=torch.from_numpy(phi).cuda())
    s = dict(case=c)
    given = {}
    if c["kind"] == "batch":
        # edge counts by the case alone; viscosities by the seed
        sizes = np.random.default_rng(c["count"]).integers(c["nmin"], c["nmax"] + 1, size=c["count"])
        bt = meshgen.batch_cavities(sizes=sizes, seed=_seed(seed))
        m = bt.mesh
        U0 = np.zeros((m.nn, 3))
    elif c["kind"] == "sst":
        m, U0, k, w = _channel_inputs(c, seed)
    else:
        m = _hex_mesh(c, seed)
        U0 = meshgen.initial_velocity(m, sigma=0.1, seed=_seed(seed))
    mesh = rt.Mesh(m)
    flow = rt.Flow(mesh, _settings(c))
    if c["kind"] == "batch":
        flow.set_field("mu", bt.mu)
        flow.set_reference_nodes(bt.ref_nodes)
    if c["kind"] == "sst":
        mu = 1e-5
        flow.set_boundary_types([rt.OA_BTYPE_WALL, rt.OA_BTYPE_WALL, rt.OA_BTYPE_SYMMETRY])
        flow.enable_turbulence(0.8, 0.8)
        given.update(k=k, omega=w, gammaK=mu + 0.85 * k / w, gammaOmega=mu + 0.5 * k / w, mu=np.full(m.nn, mu))
        y = m.coords[:, 1]
        s["ymin"] = torch.from_numpy(np.minimum(y, 1.0 - y) + 1e-4).cuda()
        s["wall"] = torch.from_numpy((np.isclose(y, 0.0) | np.isclose(y, 1.0)).astype(np.int32)).cuda()
        s["mu"] = torch.full((m.nn,), mu, dtype=torch.float64, device="cuda")
    given.update(U=U0)
    zero = ["gradU", "gradP"]
    if c["kind"] == "operators":
        given.update(p=_pressure(m, seed))
    else:
        zero.append("p")
    if c.get("hr"):
        zero.append("betaU")
    if c["kind"] == "sst":
        zero += ["srcDiagK", "srcRhsK", "srcDiagOmega", "srcRhsOmega", "gradK", "gradOmega"]
    s["start"] = [(_field(flow, n), torch.from_numpy(np.ascontiguousarray(v).ravel()).cuda()) for n, v in given.items()]
    s["zero"] = [_field(flow, n) for n in zero]
    out = {"flow": "U p mDot gradU gradP", "transient": "U p mDot gradU gradP", "batch": "U p mDot gradU gradP",
           "sst": "U p mDot gradU gradP k omega mu",
           "operators": "du mDot div gradU gradP"}[c["kind"]]
    s["out"] = {n: _field(flow, n) for n in out.split()}
    s.update(mesh=mesh, flow=flow, stream=torch.cuda.ExternalStream(flow.stream_handle()))
    torch.cuda.synchronize()
    return s


def _restart(s):
    with torch.cuda.stream(s["stream"]):
        for view, value in s["start"]:
            view.copy_(value, non_blocking=True)
        for view in s["zero"]:
            view.zero_()


def run(state):
    s, c = state, state["case"]
    if c["kind"] == "conduction":
        with torch.cuda.stream(s["stream"]):
            s["phi"].copy_(s["phi0"], non_blocking=True)
        s["diffusion"].step()
        return {"phi": s["phi"].float() if c["mixed"] else s["phi"]}
    flow = s["flow"]
    _restart(s)
    flow.initialize()
    if c["kind"] == "operators":
        systems = [flow.assemble_momentum(copy=c["copy"])]
        flow.update_mdot()
        systems.append(flow.assemble_pcorr(copy=c["copy"]))
        flow.update_div()
        flow.update_gradient("p")
        flow.update_gradient("U")
        flow.sync()
        out = dict(s["out"])
        if c["copy"]:
            out.update(A_mom=systems[0][0], b_mom=systems[0][1], A_pc=systems[1][0], b_pc=systems[1][1])
        if c["mixed"]:
            out = {k: v.float() if isinstance(v, torch.Tensor) else v.astype(np.float32) for k, v in out.items()}
        return out
    if c["kind"] == "sst":
        flow.sst_iterate(c["iters"], s["ymin"].data_ptr(), s["wall"].data_ptr(), s["mu"].data_ptr(), rtol=1e-6)
    elif c["kind"] == "transient":
        for _ in range(c["steps"]):
            flow.advance_time(2, 0.05)
            flow.simple_iterate(c["iters"])
    else:
        flow.simple_iterate(c["iters"])
    return {k: v.float() for k, v in s["out"].items()} if c["mixed"] else dict(s["out"])


# ---------------------------------------------------------------------------
# bytes and operations of one pass


def _counts(c):
    if c["kind"] == "conduction":
        n = c["n"]
        return (n + 1) ** 3, 6 * n ** 3, 15 * (n + 1) ** 3
    if c["kind"] == "batch":
        n = (c["nmin"] + c["nmax"]) / 2
        return c["count"] * (n + 1) ** 3, c["count"] * n ** 3, 7 * c["count"] * (n + 1) ** 3
    ne = c["nx"] * c["ny"] * c["nz"] * (c.get("star") or 1)
    nn = (c["nx"] + 1) * (c["ny"] + 1) * (c["nz"] + 1) * (c.get("star") or 1)
    return nn, ne, 7 * nn


def work(case):
    """Each input read and each output written once per assembly, update and
    solve of the pass (a solve: its matrix, right-hand side and solution once);
    operations of the element terms and of one matrix product per solve."""
    c = dict(case)
    nn, ne, nnz = _counts(c)
    w = 4 if c["mixed"] else 8
    if c["kind"] == "conduction":
        assemble = 40 * nn + 16 * ne + w * nnz + 8 * nn
        return dict(bytes=assemble + (w + 4) * nnz + 32 * nn, flops=600.0 * ne + 2 * nnz)
    momentum = 104 * nn + 128 * ne + (9 * nnz + 3 * nn) * w + 24 * nn
    mass_flow = 112 * nn + 224 * ne
    pcorr = w * nnz + 8 * nn + 96 * ne
    updates = 96 * ne + 8 * nn + (24 + 48) * nn + (48 + 144) * nn
    if c["kind"] == "operators":
        host = 8 * (10 * nnz + 4 * nn) if c["copy"] else 0
        return dict(bytes=momentum + mass_flow + pcorr + 2 * updates + host, flops=8000.0 * ne)
    solves = (9 * w + 4) * nnz + 6 * w * nn + (w + 4) * nnz + 16 * nn
    iteration = momentum + 2 * mass_flow + pcorr + updates + solves
    flops = 9000.0 * ne + 20 * nnz
    if c["kind"] == "sst":
        iteration += 2 * ((w + 4) * nnz + 16 * nn) + 350 * nn
        flops += 2500.0 * ne
    n = c["iters"] * c.get("steps", 1)
    return dict(bytes=n * iteration, flops=n * flops)


# ---------------------------------------------------------------------------
# the same results in 64 bits from torch alone (assemblies, field updates and
# the conduction step; a whole run of coupled iterations has no such value)

_SIGN = torch.tensor([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                      [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], dtype=torch.float64)
_EDGES = [(0, 1), (1, 2), (2, 3), (0, 3), (4, 5), (5, 6), (6, 7), (4, 7), (0, 4), (1, 5), (2, 6), (3, 7)]
_SMALL = float(np.finfo(np.float64).eps)


def _shape(s):
    """Trilinear shape functions [8] and parametric derivatives [8][3] at s in [-1/2, 1/2]^3."""
    f = 0.5 + _SIGN * s
    N = f.prod(dim=1)
    dN = torch.stack([_SIGN[:, d] * f[:, (d + 1) % 3] * f[:, (d + 2) % 3] for d in range(3)], dim=1)
    return N, dN


def _at(x, s):
    return torch.einsum("n,enk->ek", _shape(s)[0].to(x.device), x)


def _gradients(x, s):
    """Physical gradients [ne][8][3] of the shape functions at s."""
    dN = _shape(s)[1].to(x.device)
    J = torch.einsum("eni,nd->eid", x, dN)
    return torch.einsum("nd,edi->eni", dN, torch.linalg.inv(J))


def _hex_volume(v):
    """Volume [ne] of hexes v [ne][8][3] by facets about the face centres."""
    total = 0.0
    for q in meshgen.HEX_FACE_NODES.tolist():
        m = v[:, q].mean(dim=1)
        for k in range(4):
            a, b = v[:, q[k]], v[:, q[(k + 1) % 4]]
            total = total + (torch.linalg.cross(a, b) * m).sum(dim=1) / 6.0
    return total


class _Hex:
    """Control-volume geometry and the reduced-stencil graph of a hex mesh."""

    def __init__(self, m, dev):
        t = lambda a, k=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=k, device=dev)  # noqa: E731
        self.conn, self.nn, self.ne = t(m.conn, torch.int64), m.nn, m.ne
        self.xn = t(m.coords)
        x = self.x = self.xn[self.conn]
        sub = []
        for c in range(8):  # the corner's sub-volume: its vertices lie between the corner and the centre
            lo, hi = torch.minimum(_SIGN[c], torch.zeros(3)) / 2, torch.maximum(_SIGN[c], torch.zeros(3)) / 2
            v = torch.stack([_at(x, torch.where(_SIGN[j] < 0, lo, hi)) for j in range(8)], dim=1)
            sub.append(_hex_volume(v))
        self.scv = torch.stack(sub, dim=1)
        self.vol = torch.zeros(m.nn, dtype=torch.float64, device=dev).index_add_(0, self.conn.ravel(), self.scv.ravel())
        self.area, self.loc = [], []
        centre = _at(x, torch.zeros(3, dtype=torch.float64))
        for a, b in _EDGES:  # the quad (edge midpoint, face centre, element centre, face centre)
            mid = (_SIGN[a] + _SIGN[b]) / 4
            d = int((_SIGN[a] != _SIGN[b]).nonzero())
            f = [mid.clone(), mid.clone()]
            f[0][(d + 1) % 3] = 0.0
            f[1][(d + 2) % 3] = 0.0
            A = 0.5 * torch.linalg.cross(centre - _at(x, mid), _at(x, f[1]) - _at(x, f[0]))
            A = A * torch.sign((A * (x[:, b] - x[:, a])).sum(dim=1, keepdim=True))
            self.area.append(A)
            self.loc.append(mid)
        pairs = torch.tensor(_EDGES, device=dev)
        i, j = self.conn[:, pairs[:, 0]].ravel(), self.conn[:, pairs[:, 1]].ravel()
        own = torch.arange(m.nn, device=dev)
        self.keys = torch.unique(torch.cat([i * m.nn + j, j * m.nn + i, own * m.nn + own]))
        self.diag = torch.searchsorted(self.keys, own * m.nn + own)
        self.edge = {c: {q for p in _EDGES if c in p for q in p if q != c} for c in range(8)}
        self.faces = []  # boundary faces by ordinal: elements, their boundary
        fo, fe, fb = m.face_ord, m.face_elem, m.face_bnd
        side = np.zeros((m.nn, 3))
        wall = np.zeros(m.nn, bool)
        for b in range(m.bnd_velocity.shape[0]):
            nodes = m.conn[fe[fb == b][:, None], meshgen.HEX_FACE_NODES[fo[fb == b]]].ravel()
            side[nodes] = m.bnd_velocity[b]
            wall[nodes] = True
        self.side, self.wall = t(side), t(wall, torch.bool)
        for o in range(6):
            self.faces.append((meshgen.HEX_FACE_NODES[o].tolist(), t(fe[fo == o], torch.int64)))

    def ip(self, k, shifted):
        return self.loc[k] if shifted else self.loc[k] / 2

    def entry(self, elems, row, col):
        """CSR entry of element column col in the row of corner row: its own, or the diagonal's."""
        i = self.conn[elems, row]
        if col != row and col not in self.edge[row]:
            return self.diag[i]
        return torch.searchsorted(self.keys, i * self.nn + self.conn[elems, col])

    def face_area(self, elems, q, k):
        """Sub-area of boundary face q at its node k."""
        p = self.x[elems]
        a, b, d = p[:, q[k]], p[:, q[(k + 1) % 4]], p[:, q[(k + 3) % 4]]
        return 0.5 * torch.linalg.cross(p[:, q].mean(dim=1) - a, (a + d) / 2 - (a + b) / 2)

    @staticmethod
    def face_ip(q, k, shifted):
        """Parametric location of the boundary ip of face q nearest its node k."""
        s = _SIGN[q[k]] / 2
        if not shifted:
            normal = (_SIGN[q].sum(dim=0).abs() == 4)
            s = torch.where(normal, s, s / 2)
        return s


def _gradient(h, phi, shifted, urf, old):
    """Relaxed Green-Gauss gradient [nn][nc][3] of phi [nn][nc]."""
    acc = torch.zeros(h.nn, phi.shape[1], 3, dtype=torch.float64, device=phi.device)
    pe = phi[h.conn]
    for k, (a, b) in enumerate(_EDGES):
        v = torch.einsum("n,enc->ec", _shape(h.ip(k, shifted))[0].to(phi.device), pe)
        for node, sign in ((a, 1.0), (b, -1.0)):
            acc.index_add_(0, h.conn[:, node], sign * (v - pe[:, node])[:, :, None] * h.area[k][:, None, :])
    for q, elems in h.faces:
        for k in range(4):
            N = _shape(h.face_ip(q, k, shifted))[0].to(phi.device)
            v = torch.einsum("n,enc->ec", N, pe[elems]) - pe[elems, q[k]]
            acc.index_add_(0, h.conn[elems, q[k]], v[:, :, None] * h.face_area(elems, q, k)[:, None, :])
    return (1.0 - urf) * old + urf * acc / h.vol[:, None, None]


def _divergence(h, mdot):
    d = torch.zeros(h.nn, dtype=torch.float64, device=mdot.device)
    for k, (a, b) in enumerate(_EDGES):
        d.index_add_(0, h.conn[:, a], mdot[:, k]).index_add_(0, h.conn[:, b], -mdot[:, k])
    return d


def _momentum(h, st, U, gradP, div, mdot):
    """Momentum system (A [nnz][3][3], b [nn][3]) and D = V / a_ii."""
    dev, I3 = U.device, torch.eye(3, dtype=torch.float64, device=U.device)
    A = torch.zeros(h.keys.numel(), 3, 3, dtype=torch.float64, device=dev)
    b = torch.zeros(h.nn, 3, dtype=torch.float64, device=dev)
    ue, every = U[h.conn], torch.arange(h.ne, device=dev)
    for k, (L, R) in enumerate(_EDGES):
        g, a, m = _gradients(h.x, h.ip(k, st.u_grad_shifted)), h.area[k], mdot[:, k]
        up = m[:, None] * torch.where(m[:, None] > 0, ue[:, L], ue[:, R])
        for row, other, sign in ((L, R, 1.0), (R, L, -1.0)):
            nodes, flow = h.conn[:, row], sign * m
            b.index_add_(0, nodes, -sign * up)
            A.index_add_(0, h.diag[nodes], flow.clamp(min=0)[:, None, None] * I3)
            A.index_add_(0, h.entry(every, row, other), flow.clamp(max=0)[:, None, None] * I3)
            for n in range(8):
                B = -sign * st.mu * ((g[:, n] * a).sum(1)[:, None, None] * I3 + g[:, n, :, None] * a[:, None, :])
                A.index_add_(0, h.entry(every, row, n), B)
                b.index_add_(0, nodes, -torch.einsum("eij,ej->ei", B, ue[:, n]))
    for q, elems in h.faces:  # no-slip walls: tangential stress of the side velocities
        for k in range(4):
            a = h.face_area(elems, q, k)
            nrm = a / a.norm(dim=1, keepdim=True)
            P = I3 - nrm[:, :, None] * nrm[:, None, :]
            g = _gradients(h.x[elems], h.face_ip(q, k, st.u_grad_shifted))
            for n in range(8):
                B = -st.mu * ((g[:, n] * a).sum(1)[:, None, None] * P
                              + torch.einsum("eil,el->ei", P, g[:, n])[:, :, None] * a[:, None, :])
                v = h.side[h.conn[elems, n]] if n in q else ue[elems, n]
                b.index_add_(0, h.conn[elems, q[k]], -torch.einsum("eij,ej->ei", B, v))
                if n not in q:
                    A.index_add_(0, h.entry(elems, q[k], n), B)
    d = torch.diagonal(A[h.diag], dim1=1, dim2=2)
    d = (d + ((-div).clamp(min=0) + st.rho * h.vol / st.dt)[:, None]) / st.urf_u
    A[h.diag[:, None], torch.arange(3, device=dev), torch.arange(3, device=dev)] = d
    b += div[:, None] * U - gradP * h.vol[:, None]
    b[h.wall] *= st.wall_rhs_relax
    return A, b, h.vol[:, None] / (d + _SMALL)


def _face_flux(h, st, k, U, p, gradP, du):
    """Rhie-Chow volume flux of ip k, its gradients and D."""
    N = _shape(h.ip(k, st.u_shifted))[0].to(U.device)
    u, d = torch.einsum("n,enk->ek", N, U[h.conn]), torch.einsum("n,enk->ek", N, du[h.conn])
    g = _gradients(h.x, h.ip(k, st.p_grad_shifted))
    mean = torch.einsum("en,enk->ek", h.scv / h.scv.sum(1, keepdim=True), gradP[h.conn])
    dp = torch.einsum("enk,en->ek", g, p[h.conn])
    return ((u - d * (dp - mean)) * h.area[k]).sum(1), g, d


def _pcorr(h, st, U, p, gradP, du):
    A = torch.zeros(h.keys.numel(), dtype=torch.float64, device=U.device)
    b = torch.zeros(h.nn, dtype=torch.float64, device=U.device)
    every = torch.arange(h.ne, device=U.device)
    for k, (L, R) in enumerate(_EDGES):
        f, g, d = _face_flux(h, st, k, U, p, gradP, du)
        b.index_add_(0, h.conn[:, L], -st.rho * f).index_add_(0, h.conn[:, R], st.rho * f)
        for row, sign in ((L, 1.0), (R, -1.0)):
            for n in range(8):
                A.index_add_(0, h.entry(every, row, n), -sign * st.rho * (d * h.area[k] * g[:, n]).sum(1))
    ref = st.ref_node
    in_row = h.keys.div(h.nn, rounding_mode="floor") == ref
    in_row[h.diag[ref]] = False
    A[in_row] = 0.0
    b[ref] = 0.0
    return A, b


def _exact_operators(c, seed, dev):
    m, st = _hex_mesh(c, seed), _settings(c)
    h = _Hex(m, dev)
    U = torch.as_tensor(meshgen.initial_velocity(m, sigma=0.1, seed=_seed(seed)), dtype=torch.float64, device=dev)
    p = torch.as_tensor(_pressure(m, seed), dtype=torch.float64, device=dev)
    zero = lambda nc: torch.zeros(h.nn, nc, 3, dtype=torch.float64, device=dev)  # noqa: E731
    gradU = _gradient(h, U, st.u_shifted, st.grad_urf, zero(3))
    gradP = _gradient(h, p[:, None], st.p_shifted, st.grad_urf, zero(1))
    mdot = torch.stack([st.rho * (torch.einsum("n,enk->ek", _shape(h.ip(k, st.u_shifted))[0].to(dev), U[h.conn])
                                  * h.area[k]).sum(1) for k in range(12)], dim=1)
    div = _divergence(h, mdot)
    A, b, du = _momentum(h, st, U, gradP[:, 0], div, mdot)
    mdot = torch.stack([st.rho * _face_flux(h, st, k, U, p, gradP[:, 0], du)[0] for k in range(12)], dim=1)
    Ap, bp = _pcorr(h, st, U, p, gradP[:, 0], du)
    out = dict(du=du, mDot=mdot, div=_divergence(h, mdot),
               gradP=_gradient(h, p[:, None], st.p_shifted, st.grad_urf, gradP),
               gradU=_gradient(h, U, st.u_shifted, st.grad_urf, gradU))
    if c["copy"]:
        out.update(A_mom=A, b_mom=b, A_pc=Ap, b_pc=bp)
    return {k: v.reshape(-1).cpu() for k, v in out.items()}


def _exact_conduction(c, seed, dev):
    m, gamma, src, phi = _conduction_inputs(c, seed)
    t = lambda a, k=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=k, device=dev)  # noqa: E731
    conn, x, gm, ph = t(m.conn, torch.int64), t(m.coords), t(gamma), t(phi)
    nn, cross = m.nn, torch.linalg.cross
    xe, ge, pe = x[conn], gm[conn], ph[conn]
    E = xe[:, 1:] - xe[:, :1]
    inv = torch.linalg.inv(E)  # columns: gradients of N1..N3
    g = torch.cat([-inv.sum(2, keepdim=True), inv], dim=2).transpose(1, 2)
    vol = torch.zeros(nn, dtype=torch.float64, device=dev)
    vol.index_add_(0, conn.ravel(), (torch.linalg.det(E) / 24.0)[:, None].expand(-1, 4).reshape(-1))
    centre = xe.mean(1)
    rows, cols, vals = [], [], []
    b = t(src) * vol

    def add(row, col, v):
        rows.append(row), cols.append(col), vals.append(v)

    for i in range(4):
        for j in range(i + 1, 4):
            k, l = [q for q in range(4) if q not in (i, j)]
            mid = (xe[:, i] + xe[:, j]) / 2
            A = 0.5 * cross(centre - mid, (xe[:, [i, j, l]].mean(1) - xe[:, [i, j, k]].mean(1)))
            A = A * torch.sign((A * (xe[:, j] - xe[:, i])).sum(1, keepdim=True))
            flux = -((ge[:, i] + ge[:, j]) / 2)[:, None] * torch.einsum("enk,ek->en", g, A)
            for row, sign in ((i, 1.0), (j, -1.0)):
                for n in range(4):
                    add(conn[:, row], conn[:, n], sign * flux[:, n])
                b.index_add_(0, conn[:, row], -sign * (flux * pe).sum(1))
    wall = torch.zeros(nn, dtype=torch.bool, device=dev)
    side = torch.zeros(nn, dtype=torch.float64, device=dev)
    nodes = m.conn[m.face_elem[:, None], meshgen.TET_SIDE_NODES[m.face_ord]]
    wall[t(nodes.ravel(), torch.int64)] = True
    fixed = [k for k in range(len(m.bnd_kind)) if m.bnd_kind[k] == meshgen.BND_FIXED_VALUE]
    for k in fixed:
        side[t(nodes[m.face_bnd == k].ravel(), torch.int64)] = float(m.bnd_value[k])
    for o in range(4):
        el = t(m.face_elem[np.isin(m.face_bnd, fixed) & (m.face_ord == o)], torch.int64)
        q = meshgen.TET_SIDE_NODES[o].tolist()
        off = ({0, 1, 2, 3} - set(q)).pop()
        v = pe[el].clone()
        v[:, q] = side[conn[el][:, q]]
        grad = torch.einsum("enk,en->ek", g[el], v)
        for k in range(3):
            p0, p1, p2 = xe[el, q[k]], xe[el, q[(k + 1) % 3]], xe[el, q[(k + 2) % 3]]
            A = 0.5 * cross((p0 + p1 + p2) / 3 - p0, (p0 + p2) / 2 - (p0 + p1) / 2)
            G = ge[el, q[k]]
            row = conn[el, q[k]]
            add(row, conn[el, off], -G * (g[el, off] * A).sum(1))
            b.index_add_(0, row, G * (grad * A).sum(1))
    b[wall] *= 0.75
    M = torch.sparse_coo_tensor(torch.stack([torch.cat(rows), torch.cat(cols)]), torch.cat(vals), (nn, nn)).coalesce()
    at = M.indices()
    d = torch.zeros(nn, dtype=torch.float64, device=dev)
    d[at[0][at[0] == at[1]]] = M.values()[at[0] == at[1]]
    M = M.to_sparse_csr()
    # Jacobi BiCGStab to 1e-12
    y, r = torch.zeros_like(b), b.clone()
    r0, p, rho = r.clone(), r.clone(), r @ r
    target = 1e-12 * float(b.norm())
    for _ in range(4000):
        ps = p / d
        v = M @ ps
        alpha = rho / (r0 @ v)
        s = r - alpha * v
        sh = s / d
        u = M @ sh
        omega = (u @ s) / (u @ u)
        y += alpha * ps + omega * sh
        r = s - omega * u
        if float(r.norm()) <= target:
            break
        new = r0 @ r
        p = r + (new / rho) * (alpha / omega) * (p - omega * v)
        rho = new
    return {"phi": (ph + y).clamp(min=0.0).cpu()}


def exact(case, seed):
    c = dict(case)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if c["kind"] == "operators":
        return _exact_operators(c, seed, dev)
    if c["kind"] == "conduction":
        return _exact_conduction(c, seed, dev)
    return None
