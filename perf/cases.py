"""The work that is measured: whole calls of the HDDM solver's public entry points.

A case is one call on one model.  Its fields:

    call       solve        assembly, factors, interface iterations, last solve, edge solution
               resolve      the same from factors in hand (a new source on an unchanged model)
               slots        the reference's plug-in slots one by one, as its own loop calls them
               adjoint      the backward of a solve: adjoint solve and element gradient
               multi        several sources on one set of factors
               post         B, E and Je of every element from an edge solution, on device buffers
    n, h       cells per side of the cube and cell size [m] (6 n^3 tetrahedra)
    leaf       most tetrahedra in one subdomain of the jittered bisection
    npml       absorbing cells at each wall
    layers     random layers: relative permittivity 1 to 10, conductivity from `sigma` up [S/m]
    sigma      the least conductivity
    eps        the solve's residual (hddm_eps)
    precision  fp64 or fp32_ir
    sources    right-hand sides of a multi case, `design` the cells per side of an adjoint's design box

The media are lossy (wet soil and tissue at 300 MHz have 0.1 to 1 S/m).  In
them the interface iterations are well conditioned, so that two orders of
summation give the same solution to far better than `eps`.  In lossless
layered media the same iterations lose every digit in the first fifty, and
two runs that differ by a rounding cannot be compared before they converge;
the work of one iteration is the same in both.
"""
from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch

from adventure_fullwave_b200 import hddm, meshgen

MAX_LOOP = 4000  # the reference's default cap


def _case(call, n, leaf, precision="fp64", h=1.5 / 48, layers=8, sigma=0.2, eps=1e-6, sources=1, design=0):
    return dict(call=call, n=n, h=h, leaf=leaf, npml=max(1, n // 8), layers=layers, sigma=sigma, eps=eps,
                precision=precision, sources=sources, design=design)


def listed():
    return [
        # the smallest models, where launches and latency count: a first try of a geometry
        dict(name="tiny_solve", **_case("solve", 6, 162, h=0.25, layers=2)),
        # the reference's own solver loop on the plug-in table, one library call per iteration
        dict(name="c1_slots", **_case("slots", 16, 600, h=1.0 / 16)),
        # the shipped sample's shape: many subdomains of about 100 elements
        dict(name="small_subdomains_solve", **_case("solve", 21, 110, h=0.05)),
        # a design loop that changes the material: everything from the assembly on
        dict(name="c2_solve", **_case("solve", 48, 600)),
        # a new source on the same model, the sources of a scattering matrix one by one
        dict(name="c2_resolve", **_case("resolve", 48, 600)),
        # the largest: 3.1 million elements, about 5,000 subdomains of the headline model's size
        dict(name="c3_resolve", **_case("resolve", 80, 900, h=1.5 / 96)),
        # single-precision factors with refinement, for models whose factors would not fit otherwise
        dict(name="c2_resolve_fp32_ir", **_case("resolve", 48, 600, precision="fp32_ir")),
        dict(name="c5_solve_fp32_ir", **_case("solve", 63, 1000, precision="fp32_ir", h=1.5 / 112)),
        # one backward of a permittivity design
        dict(name="c4_adjoint", **_case("adjoint", 48, 600, eps=1e-8, design=12)),
        # all ports of an antenna array at once
        dict(name="multi16", **_case("multi", 33, 600, sources=16)),
        dict(name="multi16_fp32_ir", **_case("multi", 24, 1000, precision="fp32_ir", sources=16)),
        # the element results that a field plot or a dose average reads
        dict(name="c2_post", **_case("post", 48, 600)),
    ]


def draw(rng):
    call = rng.choice(["solve", "solve", "resolve", "resolve", "slots", "adjoint", "multi", "multi", "post"])
    top, low_h = {"slots": (32, 0.013), "multi": (24, 0.025)}.get(call, (60, 0.013))
    n = int(round(math.exp(rng.uniform(math.log(8), math.log(top)))))
    precision = rng.choice(["fp64", "fp64", "fp32_ir"])
    c = _case(call, n, leaf=int(round(math.exp(rng.uniform(math.log(100), math.log(1200))))), precision=precision,
              h=round(rng.uniform(low_h, 0.06), 4), layers=rng.randint(1, 8), sigma=round(rng.uniform(0.2, 1.0), 3),
              eps=rng.choice([1e-5, 1e-6, 1e-7]))
    if call == "multi":
        c["sources"] = rng.randint(2, 16)
    if call == "adjoint":
        c.update(design=max(2, n // 4), eps=1e-8)  # the gradient is quadratic in small fields
    return c


# -- inputs ---------------------------------------------------------------------


@functools.lru_cache(maxsize=24)
def _mesh(n, h, leaf, npml, layers, design):
    """The geometry and its partition: the same for every seed, as a program keeps it."""
    return meshgen.make_model("cube", n=n, size=n * h, npml=npml, layers=layers, nleaves=None, leaf_cap=leaf,
                              jitter=(0.3, 0.7), design=design, nprobes=8 if design else 0)


def _model(case, seed):
    """The mesh with the seed's materials and sources."""
    m = _mesh(case["n"], case["h"], case["leaf"], case["npml"], case["layers"], case["design"])
    rng = np.random.default_rng(seed)
    nl, npml = case["layers"], case["npml"]
    eps_r, sig = rng.uniform(1.0, 10.0, nl), case["sigma"] * rng.uniform(1.0, 1.5, nl)
    flags = np.arange(nl * (npml + 1))
    eps, sigma = m.mat_eps.copy(), m.mat_sigma.copy()
    eps[flags] = meshgen.EPS0 * eps_r[flags // (npml + 1)]
    sigma[flags] = sig[flags // (npml + 1)] + meshgen.pml_sigma(npml, case["h"])[flags % (npml + 1)]
    k = eps.shape[0] - flags.shape[0]  # the design box: a flag for each element
    eps[flags.shape[0]:] = meshgen.EPS0 * rng.uniform(2.0, 4.0, k)
    sigma[flags.shape[0]:] = case["sigma"] * rng.uniform(1.0, 1.5, k)
    lo = (npml + 0.5) * case["h"]
    probe = m.probe_edges
    if case["design"]:  # source and probes within a few cells of the design box: the fields die out over the skin depth
        lo = max(lo, 0.5 * m.size - 6 * case["h"])
        mid = 0.5 * (m.vertex_crd[m.edges[:, 0]] + m.vertex_crd[m.edges[:, 1]])
        near = np.nonzero(np.all(np.abs(mid - 0.5 * m.size) < 0.5 * m.size - lo, axis=1))[0]
        probe = np.sort(rng.choice(near, 8, replace=False)).astype(np.int32)
    src = [meshgen.dipole_source(m.edges, m.vertex_crd, rng.uniform(lo, m.size - lo, 3), value=complex(*rng.normal(size=2)))
           for _ in range(case["sources"] + (case["call"] == "resolve"))]
    return dataclasses.replace(m, mat_eps=eps, mat_sigma=sigma, sources=src, probe_edges=probe)


def _edge_values(n_edges, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(n_edges, 2, generator=g, device="cuda", dtype=torch.float64)


def prepare(case, seed):
    model = _model(case, seed)
    solver = hddm.HddmSolver(model, hddm_eps=case["eps"], hddm_max_loop=MAX_LOOP, precision=case["precision"])
    state = dict(call=case["call"], solver=solver, sources=case["sources"])
    if case["call"] in ("resolve", "adjoint"):
        solver.solve(0)
    if case["call"] == "post":
        state["x"] = _edge_values(model.n_edges, seed)
        state["out"] = [torch.empty(model.n_tets, 3, 2, dtype=torch.float64, device="cuda") for _ in range(3)]
    return state


def run(state):
    s, call = state["solver"], state["call"]
    if call == "solve":
        s.solve(0)
        return s.edge_solution()
    if call == "resolve":
        s.resolve(1)
        return s.edge_solution()
    if call == "slots":
        s.make_tmp_aij(0)
        s.solve_dom_1st()
        status = s.iteration_s_1st()
        while status == 0:
            status = s.iteration_s()
        s.solve_dom_last()
        return s.edge_solution()
    if call == "adjoint":
        j, g_eps, g_sigma, _ = s.adjoint_gradient()
        return dict(J=j, g_eps=g_eps, g_sigma=g_sigma)
    if call == "multi":
        s.solve_multi(range(state["sources"]))
        return [s.edge_solution_multi(k) for k in range(state["sources"])]
    s.post_em_E_into(state["x"].data_ptr(), *[o.data_ptr() for o in state["out"]])
    return state["out"]


# -- what a call cannot do without ------------------------------------------------


def _counts(case):
    """Sizes of the model, from its edges: the interior (and the lower
    envelope it takes, in each subdomain's ascending edge order), the
    interface slots."""
    m = _mesh(case["n"], case["h"], case["leaf"], case["npml"], case["layers"], case["design"])
    ne, ns = m.n_edges, m.nsub
    key = np.unique(m.tet_edges.astype(np.int64) + ne * m.sub_of_tet[:, None].astype(np.int64))
    edge, sub = key % ne, key // ne
    shared = np.bincount(edge, minlength=ne) > 1
    free = ~np.asarray(m.pec_edge, bool)
    interior, iface = free & ~shared, free & shared
    rank = np.cumsum(interior[edge])  # subdomains one after another, ascending edges: an interior index
    pos = np.searchsorted(key, m.tet_edges.astype(np.int64) + ne * m.sub_of_tet[:, None].astype(np.int64))
    inner = interior[m.tet_edges]
    low = np.where(inner, rank[pos], np.iinfo(np.int64).max).min(axis=1)  # an element's first interior row
    first = np.full(rank[-1] + 1 if len(rank) else 1, np.iinfo(np.int64).max)
    np.minimum.at(first, rank[pos][inner], np.broadcast_to(low[:, None], inner.shape)[inner])
    rows = np.arange(first.shape[0])
    envelope = int((rows - np.minimum(first, rows) + 1)[1:].sum())
    n_slots, n_int = int(iface[edge].sum()), int(interior[edge].sum())
    return dict(m=m, envelope=envelope, slots=n_slots, interior=n_int, iface=int(iface.sum()), sub=ns)


@functools.lru_cache(maxsize=64)
def _work(key):
    case = dict(key)
    m = _mesh(case["n"], case["h"], case["leaf"], case["npml"], case["layers"], case["design"])
    if case["call"] == "post":
        by = m.n_tets * (16 + 24 + 8 + 1 + 144) + m.n_vertices * 24 + m.n_edges * 16
        return dict(bytes=float(by), flops=570.0 * m.n_tets)
    c = _counts(case)
    fp32 = case["precision"] == "fp32_ir"
    sources = case["sources"] if case["call"] == "multi" else 1
    # iterations to `eps` in these media: as many per digit as cells in a skin depth, counted on runs of these ranges
    its = int(0.29 * -math.log10(case["eps"]) / (case["h"] * math.sqrt(case["sigma"])))
    passes = 2 if fp32 else 1
    entry = 8 if fp32 else 16
    # a subdomain's matrix row has about 12.6 entries: value and column of the interface rows, and of the interior
    # rows where their residual is taken
    nnz = 12.6 * (c["slots"] + (c["interior"] if fp32 else 0))
    matrix = c["envelope"] * entry * passes + nnz * 20  # the factor and the operators, each once
    vectors = 16 * sources * (2 * c["interior"] + 2 * c["slots"] + 10 * c["iface"])
    flops = 8.0 * sources * (2 * passes * c["envelope"] + nnz)
    by, fl = its * (matrix + vectors), its * flops
    if case["call"] in ("solve", "slots", "multi"):
        by += m.n_tets * (40 + 576) + 12.6 * (c["slots"] + c["interior"]) * 16 + c["envelope"] * 16
        fl += 3000.0 * m.n_tets + 4.0 * c["envelope"] ** 2 / max(1, c["interior"])
    return dict(bytes=float(by), flops=float(fl))


def work(case):
    return dict(_work(tuple(sorted((k, v) for k, v in case.items() if k != "name"))))


# -- the same in plain 64 bits ------------------------------------------------------

_PAIRS = ((0, 1), (0, 2), (0, 3), (1, 2), (2, 3), (1, 3))  # the edges of a tetrahedron, in the mesh's order


def _elements(m, dev):
    """Whitney elements of every tetrahedron: edge functions l s (a grad b - b grad a)
    with the global orientation s, their rotations, (rot, rot) and (u, u)."""
    p = torch.as_tensor(m.vertex_crd, device=dev)[torch.as_tensor(m.tets, device=dev).long()]
    t = torch.cat([torch.ones_like(p[..., :1]), p], 2)  # rows: 1, x, y, z of each vertex
    grad = torch.linalg.inv(t)[:, 1:, :].transpose(1, 2)  # grad of each vertex function
    vol = torch.linalg.det(p[:, 1:] - p[:, :1]).abs() / 6
    a, b = (torch.tensor([q[k] for q in _PAIRS], device=dev) for k in (0, 1))
    d = p[:, b] - p[:, a]
    s = torch.sign(d[..., 0])
    s = torch.where(s == 0, torch.sign(d[..., 1]), s)
    s = torch.where(s == 0, torch.sign(d[..., 2]), s)
    w = s * d.norm(dim=2)
    rot = 2 * w[..., None] * torch.linalg.cross(grad[:, a], grad[:, b])
    mid = 0.25 * w[..., None] * (grad[:, b] - grad[:, a])
    rr = vol[:, None, None] * rot @ rot.transpose(1, 2)
    gg = grad @ grad.transpose(1, 2)
    mm = (torch.ones(4, 4, device=dev, dtype=torch.float64) + torch.eye(4, device=dev, dtype=torch.float64)) / 20
    ia, ib = a[:, None], b[:, None]
    ja, jb = a[None, :], b[None, :]
    ss = (mm[ia, ja] * gg[:, ib, jb] - mm[ia, jb] * gg[:, ib, ja] - mm[ib, ja] * gg[:, ia, jb] + mm[ib, jb] * gg[:, ia, ja])
    ss = ss * vol[:, None, None] * w[:, :, None] * w[:, None, :]
    return rr, ss, rot, mid


def _material(m, dev):
    at = np.searchsorted(m.mat_flag, m.flag)
    return (torch.as_tensor(v[at], device=dev) for v in (m.mat_eps, m.mat_sigma))


_NU = 7.957747e5


class _System:
    """The assembled system on the free edges, solved by COCG with the diagonal until the residual stops falling."""

    def __init__(self, m, dev):
        self.m, self.dev = m, dev
        rr, self.ss, _, _ = _elements(m, dev)
        eps, sig = _material(m, dev)
        ae = torch.complex(_NU / m.omega * rr - (eps * m.omega)[:, None, None] * self.ss, sig[:, None, None] * self.ss)
        del rr
        self.te = torch.as_tensor(m.tet_edges, device=dev).long()
        self.free = torch.as_tensor(~np.asarray(m.pec_edge, bool), device=dev)
        i = self.te[:, :, None].expand(-1, 6, 6).reshape(-1)
        j = self.te[:, None, :].expand(-1, 6, 6).reshape(-1)
        keep = self.free[i] & self.free[j]
        idx = torch.stack([i[keep], j[keep]])
        del i, j
        self.a = torch.sparse_coo_tensor(idx, ae.reshape(-1)[keep], (m.n_edges, m.n_edges)).coalesce()
        ij = self.a.indices()
        d = torch.zeros(m.n_edges, dtype=torch.complex128, device=dev)
        on = ij[0] == ij[1]
        d[ij[0][on]] = self.a.values()[on]
        self.pc = torch.where(self.free, 1 / torch.where(d == 0, torch.ones_like(d), d), torch.zeros_like(d))
        self.a = self.a.to_sparse_csr()

    def solve(self, b):
        """The solution, refined once on the true residual; None if it does not converge."""
        b = torch.where(self.free, b, torch.zeros_like(b))
        x = torch.zeros_like(b)
        for _ in range(2):
            r = b - self.a @ x
            first = float(r.norm())
            if first == 0.0:
                return x
            u, z = torch.zeros_like(b), r * self.pc
            p, rz = z.clone(), (r * z).sum()
            for k in range(20000):
                q = self.a @ p
                alpha = rz / (p * q).sum()
                u += alpha * p
                r -= alpha * q
                z = r * self.pc
                new = (r * z).sum()
                p = z + (new / rz) * p
                rz = new
                if k % 50 == 49 and float(r.norm()) < 1e-13 * first:
                    break
            else:
                return None
            x = x + u
        return x

    def source(self, k):
        e, v = self.m.sources[k]
        b = torch.zeros(self.m.n_edges, dtype=torch.complex128, device=self.dev)
        return b.index_add(0, torch.as_tensor(e, device=self.dev).long(), torch.as_tensor(v, device=self.dev))


def exact(case, seed):
    if case["n"] > 64:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    m = _model(case, seed)
    if case["call"] == "post":
        _, _, rot, mid = _elements(m, dev)
        _, sig = _material(m, dev)
        x = torch.view_as_complex(_edge_values(m.n_edges, seed)) * (_NU / m.omega)
        xe = x[torch.as_tensor(m.tet_edges, device=dev).long()]
        e = torch.einsum("ti,tik->tk", xe, mid.to(xe.dtype))
        b = 1j * torch.einsum("ti,tik->tk", xe, rot.to(xe.dtype))
        return [torch.view_as_real(v.contiguous()) for v in (b, 2 * e, sig[:, None] * e)]  # as the reference scales them
    sys_ = _System(m, dev)
    if case["call"] == "multi":
        xs = [sys_.solve(sys_.source(k)) for k in range(case["sources"])]
        return None if any(x is None for x in xs) else [x.cpu().numpy() for x in xs]
    x = sys_.solve(sys_.source(1 if case["call"] == "resolve" else 0))
    if x is None:
        return None
    if case["call"] != "adjoint":
        return x.cpu().numpy()
    pe = torch.as_tensor(m.probe_edges, device=dev).long()
    rhs = torch.zeros_like(x).index_add(0, pe, x[pe].conj())
    lam = sys_.solve(rhs)
    if lam is None:
        return None
    dt = torch.as_tensor(m.design_tets, device=dev).long()
    te = sys_.te[dt]
    s = torch.einsum("ti,tij,tj->t", lam[te], sys_.ss[dt].to(x.dtype), x[te])
    return dict(J=float((x[pe].abs() ** 2).sum()), g_eps=(2 * m.omega * s.real).cpu().numpy(),
                g_sigma=(2 * s.imag).cpu().numpy())
