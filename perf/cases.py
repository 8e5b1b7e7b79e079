"""What this library's users have it do, as cases that can be timed and compared.

A case is a dict of plain values; `kind` says which entry points one pass calls:

  map      uwgpu_bin_and_map: the particle-to-element mapping a host code reads back every time step
  matrices uwgpu_bin_and_map, uwgpu_assemble, uwgpu_get_element_matrices: the drop-in for a host code that
           keeps its own solver and reads K_e, f_e, G_e, S_e and the point viscosities
  voronoi  the same mapping and assembly with discrete Voronoi weights, integration points read back
  advect   upload, uwgpu_advect_particles with a given velocity, coordinates read back
  apply    uwgpu_operator_apply: y = K x for a host code's own Krylov iteration
  solve    mapping, assembly and one FP64 Stokes solve of a linear model, velocity and pressure read back
  step     a whole time step of the benchmark's form (mixed precision): upload, mapping, assembly, solve, the step
           length from the velocity, advection, coordinates read back
  picard   solution set, then the Picard iteration of a yielding model
  network  forward and backward pass of the learned preconditioner's network

Points lie as after some advection: a fixed number per element, moved by a fraction of the element width
and stored in random order.  The models are the ones of the repository's workloads and tests: a dense layer
over a light one, spheres in a background, a Gaussian random viscosity field of contrast 1e6, and layers with
Arrhenius viscosity, Drucker-Prager yielding and limits.  Everything is made from the seed.
"""
import ctypes
import math

import numpy as np
import torch

from earthbyte_underworld_gb300 import uwgpu as U

F64 = torch.float64


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


# ------------------------------------------------------------------------------------------
# Cases
# ------------------------------------------------------------------------------------------
def listed():
    return [
        # a 2D model's mapping, every step of a small run: the latency end (2D Rayleigh-Taylor, 64 x 64, 20 points)
        dict(name="map_2d_64", kind="map", dim=2, nx=64, ny=64, nz=1, ppc=20),
        # a 3D model's mapping on a grid with odd extents
        dict(name="map_3d_45x38x51", kind="map", dim=3, nx=45, ny=38, nz=51, ppc=27),
        # a 2D yielding model whose host code assembles and solves by itself
        dict(name="matrices_2d_yield_64", kind="matrices", dim=2, nx=64, ny=64, nz=1, ppc=20, model="yield"),
        # the same in 3D: spheres, the size the oracle's solver takes in seconds
        dict(name="matrices_3d_spheres_32", kind="matrices", dim=3, nx=32, ny=32, nz=32, ppc=27, model="spheres"),
        # the integration weights most particle-in-cell models run with (10 cells per axis)
        dict(name="voronoi_3d_24", kind="voronoi", dim=3, nx=24, ny=24, nz=24, ppc=20, res=10, model="spheres"),
        # one time step's advection, second order, of a 3D model
        dict(name="advect_3d_40", kind="advect", dim=3, nx=40, ny=40, nz=40, ppc=27, order=2),
        # the FP64 operator under a host code's own Krylov iteration
        dict(name="apply_fp64_64", kind="apply", dim=3, nx=64, ny=64, nz=64, ppc=15, precision="fp64", model="spheres"),
        # the mixed form's operator, odd extents
        dict(name="apply_mixed_51x34x60", kind="apply", dim=3, nx=51, ny=34, nz=60, ppc=15, precision="mixed",
             model="field", decades=6),
        # a whole 2D step with the default solver options (CG Schur iteration, colour Gauss-Seidel), solved tight
        dict(name="solve_2d_64", kind="solve", dim=2, nx=64, ny=64, nz=1, ppc=20, model="layer", solver="default",
             levels=4),
        # two Picard iterations of a yielding 3D model, FGMRES with the scaled BFBt preconditioner, FP64
        dict(name="picard_3d_16", kind="picard", dim=3, nx=16, ny=16, nz=16, ppc=30, model="yield", solver="bfbt",
             levels=3),
        # a whole 3D time step in mixed precision, viscosity a random field over three decades: the largest case
        dict(name="step_3d_field_112", kind="step", dim=3, nx=64, ny=80, nz=112, ppc=20, model="field", decades=3,
             levels=5),
        # the learned preconditioner's network (16/32/64/128 channels), forward and backward
        dict(name="network_48", kind="network", dim=3, nx=48, ny=48, nz=48, depth=4, base=16),
    ]


def _spread(rng, lo, hi, step=1):
    """an integer in [lo, hi], uniform in its logarithm, a multiple of step"""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + 0.999)))
    return max(lo, min(hi, int(v / step) * step if step > 1 else int(v)))


def draw(rng):
    kind = rng.choice(["map", "matrices", "voronoi", "advect", "apply", "solve", "step", "picard", "network"])
    dim = 3 if kind in ("step", "network") else rng.choice([2, 3])

    def grid(lo2, hi2, lo3, hi3, step=1):
        lo, hi = (lo2, hi2) if dim == 2 else (lo3, hi3)
        n = [_spread(rng, lo, hi, step) for _ in range(dim)]
        return dict(dim=dim, nx=n[0], ny=n[1], nz=n[2] if dim == 3 else 1, ppc=rng.randint(15, 40))

    def model(*names):
        name = rng.choice(names)
        return dict(model=name, decades=rng.choice([3, 4, 6])) if name == "field" else dict(model=name)

    if kind == "map":
        return dict(kind=kind, **grid(8, 320, 6, 52))
    if kind == "matrices":
        return dict(kind=kind, **grid(8, 160, 6, 32), **model("layer", "spheres", "yield", "field"))
    if kind == "voronoi":
        return dict(kind=kind, **grid(8, 96, 4, 24), **model("layer", "spheres"), res=rng.randint(5, 10))
    if kind == "advect":
        return dict(kind=kind, **grid(8, 320, 6, 42), order=rng.choice([1, 2, 2]))
    if kind == "apply":
        return dict(kind=kind, **grid(16, 360, 8, 56), **model("spheres", "field"),
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "solve":
        return dict(kind=kind, **grid(16, 64, 8, 16, 4), **model("layer"), solver="default" if dim == 2 else "bfbt",
                    levels=3)
    if kind == "picard":
        return dict(kind=kind, **grid(12, 48, 8, 16, 4), model="yield", solver="bfbt", levels=3)
    if kind == "step":
        return dict(kind=kind, **dict(grid(1, 1, 24, 64, 8), ppc=rng.randint(15, 30)), model="field",
                    decades=rng.choice([3, 4]), levels=4)
    return dict(kind=kind, dim=3, nx=_spread(rng, 12, 47), ny=_spread(rng, 12, 47), nz=_spread(rng, 12, 47),
                depth=rng.randint(2, 4), base=rng.choice([8, 16]))


# ------------------------------------------------------------------------------------------
# Models
# ------------------------------------------------------------------------------------------
def _nel(case):
    return [case["nx"], case["ny"]] + ([case["nz"]] if case["dim"] == 3 else [])


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _points(case, g):
    """coordinates (points, dim): ppc uniform points per element, each moved by a normal 0.15 of the element width,
    reflected at the walls, in random order"""
    dim, nel, ppc = case["dim"], _nel(case), case["ppc"]
    dev = _device()
    ne = math.prod(nel)
    e = torch.arange(ne, device=dev).repeat_interleave(ppc)
    out = torch.empty((ne * ppc, dim), dtype=F64, device=dev)
    for d in range(dim):
        i = e % nel[d]
        e = e // nel[d]
        r = torch.rand(ne * ppc, generator=g, device=dev, dtype=F64)
        r += 0.15 * torch.randn(ne * ppc, generator=g, device=dev, dtype=F64).clamp(-4, 4)
        x = ((i + r) / nel[d]).abs()
        out[:, d] = torch.where(x > 1.0, 2.0 - x, x)
    return out[torch.randperm(ne * ppc, generator=g, device=dev)]


def _smooth(x, g, waves=24, corr=0.1):
    """a smooth random field of unit maximum at the points x (squared-exponential spectrum of length corr)"""
    dim = x.shape[1]
    k = torch.randn((waves, dim), generator=g, device=x.device, dtype=F64) * (math.sqrt(2.0) / corr / 2)
    ph = torch.rand(waves, generator=g, device=x.device, dtype=F64) * 2 * math.pi
    f = torch.zeros(x.shape[0], dtype=F64, device=x.device)
    for w in range(waves):
        f += torch.cos(x @ k[w] + ph[w])
    return f / f.abs().max()


def _nodes(nel):
    """node coordinates (nodes, dim), x fastest"""
    dev = _device()
    axes = [torch.arange(n + 1, device=dev, dtype=F64) / n for n in nel]
    grids = torch.meshgrid(*axes[::-1], indexing="ij")[::-1]
    return torch.stack([t.reshape(-1) for t in grids], dim=1)


def _flow(nel, g):
    """a smooth velocity on the nodes (nodes, dim) that vanishes through the walls, and a pressure per element"""
    X = _nodes(nel)
    dim = X.shape[1]
    a = 0.5 + torch.rand(dim, generator=g, device=X.device, dtype=F64)
    u = torch.empty_like(X)
    for d in range(dim):
        v = a[d] * torch.sin(math.pi * X[:, d])
        for q in range(dim):
            if q != d:
                v = v * torch.cos(math.pi * X[:, q])
        u[:, d] = v
    p = torch.randn(math.prod(nel), generator=g, device=X.device, dtype=F64)
    return u, p


def _model(case, seed):
    """points, materials, nodal temperature, previous velocity and pressure of a model, on the device"""
    g = _generator(seed)
    dim, nel = case["dim"], _nel(case)
    x = _points(case, g)
    n = x.shape[0]
    dev = x.device
    m = dict(x=x, material=torch.zeros(n, dtype=torch.int32, device=dev), eta=None, rho=None, temperature=None,
             u=None, p=None, vert=dim - 1)
    name = case.get("model", "layer")
    if name == "layer":
        below = x[:, dim - 1] < 0.2 + 0.02 * torch.cos(math.pi * x[:, 0])
        m["material"] = below.to(torch.int32)
        m["table"] = [dict(laws=[(U.LAW_MATERIAL_VISCOSITY, [1.0])], density=1.0),
                      dict(laws=[(U.LAW_MATERIAL_VISCOSITY, [0.01])], density=0.0)]
    elif name == "spheres":
        count = 12
        c = torch.rand((count, dim), generator=g, device=dev, dtype=F64)
        r = 0.05 + 0.1 * torch.rand(count, generator=g, device=dev, dtype=F64)
        v = torch.rand((count, 2), generator=g, device=dev, dtype=F64).tolist()
        m["table"] = [dict(laws=[(U.LAW_MATERIAL_VISCOSITY, [1.0])], density=0.0)]
        for s in range(count):
            m["material"][((x - c[s]) ** 2).sum(1) <= r[s] ** 2] = s + 1
            m["table"].append(dict(laws=[(U.LAW_MATERIAL_VISCOSITY, [10.0 ** (4 * v[s][0] - 2)])], density=v[s][1]))
    elif name == "field":
        f = _smooth(x, g)
        m["eta"] = 10.0 ** (0.5 * case["decades"] * f)
        m["rho"] = 0.5 * f + 0.5
        m["table"] = [dict(laws=[(U.LAW_PARTICLE_VISCOSITY, [])], density=0.0)]
    else:
        th = torch.cumsum(0.5 + torch.rand(5, generator=g, device=dev, dtype=F64), 0)
        m["material"] = torch.searchsorted(th / th[-1], x[:, dim - 1].contiguous(), right=True).clamp(max=4).to(torch.int32)
        v = torch.rand((5, 3), generator=g, device=dev, dtype=F64).tolist()
        m["table"] = []
        for a, b, c in v:
            ea = 4.0 + 4.0 * a
            m["table"].append(dict(laws=[(U.LAW_ARRHENIUS, [math.exp(-ea / 1.1), ea, 0.0, 0.1]),
                                         (U.LAW_DRUCKER_PRAGER, [0.1 + 0.9 * b, 0.6, 0.0, 1e-3]),
                                         (U.LAW_VISCOSITY_LIMITER, [1e3, 1e-3])], density=c))
        X = _nodes(nel)
        T = 1.0 - 0.7 * X[:, dim - 1]
        for _ in range(8):
            c = torch.rand(dim, generator=g, device=dev, dtype=F64)
            T = T + 0.1 * torch.exp(-((X - c) ** 2).sum(1) / (2 * 0.05 ** 2))
        m["temperature"] = T
        m["u"], m["p"] = _flow(nel, g)
    return m


def _host(t):
    return None if t is None else t.cpu().numpy()


def _options(case):
    """solver options; every solve is taken to the accuracy at which the tests compare answers"""
    if case["kind"] == "step":
        return U.default_opts(mg_levels=case["levels"], smoother=U.SMOOTHER_CHEBYSHEV, schur_type=U.SCHUR_FGMRES,
                              schur_pc=U.SCHUR_PC_SCALED_BFBT, precision=U.PREC_MIXED, scr_rtol=1e-11, a11_rtol=1e-12,
                              back_rtol=1e-12, max_inner=2000, bfbt_rtol=1e-2, bfbt_max_it=2000)
    if case["solver"] == "default":
        return U.default_opts(mg_levels=case["levels"], scr_rtol=1e-10, a11_rtol=1e-12, back_rtol=1e-12)
    return U.default_opts(mg_levels=case["levels"], schur_type=U.SCHUR_FGMRES, schur_pc=U.SCHUR_PC_SCALED_BFBT,
                          scr_rtol=1e-10, a11_rtol=1e-12, back_rtol=1e-12, max_inner=2000, bfbt_rtol=1e-2,
                          bfbt_max_it=2000)


# ------------------------------------------------------------------------------------------
# prepare / run
# ------------------------------------------------------------------------------------------
def _context(case, m, upload=True):
    dim, nel = case["dim"], _nel(case)
    ctx = U.Context(0)
    ctx.mesh_q1(dim, nel)
    ctx.bc_set(U.free_slip_mask(dim, nel))
    ctx.materials_set([U.make_material(t["laws"], density=t["density"]) for t in m["table"]])
    ctx.fields_set(_host(m["temperature"]), 1.0, m["vert"])
    coords = [_host(m["x"][:, d].contiguous()) for d in range(dim)] + [None] * (3 - dim)
    points = (*coords, _host(m["material"]), _host(m["eta"]), _host(m["rho"]))
    if upload:
        ctx.particles_upload(*points)
    return ctx, points


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind == "network":
        nel = _nel(case)
        ctx = U.Context(0)
        ctx.mesh_q1(3, nel)
        ctx.learned_create(levels=case["depth"], base=case["base"], seed=int(seed) % 100000 + 1)
        state.update(_network_data(case, seed, ctx.learned_params()))
        ctx.learned_set_params(state["params"])
        state["ctx"] = ctx
        return state
    m = _model(case, seed)
    if kind == "advect":
        g = _generator(seed + 1)
        u, p = _flow(_nel(case), g)
        state["u"], state["p"] = _host(u), _host(p)
        state["dt"] = 0.3 / max(_nel(case))
        state["ctx"], state["points"] = _context(case, m, upload=False)
        return state
    ctx, state["points"] = _context(case, m)
    state["ctx"] = ctx
    if kind == "matrices" and m["u"] is not None:
        ctx.solution_set(_host(m["u"]), _host(m["p"]))
    elif kind == "voronoi":
        ctx.weights_set(U.WEIGHTS_DVC, [case["res"]] * case["dim"])
    elif kind == "apply":
        ctx.bin_and_map(want=False)
        ctx.assemble()
        nodes = math.prod(n + 1 for n in _nel(case))
        state["x"] = _host(torch.randn(nodes * case["dim"], generator=_generator(seed + 1), device=_device(), dtype=F64))
        state["precision"] = U.PREC_MIXED if case["precision"] == "mixed" else U.PREC_FP64
        ctx.operator_apply(state["x"], state["precision"])   # builds the operator, as the first product does
    elif kind == "picard":
        state["u"], state["p"] = _host(m["u"]), _host(m["p"])
    if kind in ("solve", "picard", "step"):
        state["opts"] = _options(case)
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "map":
        perm, offsets, xi = ctx.bin_and_map()
        return dict(perm=perm, offsets=offsets, xi=xi)
    if kind == "matrices":
        ctx.bin_and_map(want=False)
        ctx.assemble()
        Ke, fe, Ge, Se = ctx.element_matrices()
        return dict(Ke=Ke, fe=fe, Ge=Ge, Se=Se, eta=ctx.point_viscosity())
    if kind == "voronoi":
        ctx.bin_and_map(want=False)
        ctx.assemble()
        xi, w = ctx.integration_points()
        return dict(xi=xi, w=w)
    if kind == "advect":
        ctx.particles_upload(*state["points"])
        ctx.solution_set(state["u"], state["p"])
        back, left = ctx.advect(state["dt"], order=case["order"], allow_fallback=True)
        x, y, z = ctx.particles()
        return dict(x=x, y=y, z=z, fell_back=back, left_mesh=left)
    if kind == "apply":
        return dict(y=ctx.operator_apply(state["x"], state["precision"]))
    if kind == "solve":
        ctx.bin_and_map(want=False)
        ctx.assemble()
        u, p, _ = ctx.solve_bsscr(state["opts"])
        return dict(u=u, p=p)
    if kind == "step":
        ctx.particles_upload(*state["points"])
        ctx.bin_and_map(want=False)
        ctx.assemble()
        u, _, _ = ctx.solve_bsscr(state["opts"])
        dt = 0.25 / (max(_nel(case)) * float(np.abs(u).max()))
        ctx.advect(dt, order=2, allow_fallback=True)
        x, y, z = ctx.particles()
        return dict(u=u, x=x, y=y, z=z)
    if kind == "picard":
        ctx.solution_set(state["u"], state["p"])
        ctx.bin_and_map(want=False)
        u, p, _, _, residual = ctx.solve_picard(state["opts"], tolerance=0.0, max_iterations=2)
        return dict(u=u, p=p, residual=residual)
    out = ctx.learned_forward(state["input"])
    gp, gi = ctx.learned_backward(state["grad"])
    return dict(out=out, grad_params=gp, grad_input=gi)


def work(case):
    dim, nel = case["dim"], _nel(case)
    ne, nn = math.prod(nel), math.prod(n + 1 for n in nel)
    kind = case["kind"]
    if kind == "network":
        flops, params, vox = 0, 0, 1
        mult = 1 << (case["depth"] - 1)
        for n in nel:
            vox *= (n + 1 + mult - 1) // mult * mult
        for l, cin, cout in _layers(case):
            flops += 2 * 27 * cin * cout * vox // 8 ** l
            params += 27 * cin * cout + cout
        return dict(bytes=4 * (7 * nn * 2 + 3 * nn * 2 + 2 * params), flops=3 * flops)
    n = ne * case["ppc"]
    xyz = 8 * dim * n
    if kind == "map":
        return dict(bytes=xyz + 4 * n + 24 * n + 4 * (ne + 1), flops=10 * dim * n)
    if kind == "advect":
        return dict(bytes=2 * xyz + 4 * n + 8 * (dim * nn + ne), flops=(80 if dim == 3 else 40) * case["order"] * n)
    nd = dim << dim
    flops = (120 if dim == 3 else 50) * n + (3600 if dim == 3 else 300) * ne
    if kind == "matrices":
        return dict(bytes=xyz + 12 * n + 8 * (nd * nd + 2 * nd + 1) * ne, flops=flops)
    if kind == "voronoi":
        return dict(bytes=xyz + 4 * n + 32 * n, flops=flops + 9 * case["res"] ** dim * ne)
    if kind == "apply":
        # the operator is symmetric: half of its blocks, and the diagonal ones' triangles
        entries = 123 if dim == 3 else 19
        word = 4 if case["precision"] == "mixed" else 8
        return dict(bytes=nn * (entries * word + 16 * dim), flops=nn * (486 if dim == 3 else 72))
    if kind == "step":
        return dict(bytes=2 * xyz + 20 * n + 8 * dim * nn, flops=flops + 160 * n)
    return dict(bytes=xyz + 4 * n + 8 * (dim * nn + ne), flops=flops)


# ------------------------------------------------------------------------------------------
# The same results in 64 bits from plain torch
# ------------------------------------------------------------------------------------------
def _located(x, nel):
    """element of every point, the points' order by element (ascending index within one), counts, local coordinates"""
    idx = [torch.clamp((x[:, d] * nel[d]).floor().long(), 0, nel[d] - 1) for d in range(x.shape[1])]
    e, mul = torch.zeros_like(idx[0]), 1
    xi = torch.empty_like(x)
    for d, n in enumerate(nel):
        e = e + mul * idx[d]
        mul *= n
        xi[:, d] = 2.0 * (x[:, d] - idx[d].to(F64) / n) * n - 1.0
    return e, torch.argsort(e, stable=True), torch.bincount(e, minlength=mul), xi


def _shape(xi):
    """shape functions (points, nodes) and their local derivatives (points, nodes, dim)"""
    dim = xi.shape[1]
    N, dN = [], []
    for a in range(1 << dim):
        f = [0.5 * (1 + (xi[:, d] if (a >> d) & 1 else -xi[:, d])) for d in range(dim)]
        N.append(math.prod(f[1:], start=f[0]))
        row = []
        for d in range(dim):
            v = torch.full_like(f[0], 0.5 if (a >> d) & 1 else -0.5)
            for q in range(dim):
                if q != d:
                    v = v * f[q]
            row.append(v)
        dN.append(torch.stack(row, 1))
    return torch.stack(N, 1), torch.stack(dN, 1)


def _element_nodes(nel):
    dev = _device()
    e = torch.arange(math.prod(nel), device=dev)
    base, mul = torch.zeros_like(e), 1
    for n in nel:
        base = base + mul * (e % n)
        e = e // n
        mul *= n + 1
    off = []
    for a in range(1 << len(nel)):
        o, mul = 0, 1
        for d, n in enumerate(nel):
            o += mul * ((a >> d) & 1)
            mul *= n + 1
        off.append(o)
    return base[:, None] + torch.tensor(off, device=dev)


def _viscosity(m, e, N, G, en, u, p):
    """viscosity and density of points in elements e (shape functions N, global derivatives G)"""
    mat = m["material"].long()
    dens = torch.tensor([t["density"] for t in m["table"]], device=N.device, dtype=F64)[mat]
    kind = m["table"][0]["laws"][0][0]
    if kind == U.LAW_PARTICLE_VISCOSITY:
        return m["eta"], m["rho"]
    if kind == U.LAW_MATERIAL_VISCOSITY:
        return torch.tensor([t["laws"][0][1][0] for t in m["table"]], device=N.device, dtype=F64)[mat], dens
    par = torch.tensor([t["laws"][0][1] + t["laws"][1][1] for t in m["table"]], device=N.device, dtype=F64)[mat]
    T = (N * m["temperature"][en[e]]).sum(1)
    eta = par[:, 0] * torch.exp(par[:, 1] / (T + par[:, 3]))
    if u is not None:
        L = torch.einsum("pad,pai->pid", G, u[en[e]])
        s = eta[:, None, None] * (L + L.transpose(1, 2))
        ind = torch.sqrt(0.5 * (s * s).sum((1, 2)))
        phi = math.atan(0.6)
        if N.shape[1] == 8:
            ood = 1.0 / (math.sqrt(3.0) * (3.0 - math.sin(phi)))
            fric, coh = 6.0 * math.sin(phi) * ood, 6.0 * par[:, 4] * math.cos(phi) * ood
        else:
            fric, coh = math.sin(phi), par[:, 4] * math.cos(phi)
        crit = torch.clamp(fric * p[e] + coh, min=0.0)
        eta = torch.where(crit < ind, torch.maximum(eta * crit / ind, torch.full_like(eta, 1e-3)), eta)
        eta = torch.clamp(eta, min=1e-3)
    return torch.clamp(eta, 1e-3, 1e3), dens


def _strain_matrix(G):
    """B (points, 3 or 6, nodes * dim) with engineering shear rows"""
    p, nodes, dim = G.shape
    pairs = [(0, 1)] if dim == 2 else [(0, 1), (0, 2), (1, 2)]
    B = torch.zeros((p, dim + len(pairs), nodes, dim), dtype=F64, device=G.device)
    for d in range(dim):
        B[:, d, :, d] = G[:, :, d]
    for r, (i, j) in enumerate(pairs):
        B[:, dim + r, :, i] = G[:, :, j]
        B[:, dim + r, :, j] = G[:, :, i]
    return B.reshape(p, dim + len(pairs), nodes * dim)


def _assembled(case, m, u=None, p=None, matrices=True, vector=None, chunk=1 << 16):
    """K_e, f_e, G_e, S_e and the slots' viscosity (matrices), or K x for a nodal vector (nodes, dim)"""
    dim, nel = case["dim"], _nel(case)
    ne, nen = math.prod(nel), 1 << dim
    nd = nen * dim
    e, order, counts, xi = _located(m["x"], nel)
    en = _element_nodes(nel)
    dev = e.device
    scale = torch.tensor([2.0 * n for n in nel], dtype=F64, device=dev)
    detj = math.prod(0.5 / n for n in nel)
    w = (2.0 ** dim / counts.to(F64))[e] * detj
    dia = torch.tensor([2.0] * dim + [1.0] * (1 if dim == 2 else 3), dtype=F64, device=dev)
    eta = torch.empty(e.shape[0], dtype=F64, device=dev)
    K = torch.zeros((ne, nd, nd), dtype=F64, device=dev) if matrices else None
    f = torch.zeros((ne, nen, dim), dtype=F64, device=dev)
    y = torch.zeros_like(vector) if vector is not None else None
    for c in range(0, e.shape[0], chunk):
        s = slice(c, c + chunk)
        sub = dict(m, material=m["material"][s], eta=None if m["eta"] is None else m["eta"][s],
                   rho=None if m["rho"] is None else m["rho"][s])
        N, dN = _shape(xi[s])
        G = dN * scale
        v, rho = _viscosity(sub, e[s], N, G, en, u, p)
        eta[s] = v
        B = _strain_matrix(G)
        if matrices:
            BD = B * (dia[None, :, None] * (w[s] * v)[:, None, None])
            K.index_add_(0, e[s], torch.bmm(BD.transpose(1, 2), B))
            F = torch.zeros((N.shape[0], nen, dim), dtype=F64, device=dev)
            F[:, :, m["vert"]] = -(w[s] * rho)[:, None] * N
            f.index_add_(0, e[s], F)
        if vector is not None:
            nodes = en[e[s]]
            strain = torch.bmm(B, vector[nodes].reshape(-1, nd, 1))[:, :, 0]
            force = torch.bmm(B.transpose(1, 2), (strain * dia * (w[s] * v)[:, None])[:, :, None])
            y.index_add_(0, nodes.reshape(-1), force.reshape(-1, dim))
    if vector is not None:
        return y
    Ge = torch.empty((ne, nen, dim), dtype=F64, device=dev)
    for a in range(nen):
        for d in range(dim):
            Ge[:, a, d] = (-1.0 if (a >> d) & 1 else 1.0) * math.prod(1.0 / nel[q] for q in range(dim) if q != d) \
                / 2 ** (dim - 1)
    Ge = Ge.reshape(ne, nd)
    Se = (Ge * Ge / torch.diagonal(K, dim1=1, dim2=2)).sum(1)
    return K, f.reshape(ne, nd), Ge, Se, eta[order]


def _free(case):
    mask = U.free_slip_mask(case["dim"], _nel(case))
    return torch.from_numpy(mask == 0).to(_device())


def _direct(case, K, f, Ge):
    """velocity (nodes, dim) and pressure of the assembled system, free-slip walls, mean-free pressure, by LU"""
    dim, nel = case["dim"], _nel(case)
    ne, nn = math.prod(nel), math.prod(n + 1 for n in nel)
    dof = (_element_nodes(nel)[:, :, None] * dim + torch.arange(dim, device=_device())).reshape(ne, -1)
    free = _free(case)
    nv = nn * dim
    A = torch.zeros((nv + ne, nv + ne), dtype=F64, device=_device())
    nd = dof.shape[1]
    A.view(-1).index_add_(0, (dof[:, :, None] * (nv + ne) + dof[:, None, :]).reshape(-1), K.reshape(-1))
    pe = torch.arange(ne, device=_device())[:, None].expand(ne, nd) + nv
    A.view(-1).index_add_(0, (dof * (nv + ne) + pe).reshape(-1), Ge.reshape(-1))
    A[nv:, :nv] = A[:nv, nv:].T
    fixed = torch.nonzero(~free)[:, 0]
    A[fixed, :] = 0.0
    A[:, fixed] = 0.0
    A[fixed, fixed] = 1.0
    A[nv:, nv:] = -1.0 / ne ** 2
    b = torch.zeros(nv + ne, dtype=F64, device=_device())
    b.index_add_(0, dof.reshape(-1), f.reshape(-1))
    b[fixed] = 0.0
    s = torch.linalg.solve(A, b)
    return s[:nv].reshape(nn, dim), s[nv:]


def _velocity_at(x, u, nel, en):
    e, _, _, xi = _located(x, nel)
    N, _ = _shape(xi)
    return (N[:, :, None] * u[en[e]]).sum(1)


def _layers(case):
    """(level, cin, cout) of the 3x3x3 layers in parameter order"""
    depth = case["depth"]
    ch = [case["base"] << l for l in range(depth)]
    out = []
    for l in range(depth):
        out += [(l, ch[l - 1] if l else 8, ch[l]), (l, ch[l], ch[l])]
    for l in range(depth - 1):
        out += [(l, ch[l + 1] + ch[l], ch[l]), (l, ch[l], ch[l])]
    return out


def _network_data(case, seed, params):
    """parameters with a small random head and biases (as after training), a residual-like input and a gradient"""
    g = _generator(seed)
    dev = _device()
    nn = math.prod(n + 1 for n in _nel(case))
    p = torch.from_numpy(params).to(dev) if params is not None else None
    head = 3 * case["base"] + 3
    inp = torch.randn((7, nn), generator=g, device=dev)
    X = _nodes(_nel(case))
    inp[6] = (3.0 * _smooth(X, g)).float()
    grad = torch.stack([_smooth(X, g) for _ in range(3)]).float() / nn
    tail = 0.1 * torch.randn(head, generator=g, device=dev)
    if p is not None:
        p[-head:] = tail
    return dict(params=_host(p), input=_host(inp), grad=_host(grad))


def _network_exact(case, state):
    nel, depth = _nel(case), case["depth"]
    nodes = [n + 1 for n in nel]
    mult = 1 << (depth - 1)
    pad = [(n + mult - 1) // mult * mult for n in nodes]
    dev = _device()
    p = torch.from_numpy(state["params"]).to(dev).double().requires_grad_()
    inp = torch.from_numpy(state["input"]).to(dev).double().requires_grad_()
    fn = torch.nn.functional
    grid = inp.reshape(1, 7, nodes[2], nodes[1], nodes[0])
    x = fn.pad(grid, (0, pad[0] - nodes[0], 0, pad[1] - nodes[1], 0, pad[2] - nodes[2], 0, 1))
    off, layers = 0, []
    for _, cin, cout in _layers(case):
        w = p[off:off + 27 * cin * cout].reshape(27, cin, cout)
        off += 27 * cin * cout
        layers.append((w, p[off:off + cout]))
        off += cout

    def stored(t):
        """the network is defined with BF16 weights and activations: rounded values, gradients passed through"""
        return t + (t.to(torch.bfloat16).double() - t).detach()

    def conv(t, k):
        w, b = layers[k]
        w = stored(w)
        z, y, xx = t.shape[2:]
        tp = fn.pad(t[0].permute(1, 2, 3, 0), (0, 0, 1, 1, 1, 1, 1, 1))
        out = b.expand(z, y, xx, b.shape[0])
        for tap in range(27):
            dx, dy, dz = tap % 3, tap // 3 % 3, tap // 9
            out = out + tp[dz:dz + z, dy:dy + y, dx:dx + xx] @ w[tap]
        return stored(torch.relu(out.permute(3, 0, 1, 2)[None]))

    skips, t = [], stored(x)
    for l in range(depth):
        t = conv(conv(t, 2 * l), 2 * l + 1)
        skips.append(t)
        if l + 1 < depth:
            t = stored(fn.avg_pool3d(t, 2))
    for l in range(depth - 2, -1, -1):
        t = torch.cat([fn.interpolate(t, scale_factor=2, mode="nearest"), skips[l]], 1)
        t = conv(conv(t, 2 * depth + 2 * l), 2 * depth + 2 * l + 1)
    base = case["base"]
    hw, hb = p[off:off + 3 * base].reshape(base, 3), p[off + 3 * base:]
    out = torch.einsum("bczyx,cd->bdzyx", t, hw) + hb.reshape(1, 3, 1, 1, 1)
    out = out[0, :, :nodes[2], :nodes[1], :nodes[0]].reshape(3, -1)
    (out * torch.from_numpy(state["grad"]).to(dev).double()).sum().backward()
    return dict(out=out.detach(), grad_params=p.grad, grad_input=inp.grad)


def exact(case, seed):
    kind = case["kind"]
    dim, nel = case["dim"], _nel(case)
    if kind == "network":
        with U.Context(0) as ctx:   # the initial weights are the library's own
            ctx.mesh_q1(3, nel)
            ctx.learned_create(levels=case["depth"], base=case["base"], seed=int(seed) % 100000 + 1)
            params = ctx.learned_params()
        return _network_exact(case, _network_data(case, seed, params))
    if kind == "voronoi":
        return None   # the result of a sequential contest between the points, compared as it is
    m = _model(case, seed)
    if kind == "map":
        e, order, counts, xi = _located(m["x"], nel)
        out = torch.zeros((e.shape[0], 3), dtype=F64, device=e.device)
        out[:, :dim] = xi[order]
        return dict(perm=None, offsets=None, xi=out)
    if kind == "matrices":
        u, p = (m["u"], m["p"]) if m["u"] is not None else (None, None)
        K, f, Ge, Se, eta = _assembled(case, m, u, p)
        return dict(Ke=K, fe=f, Ge=Ge, Se=Se, eta=eta)
    if kind == "advect":
        u, _ = _flow(nel, _generator(seed + 1))
        en = _element_nodes(nel)
        dt = 0.3 / max(nel)
        x = m["x"]
        v = _velocity_at(x, u, nel, en)
        if case["order"] == 2:
            mid = x + 0.5 * dt * v
            inside = ((mid >= 0) & (mid <= 1)).all(1, keepdim=True)
            v = torch.where(inside, _velocity_at(mid, u, nel, en), v)
        x = x + dt * v
        return dict(x=x[:, 0], y=x[:, 1], z=x[:, 2] if dim == 3 else None, fell_back=None, left_mesh=None)
    if kind == "apply":
        nn = math.prod(n + 1 for n in nel)
        x = torch.randn(nn * dim, generator=_generator(seed + 1), device=_device(), dtype=F64)
        free = _free(case)
        y = _assembled(case, m, matrices=False, vector=(x * free).reshape(nn, dim)).reshape(-1)
        return dict(y=torch.where(free, y, x))
    # dense LU: up to the size that takes a few seconds
    if kind == "step" or dim * math.prod(n + 1 for n in nel) + math.prod(nel) > 20000:
        return None
    if kind == "solve":
        K, f, Ge, _, _ = _assembled(case, m)
        u, p = _direct(case, K, f, Ge)
        return dict(u=u, p=p)
    u, p = m["u"], m["p"]
    for _ in range(2):
        before = u
        K, f, Ge, _, _ = _assembled(case, m, u, p)
        u, p = _direct(case, K, f, Ge)
    return dict(u=u, p=p, residual=float((u - before).norm() / u.norm()))
