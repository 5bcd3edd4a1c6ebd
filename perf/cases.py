"""What a user of mag_b200 has it do, as cases that can be timed and checked.

Each case is one call sequence through the public entry points (``mag_b200.Chmc``): HMC
trajectories, molecular dynamics and its single steps, the Hamiltonian, Wilson loops, the
plaquette and the per-link demon sweep, on lattices from a few thousand sites to 32^4, thin
and smeared, Wilson and Iwasaki, free and constrained, FP64 and mixed precision, single
lattices and ensembles.  ``exact`` restates each of them in plain torch in 64 bits.

Configurations are links of equilibrium roughness in a random gauge: exp(i 0.27 H) with H
Gaussian in su(3) (average plaquette about 0.65, as Iwasaki beta = 2.25 has), transformed by
random SU(3) matrices at the sites.
"""
import math

import numpy as np
import torch

RECORD = ("h_old", "h_new", "delta_h", "kinetic_old", "kinetic_new", "action_old", "action_new", "plaq_sum_old",
          "plaq_sum_new", "rect_sum_old", "rect_sum_new", "uniform", "reunit_maxdev", "avg_plaquette")
C1 = -0.331
RHO = 0.1
E_MAX = 1e5
ROUGHNESS = 0.27


def _case(kind, dims, name=None, **kw):
    c = {"kind": kind, "L0": dims[0], "L1": dims[1], "L2": dims[2], "L3": dims[3], "action": "iwasaki", "beta": 2.25,
         "mag": 2, "n_stout": 0, "n_steps": 8, "precision": "fp64", "integrator": "fg", "accept": "metropolis"}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one trajectory of a small thin-link lattice with the demon accept: 33 short forces and
        # their updates, nothing fills the GPU
        _case("trajectory", (8, 8, 8, 8), "trajectory 8x8x8x8 thin", accept="demon"),
        # one FP64 trajectory of a production-like lattice smeared three times
        _case("trajectory", (16, 16, 16, 32), "trajectory 16x16x16x32", n_stout=3, n_steps=12),
        # one mixed-precision trajectory of the large lattice: the longest call of a run
        _case("trajectory", (32, 32, 32, 32), "trajectory 32x32x32x32 mixed", n_stout=3, n_steps=16,
              precision="mixed"),
        # an ensemble of uneven chains advancing together: n8 8^4, n12 12^4 and n16 16^4 lattices
        _case("ensemble", (8, 8, 8, 8), "ensemble of 24 mixed", n8=12, n12=8, n16=4, n_stout=1, precision="mixed"),
        # leapfrog molecular dynamics without accept step on a ragged free lattice, Wilson action
        _case("md", (6, 10, 14, 9), "md 6x10x14x9 Wilson", action="wilson", mag=0, n_stout=2, n_steps=6,
              integrator="leapfrog", beta=5.6),
        # the building block of a user's own integrator: P += dt F(U), FP64, through three smearing levels
        _case("kick", (24, 24, 24, 24), "kick 24x24x24x24", n_stout=3),
        # the same in mixed precision on uneven extents, one smearing level, free links
        _case("kick", (20, 12, 28, 18), "kick 20x12x28x18 mixed", n_stout=1, mag=0, precision="mixed"),
        # the Hamiltonian of a smeared lattice, as a user's own accept step takes it
        _case("hamiltonian", (24, 24, 24, 48), "hamiltonian 24x24x24x48", n_stout=3),
        # planar Wilson loops up to 8 x 8 of one lattice
        _case("loops", (24, 24, 24, 48), "loops 24x24x24x48", R=8, T=8),
        # the measurements taken on every chain of an ensemble: plaquette and loops up to 4 x 4
        _case("chains", (8, 8, 8, 8), "loops of 24 chains", n8=12, n12=8, n16=4, R=4, T=4, n_stout=1,
              precision="mixed"),
        # the smallest call: the average plaquette of a small lattice
        _case("plaquette", (8, 8, 8, 8), "plaquette 8x8x8x8"),
        # one per-link demon sweep, sequential over the links
        _case("demon", (6, 6, 6, 6), "demon 6x6x6x6", mag=0),
    ]


def _dims(rng, vmin, vmax, even, lmin=4, lmax=48):
    while True:
        v = math.exp(rng.uniform(math.log(vmin), math.log(vmax)))
        f = [math.exp(rng.uniform(-0.45, 0.45)) for _ in range(4)]
        scale = (v / (f[0] * f[1] * f[2] * f[3])) ** 0.25
        d = [int(round(scale * x)) for x in f]
        if even:
            d = [2 * max(1, round(x / 2)) for x in d]
        if all(lmin <= x <= lmax for x in d) and vmin <= d[0] * d[1] * d[2] * d[3] <= vmax:
            return d


def draw(rng):
    kind = rng.choice(["trajectory", "trajectory", "trajectory", "ensemble", "md", "md", "kick", "kick", "kick",
                       "hamiltonian", "loops", "loops", "chains", "plaquette", "demon"])
    kw = {"action": rng.choice(["iwasaki", "iwasaki", "wilson"]), "mag": rng.choice([0, 2, 2]),
          "n_stout": rng.randrange(4), "n_steps": rng.randrange(3, 17), "precision": rng.choice(["fp64", "mixed"]),
          "integrator": rng.choice(["fg", "fg", "leapfrog"]), "accept": rng.choice(["metropolis", "demon"])}
    kw["beta"] = round(rng.uniform(2.0, 2.6) if kw["action"] == "iwasaki" else rng.uniform(5.4, 6.2), 3)
    even = kw["mag"] == 2
    if kind in ("ensemble", "chains"):
        kw["n_steps"] = rng.randrange(3, 9)
        kw["n_stout"] = rng.randrange(3)
        kw.update(n8=rng.randrange(1, 17), n12=rng.randrange(0, 9), n16=rng.randrange(0, 5))
        if kind == "chains":
            kw.update(R=rng.randrange(2, 7), T=rng.randrange(2, 7))
        return _case(kind, (8, 8, 8, 8), **kw)
    if kind in ("trajectory", "md"):
        while True:
            d = _dims(rng, 1000, 400000, even)
            c = _case(kind, d, **kw)
            # half of the largest listed case's work
            if _forces(c) * _force_flops(c) * (1 if c["precision"] == "fp64" else 0.5) <= 0.25 * 64 * _force_flops(
                    {**c, "L0": 32, "L1": 32, "L2": 32, "L3": 32, "n_stout": 3, "action": "iwasaki"}):
                return c
    if kind in ("kick", "hamiltonian"):
        return _case(kind, _dims(rng, 2000, 700000, even), **kw)
    if kind == "loops":
        kw.update(R=rng.randrange(1, 11), T=rng.randrange(1, 13))
        return _case(kind, _dims(rng, 2000, 700000, even), **kw)
    if kind == "plaquette":
        return _case(kind, _dims(rng, 500, 300000, even), **kw)
    kw.update(precision="fp64", mag=0)
    return _case("demon", _dims(rng, 256, 4096, False), **kw)


# ------------------------------------------------------------------- inputs
def _dims_of(case):
    return (case["L0"], case["L1"], case["L2"], case["L3"])


def _chains(case):
    """Extents and beta of each chain of the case's context."""
    if case["kind"] in ("ensemble", "chains"):
        dims = [(8,) * 4] * case["n8"] + [(12,) * 4] * case["n12"] + [(16,) * 4] * case["n16"]
        return [(d, case["beta"] + 0.01 * (k % 7)) for k, d in enumerate(dims)]
    return [(_dims_of(case), case["beta"])]


def _volume(d):
    return d[0] * d[1] * d[2] * d[3]


def _su3_algebra(n, gen):
    """n Gaussian Hermitian traceless matrices, Tr H^2 of mean 8."""
    x = torch.randn((n, 3, 3, 2), generator=gen, device="cuda", dtype=torch.float64)
    a = torch.view_as_complex(x)
    h = (a + a.mH) * 0.5 * math.sqrt(2.0)
    t = torch.diagonal(h, dim1=-2, dim2=-1).sum(-1).real / 3
    return h - t[:, None, None] * torch.eye(3, device="cuda", dtype=torch.complex128)


def _links(dims, gen):
    """(V, 4, 3, 3) links on the GPU, x0 fastest."""
    V = _volume(dims)
    u = torch.linalg.matrix_exp(1j * ROUGHNESS * _su3_algebra(4 * V, gen))
    u = u.reshape(dims[3], dims[2], dims[1], dims[0], 4, 3, 3)
    g = torch.linalg.matrix_exp(2j * _su3_algebra(V, gen)).reshape(dims[3], dims[2], dims[1], dims[0], 3, 3)
    for mu in range(4):
        u[..., mu, :, :] = g @ u[..., mu, :, :] @ _at(g, mu, 1).mH
    return u.reshape(V, 4, 3, 3)


def _momenta(dims, gen):
    V = _volume(dims)
    return _su3_algebra(4 * V, gen).reshape(V, 4, 3, 3)


def _generator(seed):
    return torch.Generator("cuda").manual_seed(seed)


def _pinned(V, dtype=torch.complex128):
    return torch.empty((V, 4, 3, 3), dtype=dtype, pin_memory=True)


def prepare(case, seed):
    from mag_b200 import Chmc

    kw = {k: case[k] for k in ("action", "mag", "n_stout", "n_steps", "precision", "integrator", "accept")}
    chains = _chains(case)
    ctx = Chmc(chains=[{"dims": d, "beta": b} for d, b in chains], rho=RHO, c1=C1, e_max=E_MAX, seed=seed, **kw)
    state = {"case": case, "ctx": ctx, "seed": seed, "out": [], "narrow": {}}
    gen = _generator(seed)
    for k, (d, _) in enumerate(chains):
        buf = _pinned(_volume(d))
        buf.copy_(_links(d, gen))
        ctx.set_gauge(buf.numpy(), chain=k)
        state["out"].append(buf)
    if case["kind"] in ("md", "kick", "hamiltonian"):
        buf = _pinned(_volume(chains[0][0]))
        buf.copy_(_momenta(chains[0][0], gen))
        ctx.init_momentum(buf.numpy())
        state["momentum"] = buf
    torch.cuda.synchronize()
    return state


# --------------------------------------------------------------------- calls
def _links_out(state, k=0):
    """The links of a chain, in the precision they were integrated with."""
    state["ctx"].get_gauge(k, out=state["out"][k].numpy())
    return _computed(state, k, state["out"][k])


def _momentum_out(state):
    state["ctx"].get_momentum(out=state["momentum"].numpy())
    return _computed(state, "momentum", state["momentum"])


def _computed(state, key, buf):
    if state["case"]["precision"] != "mixed":
        return buf
    if key not in state["narrow"]:
        state["narrow"][key] = torch.empty(buf.shape, dtype=torch.complex64)
    return state["narrow"][key].copy_(buf)


def _records(case, recs):
    real = np.float32 if case["precision"] == "mixed" else np.float64
    return {"records": np.array([[r[k] for k in RECORD] for r in recs], real),
            "accept": np.array([r["accept"] for r in recs], np.int64)}


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind in ("trajectory", "ensemble"):
        res = _records(case, ctx.run_chmc(1)[0])
        res["links"] = [_links_out(state, k) for k in range(ctx.n_chains)]
        return res
    if kind == "md":
        ctx.force_gradient_integrator()
        return {"links": _links_out(state), "momentum": _momentum_out(state)}
    if kind == "kick":
        ctx.evolve_momentum(0.02)
        return {"momentum": _momentum_out(state)}
    if kind == "hamiltonian":
        h, parts = ctx.get_hamiltonian()
        return {"hamiltonian": h, "kinetic": parts[0], "action": parts[1]}
    if kind == "loops":
        return {"loops": ctx.wilson_loops(case["R"], case["T"])}
    if kind == "chains":
        return {"plaquette": np.array([ctx.avg_plaquette(k) for k in range(ctx.n_chains)]),
                "loops": np.stack([ctx.wilson_loops(case["R"], case["T"], chain=k) for k in range(ctx.n_chains)])}
    if kind == "plaquette":
        return {"plaquette": ctx.avg_plaquette()}
    d = ctx.demon_microcanonical(1, E_MAX, seed=state["seed"], update_links=True)
    return {"energy": d["demon_energy"], "accepted": d["accepted"], "rejected": d["rejected"],
            "links": _links_out(state)}


# ---------------------------------------------------------------------- work
def _forces(case):
    return case["n_steps"] * (4 if case["integrator"] == "fg" else 1)


def _force_flops(case):
    """One force of one site: staples, and per smearing level the forward step, Lambda and the
    chain rule (complex product of 3x3 matrices 198, of which special unitary ones need 174)."""
    staple = 33000 if case["action"] == "iwasaki" else 9000
    V = sum(_volume(d) for d, _ in _chains(case))
    return V * (staple + case["n_stout"] * (10500 + 5700 + 28500))


def work(case):
    kind = case["kind"]
    V = sum(_volume(d) for d, _ in _chains(case))
    link, alg = 576, 256  # bytes of a site's four links and of four algebra elements in FP64
    action = 6 * 1400 if case["action"] == "iwasaki" else 6 * 420
    smear = case["n_stout"] * 10500
    if kind in ("trajectory", "ensemble"):
        return {"bytes": 2.0 * V * link,
                "flops": float(_forces(case) * _force_flops(case) + 2 * V * (action + smear) + V * 6 * 420)}
    if kind == "md":
        return {"bytes": 2.0 * V * (link + alg), "flops": float(_forces(case) * _force_flops(case))}
    if kind == "kick":
        return {"bytes": 1.0 * V * (link + 2 * alg), "flops": float(_force_flops(case))}
    if kind == "hamiltonian":
        return {"bytes": 1.0 * V * (link + alg), "flops": float(V * (action + smear))}
    if kind in ("loops", "chains"):
        # spatial lines once per direction and length, then one trace of a product per loop
        return {"bytes": 1.0 * V * link, "flops": float(V * 3 * case["R"] * (198 + 36 * case["T"]))}
    if kind == "plaquette":
        return {"bytes": 1.0 * V * link, "flops": float(V * 6 * 420)}
    return {"bytes": 2.0 * V * link, "flops": float(V * 4 * 168 * 700)}


# --------------------------------------------------------- 64-bit restatement
def _at(a, mu, k):
    """a(x + k e_mu) of a field indexed [x3, x2, x1, x0, ...]."""
    return torch.roll(a, -k, dims=3 - mu)


def _split(u, dims):
    u = u.reshape(dims[3], dims[2], dims[1], dims[0], 4, 3, 3)
    return [u[..., mu, :, :].contiguous() for mu in range(4)]


def _join(u):
    return torch.stack(u, dim=-3).reshape(-1, 4, 3, 3)


def _retr(a, b):
    """Re Tr a b^dag at every site."""
    return (a.real * b.real + a.imag * b.imag).sum((-1, -2))


def _herm(m):
    """Hermitian traceless part."""
    h = (m + m.mH) * 0.5
    t = torch.diagonal(h, dim1=-2, dim2=-1).sum(-1).real / 3
    return h - t[..., None, None] * torch.eye(3, device=m.device, dtype=m.dtype)


def _sums(u, rect):
    p = r = 0.0
    for mu in range(1, 4):
        for nu in range(mu):
            a = u[mu] @ _at(u[nu], mu, 1)
            b = u[nu] @ _at(u[mu], nu, 1)
            p = p + _retr(a, b).sum()
            if rect:
                x = a @ _at(_at(u[nu], mu, 1), nu, 1)
                y = u[nu] @ _at(u[nu] @ _at(u[mu], nu, 1), nu, 1)
                r = r + _retr(x, y).sum()
                x = u[mu] @ _at(u[mu] @ _at(u[nu], mu, 1), mu, 1)
                y = b @ _at(_at(u[mu], mu, 1), nu, 1)
                r = r + _retr(x, y).sum()
    return p, r


def _smear(u, levels):
    for _ in range(levels):
        new = []
        for mu in range(4):
            s = 0
            for nu in range(4):
                if nu == mu:
                    continue
                un = u[nu]
                s = s + un @ _at(u[mu], nu, 1) @ _at(un, mu, 1).mH
                s = s + _at(un.mH @ u[mu] @ _at(un, mu, 1), nu, -1)
            q = _herm(-1j * RHO * (s @ u[mu].mH))
            new.append(torch.linalg.matrix_exp(1j * q) @ u[mu])
        u = new
    return u


def _action(case, beta, u):
    """(action, plaquette sum, rectangle sum) of the smeared links."""
    u = _smear(u, case["n_stout"])
    p, r = _sums(u, True)
    if case["action"] == "iwasaki":
        return beta / 3 * (-(1 - 8 * C1) * p - C1 * r), p, r
    return -beta / 3 * p, p, r


def _kinds(case, dims):
    """Per direction: which links are constrained at all, first and last of their segment."""
    m, out = case["mag"], []
    x = torch.meshgrid(*[torch.arange(n, device="cuda") for n in dims[::-1]], indexing="ij")[::-1]
    for mu in range(4):
        on = torch.full(dims[::-1], m > 0, device="cuda")
        for i in range(4):
            if m and i != mu:
                on = on & (x[i] % m == 0)
        out.append((on, on & (x[mu] % max(m, 1) == 0), on & (x[mu] % max(m, 1) == m - 1)))
    return out


def _force(case, beta, u, kinds):
    v = [a.detach().requires_grad_(True) for a in u]
    with torch.enable_grad():
        s = _action(case, beta, v)[0]
        grad = torch.autograd.grad(s, v)
    f = []
    for mu in range(4):
        g = -_herm(1j * u[mu] @ grad[mu].mH)
        if case["mag"]:
            on, _, last = kinds[mu]
            pair = _at(g, mu, 1) - u[mu].mH @ g @ u[mu]
            g = torch.where(on[..., None, None], pair, g)
            g = torch.where(last[..., None, None], torch.zeros_like(g), g)
        f.append(g)
    return f


def _evolve(case, u, p, eps, kinds):
    new = []
    for mu in range(4):
        e = torch.linalg.matrix_exp(1j * eps * p[mu])
        if not case["mag"]:
            new.append(e @ u[mu])
            continue
        on, first, last = (k[..., None, None] for k in kinds[mu])
        left = torch.where(on, _at(e, mu, -1), e) @ u[mu]
        a = torch.where(on & first, u[mu], left)
        new.append(torch.where(on & ~last, a @ e.mH, a))
    return new


def _integrate(case, beta, u, p, kinds):
    dt = 1.0 / case["n_steps"]

    def kick(at, eps):
        f = _force(case, beta, at, kinds)
        return [a + eps * b for a, b in zip(p, f)]

    if case["integrator"] == "leapfrog":
        u = _evolve(case, u, p, dt / 2, kinds)
        for i in range(case["n_steps"]):
            p = kick(u, dt)
            u = _evolve(case, u, p, dt if i < case["n_steps"] - 1 else dt / 2, kinds)
        return u, p
    al, be, ga = (3 - math.sqrt(3)) * dt / 6, dt / math.sqrt(3), (2 - math.sqrt(3)) * dt * dt / 12
    u = _evolve(case, u, p, al, kinds)
    for i in range(case["n_steps"]):
        for half in range(2):
            p = kick(_evolve(case, u, _force(case, beta, u, kinds), ga, kinds), dt / 2)
            u = _evolve(case, u, p, be if half == 0 else (2 * al if i < case["n_steps"] - 1 else al), kinds)
    new = []
    for a in u:  # rows 0 and 1 orthonormalised, row 2 their conjugate cross product
        r0 = a[..., 0, :] / torch.linalg.vector_norm(a[..., 0, :], dim=-1, keepdim=True)
        r1 = a[..., 1, :] - (r0.conj() * a[..., 1, :]).sum(-1, keepdim=True) * r0
        r1 = r1 / torch.linalg.vector_norm(r1, dim=-1, keepdim=True)
        new.append(torch.stack([r0, r1, torch.linalg.cross(r0, r1).conj()], dim=-2))
    return new, p


def _kinetic(p, kinds, mag):
    k = 0.0
    for mu in range(4):
        t = _retr(p[mu], p[mu])
        k += (t * (~kinds[mu][2]) if mag else t).sum().item()
    return 0.5 * k


def _philox(seed, c):
    """Philox-4x32-10 (Salmon et al., SC'11) of counters c (four uint64 arrays below 2^32)."""
    m32 = np.uint64(0xFFFFFFFF)
    k0, k1 = np.uint64(seed & 0xFFFFFFFF), np.uint64((seed >> 32) & 0xFFFFFFFF)
    for _ in range(10):
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> np.uint64(32)) ^ c[1] ^ k0, b & m32, (a >> np.uint64(32)) ^ c[3] ^ k1, a & m32]
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & m32, (k1 + np.uint64(0xBB67AE85)) & m32
    return c


def _philox_momenta(dims, seed, traj):
    n = 4 * _volume(dims)
    link, xi = np.arange(n, dtype=np.uint64), []
    for j in range(2):
        c = _philox(seed, [link] + [np.full(n, v, np.uint64) for v in (j, traj, 1)])
        for k in range(2):
            r = np.sqrt(-2 * np.log((c[2 * k].astype(np.float64) + 0.5) / 2.0**32))
            a = 2 * np.pi * ((c[2 * k + 1].astype(np.float64) + 0.5) / 2.0**32)
            xi += [r * np.cos(a), r * np.sin(a)]
    s2, s6 = 1 / math.sqrt(2), 1 / math.sqrt(6)
    p = np.zeros((n, 3, 3), np.complex128)
    p[:, 0, 0], p[:, 1, 1] = xi[2] * s2 + xi[7] * s6, -xi[2] * s2 + xi[7] * s6
    p[:, 2, 2] = -2 * xi[7] * s6
    for (i, j), a, b in (((0, 1), 0, 1), ((0, 2), 3, 4), ((1, 2), 5, 6)):
        p[:, i, j] = (xi[a] - 1j * xi[b]) * s2
        p[:, j, i] = p[:, i, j].conj()
    return torch.from_numpy(p).cuda().reshape(-1, 4, 3, 3)


def _uniform(seed, traj):
    c = _philox(seed, [np.array([v], np.uint64) for v in (0, 0, traj, 3)])
    return (int(c[0][0] >> np.uint64(5)) * 67108864.0 + int(c[1][0] >> np.uint64(6))) / 9007199254740992.0


def _trajectory(case, seed, dims, beta, u0):
    kinds = _kinds(case, dims)
    p0 = _split(_philox_momenta(dims, seed, 0), dims)
    s0, pl0, re0 = (float(v) for v in _action(case, beta, u0))
    k0 = _kinetic(p0, kinds, case["mag"])
    u1, p1 = _integrate(case, beta, u0, p0, kinds)
    s1, pl1, re1 = (float(v) for v in _action(case, beta, u1))
    k1 = _kinetic(p1, kinds, case["mag"])
    dh = (k1 - k0) + (s1 - s0)
    x = _uniform(seed, 0)
    ok = x < math.exp(min(0.0, -dh)) if case["accept"] == "metropolis" else max(abs(pl1 - pl0), abs(re1 - re0)) < E_MAX
    u = u1 if ok else u0
    plaq = float(_sums(u, False)[0]) / (18 * _volume(dims))
    rec = [k0 + s0, k1 + s1, dh, k0, k1, s0, s1, pl0, pl1, re0, re1, x, 0.0, plaq]
    return {"records": np.array([rec]), "accept": np.array([int(ok)], np.int64), "links": [_join(u)]}


def _loops(u, R, T, V):
    out = torch.zeros((R, T), dtype=torch.float64)
    times, t = [], None
    for k in range(T):
        t = u[3] if t is None else t @ _at(u[3], 3, k)
        times.append(t)
    for i in range(3):
        s = None
        for r in range(R):
            s = u[i] if s is None else s @ _at(u[i], i, r)
            for k in range(T):
                out[r, k] += _retr(s @ _at(times[k], i, r + 1), times[k] @ _at(s, 3, k + 1)).sum().item()
    return out / (3 * V)


def exact(case, seed):
    kind = case["kind"]
    chains = _chains(case)
    dims, beta = chains[0]
    V = _volume(dims)
    if kind in ("ensemble", "demon"):
        return None
    if kind in ("trajectory", "md") and V * _forces(case) * (1 + 3 * case["n_stout"]) > 1.5e6:
        return None
    if kind == "kick" and V * (1 + case["n_stout"]) > 1.5e6:
        return None
    gen = _generator(seed)
    with torch.no_grad():
        fields = [_split(_links(d, gen), d) for d, _ in chains]
        u = fields[0]
        if kind == "trajectory":
            return _trajectory(case, seed, dims, beta, u)
        if kind == "plaquette":
            return {"plaquette": float(_sums(u, False)[0]) / (18 * V)}
        if kind == "loops":
            return {"loops": _loops(u, case["R"], case["T"], V)}
        if kind == "chains":
            return {"plaquette": np.array([float(_sums(f, False)[0]) / (18 * _volume(d))
                                           for f, (d, _) in zip(fields, chains)]),
                    "loops": torch.stack([_loops(f, case["R"], case["T"], _volume(d))
                                          for f, (d, _) in zip(fields, chains)])}
        kinds = _kinds(case, dims)
        p = _split(_momenta(dims, gen), dims)
        if kind == "hamiltonian":
            s, k = float(_action(case, beta, u)[0]), _kinetic(p, kinds, case["mag"])
            return {"hamiltonian": s + k, "kinetic": k, "action": s}
        if kind == "kick":
            f = _force(case, beta, u, kinds)
            return {"momentum": _join([a + 0.02 * b for a, b in zip(p, f)])}
        u, p = _integrate(case, beta, u, p, kinds)
        return {"links": _join(u), "momentum": _join(p)}
