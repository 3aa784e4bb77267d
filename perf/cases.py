"""Measured cases of the framework, through the calls a host program makes.

A case is one of

  assemble  re-assembly for a kept contact list: the Newton iterate's node
            state on the device, then the tets, cohesive zones and contacts
            into the matrix and the rhs;
  attempt   two Newton iterates whose contacts differ: increment from the
            host, contact detection, structure, assembly (no solve);
  step      one implicit step from a saved frame: three Newton iterations
            (the reference's minIterations) of detection, structure, assembly
            and solve, then the accept and the damage commit;
  solve     the linear solve of an assembled system, to the call's default
            tolerance;
  forward   the warm-start network on every node of a model;
  gradient  the gradient of one training batch of that network.

The meshes are the package's own generators (beam, polycrystal cube between
rigid platens, batches of independent cubes, two colliding ice blocks).  What
the matrix's pattern hangs on is the model's and the same for every seed: the
mesh, which cohesive zones have failed, the contact list that an assembly or a
solve keeps, and the positions of the two iterates of an attempt.  Everything
else comes from the seed.
"""
from __future__ import annotations

import math
from functools import lru_cache

import numpy as np
import torch

from icflow_b200 import mesh as M
from icflow_b200.gpu_functionality import GPU_Functionality
from icflow_b200.model_prms import config_prms
from icflow_b200.warm_start import MLP

TIME_STEP = {"beam": 1e-4, "cube": 1e-5, "batch": 1e-5, "ice": 5e-6}


def _case(name, kind, model="", n=0, grains=0, mixed=False):
    return {"name": name, "kind": kind, "model": model, "n": n, "grains": grains, "mixed": mixed}


def listed():
    return [
        # the smallest model, launch and latency bound: a cantilever whose
        # 2304 tets are re-assembled thousands of times in a loading run
        _case("assemble beam", "assemble", "beam"),
        # the medium polycrystal, 196,608 tets and its contacts
        _case("assemble cube 32", "assemble", "cube", 32, 128),
        # the benchmark's polycrystal, 1,572,864 tets, in both precisions
        _case("assemble cube 64", "assemble", "cube", 64, 2048),
        _case("assemble cube 64 mixed", "assemble", "cube", 64, 2048, True),
        # sixteen uneven specimens in one launch, FP32-mixed as such batches run
        _case("assemble batch 16 mixed", "assemble", "batch", 16, 0, True),
        # Newton iterates of a contact that moves: the list changes each time
        _case("attempt cube 11", "attempt", "cube", 11, 9),
        _case("attempt cube 32", "attempt", "cube", 32, 128),
        # implicit steps of the colliding blocks, at the warm start's size and larger
        _case("step ice 8", "step", "ice", 8, 8),
        _case("step ice 22", "step", "ice", 22, 24),
        # the linear solve of the polycrystal under load
        _case("solve cube 15", "solve", "cube", 15, 24),
        _case("solve cube 32", "solve", "cube", 32, 128),
        # one training batch of the warm-start network, at the batch size it is
        # fitted with
        _case("gradient 4096", "gradient", "", 4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["assemble", "assemble", "assemble", "attempt", "attempt", "step", "solve", "solve",
                       "forward", "gradient"])
    if kind in ("forward", "gradient"):
        n = _log_int(rng, 300, 60000 if kind == "forward" else 30000)
        return {k: v for k, v in _case("", kind, "", n).items() if k != "name"}
    if kind == "step":
        model = "ice"
    elif kind == "assemble":
        model = rng.choice(["cube", "cube", "batch"])
    else:
        model = "cube"
    top = {"assemble": 40, "attempt": 32, "step": 22, "solve": 32}[kind]
    n = rng.randint(2, 12) if model == "batch" else _log_int(rng, 5, top)
    # the benchmark's grains hold 128 to 256 hexahedra each
    cells = n ** 3 if model == "cube" else n ** 2 * max(1, n // 2)
    grains = 0 if model == "batch" else max(2, cells // rng.randint(128, 256))
    mixed = kind in ("assemble", "attempt") and rng.random() < 0.4
    return {k: v for k, v in _case("", kind, model, n, grains, mixed).items() if k != "name"}


# ---- inputs --------------------------------------------------------------------

@lru_cache(maxsize=12)
def _mesh(model, n, grains):
    """(collection, initial velocities or None, grain pair of every CZ)."""
    if model == "beam":
        coll = M.cantilever()
        return coll, None, coll.meshes[0].cz_grains
    if model == "cube":
        coll = M.polycrystal(n=n, grains=grains, seed=0)
        return coll, None, coll.meshes[0].cz_grains
    if model == "batch":
        coll, _ = M.batched_specimens(n, seed=0)
        v0 = None
    else:
        coll, v0 = M.ice_impact(n=n, grains=grains, seed=1)
    pairs, at = [], 0
    for m in coll.meshes:  # grains numbered apart per body
        pairs.append(m.cz_grains + at)
        at += int(m.granule.max()) + 1
    return coll, v0, np.concatenate(pairs)


def _prms():
    return config_prms(penaltyK=1e8)


def _inputs(case, seed):
    """The frame of a run under way: node state, increment, per-boundary
    strengths, and cohesive zones of which a tenth are damaged and one in a
    hundred has failed."""
    model = case["model"]
    coll, v0, pairs = _mesh(model, case["n"], case["grains"])
    rng, fixed = np.random.default_rng([seed, 17]), np.random.default_rng([case["n"], case["grains"]])
    nn, nc = len(coll.x0), len(coll.czs)
    noise = lambda s, r=rng: (r.random((nn, 3)) - 0.5) * s  # noqa: E731
    h = TIME_STEP[model]
    failed = (fixed.random(nc) < 0.01).astype(np.int32)
    frame = noise(0.0)  # where the kept contact list was found
    if model == "ice":  # 22 us after the blocks' start: just in contact
        t = 2.2e-5 * (1 + 0.02 * rng.random())
        u, v, a = v0 * t + noise(1e-7), v0 + noise(1e-2), noise(1e2)
        dus = [v * h]
    elif model == "beam":
        u, v, a = noise(2e-6), noise(1e-2), noise(1.0)
        dus = [noise(2e-6)]
    else:  # compressed along z by 1e-4
        frame = noise(2e-9, fixed)
        frame[:, 2] -= 1e-4 * (coll.x0[:, 2] - 0.5e-3)
        of = fixed if case["kind"] == "attempt" else rng
        u, dus = frame + noise(2e-9, of), [noise(2e-9, of), noise(2e-9, of)]
        v, a = noise(1e-3), noise(1e-1)
    for z in (frame, u, v, a, *dus):
        z[coll.anchored] = 0.0
    # largest openings so far from 1 to 10 % of the shortest critical one
    d = 0.02 + 0.18 * rng.random((nc, 6))
    strength = M.lognormal_strengths(nc, seed=seed, granule_pairs=pairs)
    q = _ppr(_prms(), strength.max())
    d *= 0.5 * min(q["deln"], q["delt"])
    d[rng.random(nc) >= 0.1] = 0.0
    # a beam and a batch of independent specimens run without contact
    return dict(coll=coll, contact=model in ("cube", "ice"), h=h, frame=frame, u=u, v=v, a=a, dus=dus,
                strength=strength, pmax=np.ascontiguousarray(d[:, :3]), tmax=np.ascontiguousarray(d[:, 3:]),
                failed=failed)


def _net_inputs(case, seed):
    """Trained-like parameters, normalised inputs of the impact's scale, and
    the corrections they are fitted to."""
    rng = np.random.default_rng([seed, 29])
    n = case["n"]
    scale = np.repeat([1e-4, 2.5, 1e4, 1e-5, 1e-5], 3)
    x = (rng.normal(size=(n, 15)) * scale).astype(np.float32)
    y = rng.normal(size=(n, 3)).astype(np.float32)
    w = [rng.normal(0, math.sqrt(2 / 15), (64, 15)), rng.normal(0, 0.1, 64), rng.normal(0, math.sqrt(2 / 64), (64, 64)),
         rng.normal(0, 0.1, 64), rng.normal(0, 0.125, (3, 64)), rng.normal(0, 0.1, 3)]
    norm = np.concatenate([rng.normal(0, 0.1, 15) * scale, 1 / scale, np.ones(3)]).astype(np.float32)
    return x, y, [p.astype(np.float32) for p in w], norm


class _DeviceArray:
    """A device buffer of a context as torch sees it; it keeps the context."""

    def __init__(self, gf, ptr, shape, kind):
        self.gf = gf
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": kind, "version": 3}


def _views(gf, *names):
    b = gf.DeviceBuffers()
    what = {"vals": (b.vals, (b.nnz, 3, 3), "<f8"), "rhs": (b.rhs, (b.N, 3), "<f8"),
            "rows": (b.csr_rows, (b.N + 1,), "<i4"), "cols": (b.csr_cols, (b.nnz,), "<i4")}
    return {k: torch.as_tensor(_DeviceArray(gf, *what[k]), device="cuda") for k in names}


def _load(inp, mixed):
    """A context that holds the model and its frame."""
    gf = GPU_Functionality(0)
    gf.prms = _prms()
    gf.mc = inp["coll"]
    gf.SetConstants()
    gf.SetPrecision(1 if mixed else 0)
    gf.TransferStaticDataToDevice()
    gf.SetCZStrengths(inp["strength"], inp["strength"])
    gf.TransferPCSR(inp["pmax"], inp["tmax"], inp["failed"])
    gf.TransferNodesToGPU(inp["frame"], inp["v"], inp["a"])
    if inp["contact"]:
        gf.DetectContacts()
    gf.CreateStructure(copy_back=False)
    gf.SetNodeState(inp["u"], inp["v"], inp["a"])
    gf.SetDU(inp["dus"][0])
    gf.InferTentativeValues(inp["h"])
    return gf


def prepare(case, seed):
    if case["kind"] in ("forward", "gradient"):
        x, y, w, norm = _net_inputs(case, seed)
        net = MLP(0)
        net.set_params(np.concatenate([p.ravel() for p in w]), norm)
        return dict(kind=case["kind"], net=net, x=x, y=y)
    inp = _inputs(case, seed)
    gf = _load(inp, case["mixed"])
    s = dict(inp, kind=case["kind"], gf=gf)
    if case["kind"] == "assemble":
        s["out"] = _views(gf, "vals", "rhs")
    elif case["kind"] == "solve":
        gf.AssembleElemsAndCZs(inp["h"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "forward":
        return s["net"].forward(s["x"])
    if kind == "gradient":
        return s["net"].grad(s["x"], s["y"])
    gf = s["gf"]
    if kind == "assemble":
        gf.InferTentativeValues(s["h"])
        c = gf.AssembleElemsAndCZs(s["h"])
        return dict(s["out"], counts=[c.nCZDamaged, c.nCZFailedThisStep, c.nImpactsActive])
    if kind == "solve":
        return gf.Solve(want_dx=True)[2]
    if kind == "attempt":
        for du in s["dus"]:
            gf.SetDU(du)
            gf.InferTentativeValues(s["h"])
            gf.DetectContacts()
            gf.CreateStructure(copy_back=False)
            c = gf.AssembleElemsAndCZs(s["h"])
        return dict(_views(gf, "rows", "cols", "vals", "rhs"), impacts=gf.c_itet,
                    counts=[c.nCZDamaged, c.nCZFailedThisStep, c.nImpactsActive])
    # one step from the saved frame
    h = s["h"]
    gf.TransferPCSR(s["pmax"], s["tmax"], s["failed"])
    gf.SetNodeState(s["u"], s["v"], s["a"])
    gf.SetDU(s["dus"][0])
    for _ in range(3):
        gf.InferTentativeValues(h)
        gf.DetectContacts()
        gf.CreateStructure(copy_back=False)
        gf.AssembleElemsAndCZs(h)
        gf.Solve()
        gf.ApplyDx()
    gf.AcceptTentativeValues(h)
    cz = gf.TransferUpdatedStateToHost(want_forces=False)
    u, v, a, _ = gf.GetNodeState()
    return dict(u=u, v=v, a=a, pmax=cz["pmax"], tmax=cz["tmax"], failed=cz["failed"], avg=cz["avg"])


# ---- work ------------------------------------------------------------------------

@lru_cache(maxsize=32)
def _sizes(model, n, grains):
    """Tets, CZs, nodes, rows, surface elements, blocks and contacts."""
    coll, _, _ = _mesh(model, n, grains)
    key = []
    for units in (coll.elems, coll.czs):
        al = coll.alt[units].astype(np.int64)
        i, j = np.triu_indices(al.shape[1])
        lo, hi = np.minimum(al[:, i], al[:, j]), np.maximum(al[:, i], al[:, j])
        key.append(np.unique((lo << 32 | hi)[lo >= 0]))
    blocks = len(np.unique(np.concatenate(key)))
    # contacts: about two thirds of the CZs on a polycrystal (split nodes)
    contacts = int(0.65 * len(coll.czs)) if model == "cube" else (n * n * 8 if model == "ice" else 0)
    return dict(tets=len(coll.elems), czs=len(coll.czs), nodes=len(coll.x0), rows=coll.n_active,
                surf=len(coll.selem), blocks=blocks, contacts=contacts)


def work(case):
    """Bytes with every input read once and every output written once, and the
    floating-point operations of the formulas."""
    kind, n = case["kind"], case["n"]
    if kind in ("forward", "gradient"):
        mac = 15 * 64 + 64 * 64 + 64 * 3
        back = kind == "gradient"
        return {"bytes": 4 * n * 18 + 4 * 5315 * (2 if back else 1), "flops": 2 * mac * n * (3 if back else 1)}
    z = _sizes(case["model"], n, case["grains"])
    asm = dict(
        bytes=(72 * z["blocks"] + 24 * z["rows"] + 168 * z["nodes"] + 16 * z["tets"] + 180 * z["czs"] +
               16 * z["contacts"]),
        flops=1100 * z["tets"] + 1500 * z["czs"] + 2000 * z["contacts"])
    if kind == "assemble":
        return asm
    # detection reads every surface element and node, structure writes the
    # columns and the contacts' blocks
    it = dict(bytes=asm["bytes"] + 16 * z["surf"] + 32 * z["nodes"] + 4 * z["blocks"] + 32 * z["contacts"],
              flops=asm["flops"] + 100 * z["surf"])
    if kind == "attempt":
        return {k: 2 * v for k, v in it.items()}
    # MINRES iterations to the default tolerance, from its runs
    its = 24 * n + 12 if case["model"] == "ice" else 45 * n + 20
    solve = dict(bytes=76 * z["blocks"] + 52 * z["rows"], flops=its * (36 * z["blocks"] + 60 * z["rows"]))
    if kind == "solve":
        return solve
    return {k: 3 * (it[k] + solve[k]) for k in solve}


# ---- the same values in plain 64-bit arithmetic -----------------------------------

def _ppr(p, strength):
    """Constants of the Park-Paulino-Roesler law for one strength (or an array)."""
    a, b, rn, rt = p.alpha, p.beta, p.lambda_n, p.lambda_t
    m, n = a * (a - 1) * rn * rn / (1 - a * rn * rn), b * (b - 1) * rt * rt / (1 - b * rt * rt)
    gn, gt = (a / m) ** m, (b / n) ** n
    if p.phi_n < p.phi_t:
        gt = -p.phi_t * gt
    else:
        gn = -p.phi_n * gn
    deln = p.phi_n / strength * a * rn * (1 - rn) ** (a - 1) * (a / m + 1) * (a / m * rn + 1) ** (m - 1)
    delt = p.phi_t / strength * b * rt * (1 - rt) ** (b - 1) * (b / n + 1) * (b / n * rt + 1) ** (n - 1)
    return dict(m=m, n=n, gn=gn, gt=gt, deln=deln, delt=delt, mnt=max(p.phi_n - p.phi_t, 0.0),
                mtn=max(p.phi_t - p.phi_n, 0.0))


def _axis(a, p, gam, mac, x):
    """One axis of the PPR potential: its factor and two derivatives."""
    o, s = 1 - x, p / a + x
    f = gam * o ** a * s ** p + mac
    d = p * o ** a * s ** (p - 1) - a * o ** (a - 1) * s ** p
    dd = ((p * p - p) * o ** a * s ** (p - 2) + (a * a - a) * o ** (a - 2) * s ** p -
          2 * a * p * o ** (a - 1) * s ** (p - 1))
    return f, d, dd


def _law(p, strength, pmax, tmax, opn, opt):
    """Tn, Tt, Dnn, Dtt, Dnt and failure of every Gauss point."""
    q = _ppr(p, strength)
    normal = lambda x: _axis(p.alpha, q["m"], q["gn"], q["mnt"], x / q["deln"])  # noqa: E731
    shear = lambda x: _axis(p.beta, q["n"], q["gt"], q["mtn"], x / q["delt"])  # noqa: E731
    cn, ct = q["gn"] / q["deln"], q["gt"] / q["delt"]
    cnn, ctt = cn / q["deln"], ct / q["delt"]
    zero = torch.zeros_like(opn)
    touch = opn < 0
    now = torch.where(touch, zero, opn)
    nf, nd, ndd = normal(now)
    tf, td, tdd = shear(opt)
    tn, tt = cn * nd * tf, ct * td * nf
    fail = (opn > q["deln"]) | (opt > q["delt"]) | (tt < -1e-9)
    fail |= (opt > q["delt"] * p.lambda_t / 5) & (tt < 0.05 * strength)
    fail |= ~touch & ((tn < -1e-9) | ((opn > q["deln"] * p.lambda_n / 5) & (tn < 0.05 * strength)))
    pf, pd, _ = normal(pmax)
    mf, md, _ = shear(tmax)
    ndd0, tdd0 = normal(zero)[2], shear(zero)[2]
    nload, tload = ~touch & (opn >= pmax), opt >= tmax
    both = nload & tload
    # normal: loading, or along the secant of the largest opening
    mf_n = torch.where(both, tf, mf)
    peak = cn * pd * mf
    slope = torch.where(pmax > 0, peak / torch.where(pmax > 0, pmax, zero + 1), cnn * ndd0 * mf)
    unload = torch.where((pmax > 0) | touch, slope * opn, zero)
    Tn = torch.where(nload, cn * nd * mf_n, unload)
    Dnn = torch.where(nload, cnn * ndd * mf_n, slope)
    # shear, against the normal factor of the largest (or zero, in touch) opening
    pf_t = torch.where(touch | both, nf, pf)
    peak = ct * md * pf_t
    slope = torch.where(tmax > 0, peak / torch.where(tmax > 0, tmax, zero + 1), ctt * tdd0 * pf_t)
    unload = torch.where(tmax > 0, slope * opt, zero)
    Tt = torch.where(tload, ct * td * pf_t, unload)
    Dtt = torch.where(tload, ctt * tdd * pf_t, slope)
    Dnt = torch.where(both, cn * ct * nd * td, zero)
    return Tn, Tt, Dnn, Dtt, Dnt, fail


def _tets(p, h, X, C, v, a):
    """Blocks [e, 4, 4, 3, 3] and rhs [e, 4, 3] of corotational tets."""
    edge = X[:, 1:] - X[:, :1]
    V = torch.linalg.det(edge).abs() / 6
    g = torch.linalg.inv(edge).transpose(1, 2)
    g = torch.cat([-g.sum(1, keepdim=True), g], 1)

    def frame(x):
        c0 = torch.nn.functional.normalize(x[:, 1] - x[:, 0], dim=1)
        c1 = torch.nn.functional.normalize(torch.linalg.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0]), dim=1)
        return torch.stack([c0, c1, torch.linalg.cross(c1, c0)], 2)

    R = frame(C) @ frame(X).transpose(1, 2)
    lam, mu = p.nu * p.Y / ((1 + p.nu) * (1 - 2 * p.nu)), p.Y / (2 * (1 + p.nu))
    g = g @ R.transpose(1, 2)  # gradients in the current frame
    gg = torch.einsum("eai,ebj->eabij", g, g)
    eye = torch.eye(3, dtype=X.dtype, device=X.device)
    dot = torch.einsum("eabii->eab", gg)
    K = V[:, None, None, None, None] * (lam * gg + mu * gg.transpose(3, 4) + mu * dot[..., None, None] * eye)
    mass = p.rho / 20 * V[:, None, None] * (1 + torch.eye(4, dtype=X.dtype, device=X.device))
    moved = C - X @ R.transpose(1, 2)
    f = torch.einsum("eabij,ebj->eai", K, moved)
    damp = p.dampingMass * mass @ v + p.dampingStiffness * torch.einsum("eabij,ebj->eai", K, v)
    rhs = -f - damp - mass @ a
    rhs[:, :, 2] += (p.gravity * p.rho / 4 * V)[:, None]
    sc = 1 + p.dampingStiffness * p.NewmarkGamma / (h * p.NewmarkBeta)
    mc = (1 / (h * h) + p.dampingMass * p.NewmarkGamma / h) / p.NewmarkBeta
    return sc * K + mc * mass[..., None, None] * eye, rhs


def _zones(p, strength, C, pmax, tmax):
    """Blocks [c, 6, 6, 3, 3] and rhs [c, 6, 3] of the cohesive zones."""
    mid = 0.5 * (C[:, :3] + C[:, 3:])
    n = torch.linalg.cross(mid[:, 1] - mid[:, 0], mid[:, 0] - mid[:, 2])
    area = n.norm(dim=1)  # twice the mid-plane triangle's
    r0 = torch.nn.functional.normalize(mid[:, 1] - mid[:, 0], dim=1)
    r2 = n / area[:, None]
    R = torch.stack([r0, torch.linalg.cross(r2, r0), r2], 1)
    sf = torch.tensor([[1 / 6, 1 / 6, 2 / 3], [1 / 6, 2 / 3, 1 / 6], [2 / 3, 1 / 6, 1 / 6]], dtype=C.dtype, device=C.device)
    gap = torch.einsum("cij,gn,cnj->cgi", R, sf, C[:, :3] - C[:, 3:])
    opn, opt = gap[..., 2], gap[..., :2].norm(dim=2)
    Tn, Tt, Dnn, Dtt, Dnt, fail = _law(p, strength[:, None], pmax, tmax, opn, opt)
    e = torch.where(opt[..., None] < 1e-20, torch.zeros_like(gap[..., :2]), gap[..., :2] / opt.clamp_min(1e-300)[..., None])
    T = torch.cat([Tt[..., None] * e, Tn[..., None]], 2)
    ee = e[..., :, None] * e[..., None, :]
    eye = torch.eye(2, dtype=C.dtype, device=C.device)
    D = torch.zeros(*opn.shape, 3, 3, dtype=C.dtype, device=C.device)
    D[..., :2, :2] = Dtt[..., None, None] * ee + (Tt / opt.clamp_min(1e-300))[..., None, None] * (eye - ee)
    D[..., 2, 2] = Dnn
    D[..., :2, 2] = D[..., 2, :2] = Dnt[..., None] * e
    live = (~fail.any(1)).to(C.dtype) * area / 6
    s = torch.cat([sf, -sf], 1)
    K = torch.einsum("c,ga,gb,cki,cgkl,clj->cabij", live, s, s, R, D, R)
    return K, -torch.einsum("c,ga,cki,cgk->cai", live, s, R, T)


def _contacts(p, x):
    """Blocks [i, 4, 4, 3, 3] and rhs [i, 4, 3] of node-face contacts x [i, 4, 3]:
    half the penalty times the squared distance to the triangle."""
    P, A = x[:, 0], x[:, 1:]
    dots = lambda y, z: (y * z).sum(1)  # noqa: E731
    # closest feature: the foot point on the plane, else the nearest edge's
    e0, e1, w = A[:, 1] - A[:, 0], A[:, 2] - A[:, 0], P - A[:, 0]
    a, b, c, d, e = dots(e0, e0), dots(e0, e1), dots(e1, e1), dots(e0, w), dots(e1, w)
    det = a * c - b * b
    s, t = (c * d - b * e) / det, (a * e - b * d) / det
    inside = (s >= 0) & (t >= 0) & (s + t <= 1)
    bary = torch.stack([1 - s - t, s, t], 1)
    best = torch.where(inside, torch.zeros_like(s), torch.full_like(s, math.inf))
    feature = torch.zeros(len(x), dtype=torch.long, device=x.device)  # 0 plane, 1-3 edge, 4-6 vertex
    for k, (i, j) in enumerate(((0, 1), (1, 2), (2, 0))):
        g = A[:, j] - A[:, i]
        r = (dots(P - A[:, i], g) / dots(g, g)).clamp(0, 1)
        d2 = (P - A[:, i] - r[:, None] * g).square().sum(1)
        new = ~inside & (d2 < best)
        best = torch.where(new, d2, best)
        feature = torch.where(new, torch.where(r <= 0, 4 + i, torch.where(r >= 1, 4 + j, 1 + k)), feature)
        w3 = torch.zeros_like(bary)
        w3[:, i], w3[:, j] = 1 - r, r
        bary = torch.where(new[:, None], w3, bary)

    def plane(y):
        nrm = torch.linalg.cross(y[2] - y[1], y[3] - y[1])
        return torch.dot(y[0] - y[1], nrm) ** 2 / torch.dot(nrm, nrm)

    def edge(i, j):
        def f(y):
            q, g = y[0] - y[1 + i], y[1 + j] - y[1 + i]
            return torch.dot(q, q) - torch.dot(q, g) ** 2 / torch.dot(g, g)
        return f

    def vertex(i):
        return lambda y: (y[0] - y[1 + i]).square().sum()

    K = torch.zeros(len(x), 4, 3, 4, 3, dtype=x.dtype, device=x.device)
    grad = torch.zeros(len(x), 4, 3, dtype=x.dtype, device=x.device)
    for k, f in enumerate([plane, edge(0, 1), edge(1, 2), edge(2, 0), vertex(0), vertex(1), vertex(2)]):
        at = torch.nonzero(feature == k).squeeze(1)
        if len(at):
            K[at] = torch.func.vmap(torch.func.hessian(f))(x[at])
            grad[at] = torch.func.vmap(torch.func.grad(f))(x[at])
    F = 0.5 * p.penaltyK * grad[:, 0]
    rhs = torch.cat([-F[:, None], bary[:, :, None] * F[:, None]], 1)
    return 0.5 * p.penaltyK * K.permute(0, 1, 3, 2, 4), rhs


def _exact_assembly(case, seed):
    """The matrix's upper blocks, rows then columns ascending, and the rhs."""
    inp, p = _inputs(case, seed), _prms()
    coll, h = inp["coll"], inp["h"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    T = lambda z: torch.as_tensor(np.asarray(z), device=dev)  # noqa: E731
    u, v, a, du = T(inp["u"]), T(inp["v"]), T(inp["a"]), T(inp["dus"][0])
    X, alt = T(coll.x0), T(coll.alt).long()
    # Newmark predictor of the iterate
    beta, gamma = p.NewmarkBeta, p.NewmarkGamma
    an = a * (1 - 1 / (2 * beta)) + du / (h * h * beta) - v / (h * beta)
    vn = v + h * ((1 - gamma) * a + gamma * an)
    C = X + u + du
    parts = []
    el = T(coll.elems).long()
    parts.append((el, *_tets(p, h, X[el], C[el], vn[el], an[el])))
    live = T(inp["failed"]) == 0
    if int(live.sum()):
        cz = T(coll.czs).long()[live]
        parts.append((cz, *_zones(p, T(inp["strength"])[live], C[cz], T(inp["pmax"])[live], T(inp["tmax"])[live])))
    if inp["contact"]:  # the kept list
        gf = _load(inp, False)
        imp = torch.as_tensor(gf.c_itet, device=dev).long()
        gf.close()
        imp = imp[(alt[imp] >= 0).any(1)]
        if len(imp):
            parts.append((imp, *_contacts(p, C[imp])))
    keys, blocks = [], []
    N = coll.n_active
    rhs = torch.zeros(N, 3, dtype=torch.float64, device=dev)
    for units, K, r in parts:
        al = alt[units]
        k = al.shape[1]
        row, col = al[:, :, None].expand(-1, k, k), al[:, None, :].expand(-1, k, k)
        keep = (row >= 0) & (col >= row)
        keys.append((row << 32 | col)[keep])
        blocks.append(K[keep])
        rhs.index_add_(0, al[al >= 0], r[al >= 0])
        del K
    keys = torch.cat(keys)
    slots, at = torch.unique(keys, return_inverse=True)
    vals = torch.zeros(len(slots), 3, 3, dtype=torch.float64, device=dev)
    vals.index_add_(0, at, torch.cat(blocks))
    return dict(vals=vals, rhs=rhs, counts=None)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("forward", "gradient"):
        x, y, w, norm = _net_inputs(case, seed)
        W1, b1, W2, b2, W3, b3 = w64 = [torch.tensor(p, dtype=torch.float64, requires_grad=True) for p in w]
        sh, sc = torch.tensor(norm[:15]).double(), torch.tensor(norm[15:30]).double()
        gelu = torch.nn.functional.gelu
        z = gelu((torch.tensor(x).double() - sh) * sc @ W1.T + b1)
        out = gelu(z @ W2.T + b2) @ W3.T + b3
        if kind == "forward":
            return out.detach()
        loss = (out - torch.tensor(y).double()).square().mean()
        g = torch.autograd.grad(loss, w64)
        return torch.cat([z.reshape(-1) for z in g]), float(loss)
    if kind == "assemble":
        return _exact_assembly(case, seed)
    if kind == "solve":
        # the assembled system is the input; dense where that fits the time
        if _sizes(case["model"], case["n"], case["grains"])["rows"] > 8000:
            return None
        inp = _inputs(case, seed)
        gf = _load(inp, case["mixed"])
        gf.AssembleElemsAndCZs(inp["h"])
        b = {k: z.clone() for k, z in _views(gf, "rows", "cols", "vals", "rhs").items()}
        gf.close()
        N = len(b["rhs"])
        row = torch.repeat_interleave(torch.arange(N, device="cuda"), b["rows"].diff().long())
        col = b["cols"].long()
        A = torch.zeros(N, 3, N, 3, dtype=torch.float64, device="cuda")
        A[col, :, row] = b["vals"].transpose(1, 2)
        A[row, :, col] = b["vals"]
        return torch.linalg.solve(A.reshape(3 * N, 3 * N), b["rhs"].reshape(-1)).reshape(N, 3)
    return None  # a step's and an attempt's contact lists are decided by the path itself
