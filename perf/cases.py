"""Workloads of this package as a user's program runs them, with 64-bit references.

Every case goes through a public entry point:

  md       SeAEvaluator, compressed model, one water frame per step: from host
           coordinates to host results (compute), on the device (replay), or
           with a neighbor list kept with a skin between rebuilds
  batch    BatchEvaluator: many uneven water / Cu frames in one step
  plain    SeAEvaluator, uncompressed model in FP64
  train    SeATrainer.train_step: energy / force / virial loss, backward, Adam
  engine   ForwardLower: an MD engine's extended system and list
  tabulate torch.ops.deepmd.tabulate_fusion_se_a with its backward, and with
           the backward of that where ``second`` is set
  ops      copy_coord, build_nlist, prod_env_mat_a, prod_force_a and
           prod_virial_a one after another

Sizes: 64, 4,096 and 110,592 molecules are the 192-, 12,288- and 331,776-atom
water boxes of the benchmark; the others are odd sizes between them. The model
is the benchmark's (rcut 6, sel 46 / 92, embedding 25-50-100, fitting 3 x 240;
a third species with sel 60 for the batch).

The network of the compressed model runs in FP32, so a program that keeps its
state in FP32 is what takes its energies, forces and virials here; the FP64
paths return FP64.
"""

import importlib
import importlib.util
import math
import os
import sys

import numpy as np
import torch

NAME = "deepmd_kit_lr_pt_b200"
RCUT, SMTH, SKIN = 6.0, 0.5, 2.0
NEURON, AXIS, FITTING = (25, 50, 100), 16, (240, 240, 240)
PREFS = (0.02, 1000.0, 0.02)  # energy, force and virial prefactors of the loss
LR = 1e-4


def _package(name):
    """Module ``name`` of this repository's package (its folder's name is no
    Python identifier)."""
    if NAME not in sys.modules:
        d = os.path.join(os.getcwd(), "deepmd-kit-lr-pt_b200")
        spec = importlib.util.spec_from_file_location(
            NAME, os.path.join(d, "__init__.py"), submodule_search_locations=[d])
        sys.modules[NAME] = mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
    return importlib.import_module(f"{NAME}.{name}")


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # a small box in a host program's MD loop: latency of one call
        {"name": "md-192-host", "kind": "md", "molecules": 64, "form": "host"},
        # the benchmark's frame, coordinates already on the device
        {"name": "md-12288", "kind": "md", "molecules": 4096, "form": "device"},
        # the largest frame, stepping with a list kept between rebuilds
        {"name": "md-331776-skin", "kind": "md", "molecules": 110592, "form": "skin"},
        # labelling many small structures at once, three species
        {"name": "batch-128", "kind": "batch", "frames": 128, "atoms": 3000},
        # the uncompressed model in FP64, an odd size
        {"name": "plain-f64-3993", "kind": "plain", "molecules": 1331},
        # training in FP32 (the benchmark's batch) and in FP64 (small batch)
        {"name": "train-f32-16", "kind": "train", "frames": 16, "molecules": 64,
         "dtype": "float32"},
        {"name": "train-f64-4", "kind": "train", "frames": 4, "molecules": 64,
         "dtype": "float64"},
        # one domain of an MD engine, an odd size
        {"name": "engine-3993", "kind": "engine", "molecules": 1331},
        # the compressed embedding inside a torch program: forward and backward,
        # and, in FP64 on a small frame, the second derivative as well
        {"name": "tabulate-f32-12288", "kind": "tabulate", "atoms": 12288, "neighbors": 92,
         "dtype": "float32", "second": False},
        {"name": "tabulate-f64-192", "kind": "tabulate", "atoms": 192, "neighbors": 46,
         "dtype": "float64", "second": True},
        # the single operators, as a host program that keeps the reference's
        # operator sequence calls them
        {"name": "ops-f64-1536", "kind": "ops", "molecules": 512, "dtype": "float64"},
        {"name": "ops-f32-12288", "kind": "ops", "molecules": 4096, "dtype": "float32"},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["md", "md", "md", "batch", "plain", "train", "engine", "tabulate", "ops"])
    dtype = rng.choice(["float32", "float64"])
    if kind == "md":
        form = rng.choice(["host", "device", "skin"])
        return {"kind": kind, "molecules": size(27, 30000), "form": form}
    if kind == "batch":
        return {"kind": kind, "frames": size(4, 128), "atoms": size(300, 3000)}
    if kind == "plain":
        return {"kind": kind, "molecules": size(27, 4096)}
    if kind == "train":
        return {"kind": kind, "frames": size(1, 16 if dtype == "float32" else 8),
                "molecules": size(27, 125), "dtype": dtype}
    if kind == "engine":
        return {"kind": kind, "molecules": size(64, 8000)}
    if kind == "tabulate":
        return {"kind": kind, "atoms": size(64, 12288), "neighbors": rng.randint(20, 120),
                "dtype": dtype, "second": rng.random() < 0.5}
    return {"kind": kind, "molecules": size(27, 4096), "dtype": dtype}


# ----------------------------------------------------------------- inputs --
def _water(molecules, rng):
    """Liquid water: the O on a random subset of a grid of 3.104 A, every atom
    moved by a thermal N(0, 0.03 A). Returns (coord, atype, box edge)."""
    n = int(math.ceil(molecules ** (1 / 3) - 1e-9))
    edge = 3.1043 * n
    site = np.sort(rng.choice(n**3, molecules, replace=False))
    o = np.stack([site // (n * n), site // n % n, site % n], -1) * 3.104
    o = o + rng.uniform(-0.3, 0.3, o.shape)
    q = rng.normal(size=(molecules, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    a = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y + z * w), 2 * (x * z - y * w)], -1)
    b = np.stack([2 * (x * y - z * w), 1 - 2 * (x * x + z * z), 2 * (y * z + x * w)], -1)
    half = np.deg2rad(104.52) / 2
    s, c = 0.9572 * np.sin(half), 0.9572 * np.cos(half)
    coord = np.stack([o, o + s * a + c * b, o - s * a + c * b], 1).reshape(-1, 3)
    coord = coord + rng.normal(0.0, 0.03, coord.shape)
    return np.mod(coord, edge), np.tile(np.array([0, 1, 1], np.int32), molecules), edge


def _copper(atoms, rng):
    """FCC copper with vacancies, N(0, 0.05 A) around the sites."""
    k = max(2, int(math.ceil((atoms / 4) ** (1 / 3) - 1e-9)))
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    basis = np.array([[0, 0, 0], [0, 0.5, 0.5], [0.5, 0, 0.5], [0.5, 0.5, 0]])
    p = ((g + basis) * 3.615).reshape(-1, 3)
    p = p[np.sort(rng.choice(p.shape[0], atoms, replace=False))]
    p = p + rng.normal(0.0, 0.05, p.shape)
    return np.mod(p, 3.615 * k), np.full(atoms, 2, np.int32), 3.615 * k


def _frames(case, rng):
    """The batch: uneven frames from 24 to case["atoms"] atoms, water and
    copper in turn; the sizes are the case's, the positions the seed's."""
    sizes = np.random.default_rng([case["frames"], case["atoms"]])
    out = []
    for f in range(case["frames"]):
        n = int(math.exp(sizes.uniform(math.log(24), math.log(case["atoms"]))))
        out.append(_water(max(8, n // 3), rng) if f % 2 == 0 else _copper(max(24, n), rng))
    return out


def _box(edge):
    return np.diag([edge] * 3)


def _pairs(coord, atype, edge, centers, rc):
    """Neighbors of the first ``centers`` atoms within rc, for a cubic box
    (``edge`` >= rc) or an open system (None): center, neighbor and the
    vector between them, in FP64, sorted by center, neighbor type and distance,
    and the rank within (center, type)."""
    dev = coord.device
    shifts = torch.zeros((1, 3), dtype=torch.float64, device=dev)
    wrap = edge is not None and edge >= 2 * rc
    if edge is not None and not wrap:
        g = torch.tensor([-1.0, 0.0, 1.0], dtype=torch.float64, device=dev) * edge
        shifts = torch.cartesian_prod(g, g, g)
    n, ci, cj, cv = coord.shape[0], [], [], []
    c32 = coord.float()
    step = max(1, (1 << 26) // n)
    for s in shifts:
        for a in range(0, centers, step):
            b = min(centers, a + step)
            d2 = torch.zeros((b - a, n), device=dev)
            for k in range(3):
                d = c32[None, :, k] - c32[a:b, None, k] + s[k].float()
                if wrap:
                    d -= edge * torch.round(d / edge)
                d2 += d * d
            i, j = (d2 < (rc + 0.01) ** 2).nonzero(as_tuple=True)
            i = i + a
            v = coord[j] + s - coord[i]
            if wrap:
                v -= edge * torch.round(v / edge)
            keep = (v.square().sum(1) < rc * rc) & ((i != j) | bool(s.abs().sum() > 0))
            ci.append(i[keep])
            cj.append(j[keep])
            cv.append(v[keep])
    i, j, v = torch.cat(ci), torch.cat(cj), torch.cat(cv)
    nt = int(atype.max()) + 1
    o = torch.sort(v.square().sum(1).float(), stable=True)[1]
    o = o[torch.sort((i * nt + atype[j])[o], stable=True)[1]]
    i, j, v = i[o], j[o], v[o]
    key = i * nt + atype[j]
    count = torch.bincount(key, minlength=centers * nt)
    first = torch.cumsum(count, 0) - count
    return i, j, v, torch.arange(i.numel(), device=dev) - first[key]


def _slots(coord, atype, edge, centers, sel):
    """(vector [centers, nnei, 3], neighbor [centers, nnei] or -1) of every
    center's nearest neighbors of each type, in the model's slots."""
    dev = coord.device
    i, j, v, rank = _pairs(coord, atype, edge, centers, RCUT)
    cap = torch.tensor(sel, device=dev)
    off = torch.cumsum(cap, 0) - cap
    t = atype[j].long()
    keep = rank < cap[t]
    i, j, v, slot = i[keep], j[keep], v[keep], (off[t] + rank)[keep]
    nn = int(sum(sel))
    vec = torch.zeros((centers, nn, 3), dtype=torch.float64, device=dev)
    nbr = torch.full((centers, nn), -1, dtype=torch.long, device=dev)
    vec[i, slot], nbr[i, slot] = v, j
    return vec, nbr


def _env(vec, nbr):
    """Smooth environment rows (1, x/r, y/r, z/r) s(r) / r before
    normalisation; zero in empty slots."""
    on = nbr >= 0
    r2 = torch.where(on, vec.square().sum(-1), 1.0)
    r = r2.sqrt()
    u = (r - SMTH) / (RCUT - SMTH)
    sw = torch.where(r < SMTH, 1.0, u**3 * (-6 * u * u + 15 * u - 10) + 1) * on * (r < RCUT)
    return torch.cat([(sw / r)[..., None], vec * (sw / r2)[..., None]], -1)


def _dev(frame):
    coord, atype, edge = frame
    return (torch.tensor(coord, dtype=torch.float64, device="cuda"),
            torch.tensor(atype, device="cuda"), edge)


def _model(seed, sel):
    """Seeded weights, N(0, 1 / fan_in) and N(0, 1) biases, and the statistics
    of a 64-molecule box (and a copper box for the third species): what a
    trained model file holds, in numpy."""
    rng = np.random.default_rng([7, seed])

    def layer(n_in, n_out):
        return rng.normal(0, n_in**-0.5, (n_in, n_out)), rng.normal(0, 1, n_out)

    emb = [[layer(a, b) for a, b in zip((1,) + NEURON, NEURON)] for _ in sel]
    fit = []
    for _ in sel:
        ls = [layer(a, b) for a, b in zip((NEURON[-1] * AXIS,) + FITTING, FITTING)]
        fit.append({"layers": [(W, b, rng.normal(0.1, 0.001, len(b)) if W.shape[0] == len(b)
                                else None) for W, b in ls], "out": layer(FITTING[-1], 1)})
    frames = [_water(64, rng)] + ([_copper(100, rng)] if len(sel) > 2 else [])
    nn = int(sum(sel))
    avg, std, near = np.zeros((len(sel), nn, 4)), np.ones((len(sel), nn, 4)), RCUT
    for f in frames:
        c, t, edge = _dev(f)
        vec, nbr = _slots(c, t, edge, c.shape[0], sel)
        near = min(near, float(vec.square().sum(-1)[nbr >= 0].min().sqrt()))
        e = _env(vec, nbr)
        for ty in sorted(set(f[1].tolist())):
            x = e[t == ty]
            avg[ty, :, 0] = float(x[..., 0].mean())
            std[ty, :, 0] = max(1e-2, float(x[..., 0].std(unbiased=False)))
            std[ty, :, 1:] = max(1e-2, float(x[..., 1:].square().mean()
                                             - x[..., 1:].mean() ** 2) ** 0.5)
    return {"sel": sel, "emb": emb, "fit": fit, "avg": avg, "std": std, "near": near}


def _params(m, tables):
    """The model as this package takes it."""
    workload, table = _package("workload"), _package("table")
    cfg = workload.SeAConfig(rcut=RCUT, rcut_smth=SMTH, sel=m["sel"], neuron=NEURON,
                             axis_neuron=AXIS, fitting=FITTING)
    p = workload.SeAParams(cfg=cfg, emb=m["emb"], fit=m["fit"],
                           bias_atom_e=np.zeros(len(m["sel"])),
                           davg=m["avg"].reshape(len(m["sel"]), -1),
                           dstd=m["std"].reshape(len(m["sel"]), -1))
    if tables:
        p.tables = [(t.cpu().numpy(), info) for t, info in table.build_tables_device(
            p.emb, p.davg, p.dstd, cfg.sel, m["near"], SMTH, RCUT)]
    return p


def _sel(case):
    return (46, 92, 60) if case["kind"] == "batch" else (46, 92)


def _frame(case, seed):
    return _water(case["molecules"], np.random.default_rng([1, seed]))


def _train_inputs(case, seed):
    """Frames of a training batch and their labels."""
    rng = np.random.default_rng([2, seed])
    frames = [_water(case["molecules"], rng) for _ in range(case["frames"])]
    n = sum(f[1].size for f in frames)
    return frames, (rng.normal(0, 10, len(frames)), rng.normal(0, 1, (n, 3)),
                    rng.normal(0, 10, (len(frames), 9)))


def _extended(case, seed):
    """An engine's system: the box's atoms, then the periodic images within
    rcut + skin of the box."""
    c, t, edge = _dev(_frame(case, seed))
    g = torch.tensor([-1.0, 0.0, 1.0], dtype=torch.float64, device="cuda") * edge
    coords, types = [c], [t]
    for s in torch.cartesian_prod(g, g, g):
        if bool(s.abs().sum() > 0):
            x = c + s
            keep = ((x > -(RCUT + SKIN)) & (x < edge + RCUT + SKIN)).all(1)
            coords.append(x[keep])
            types.append(t[keep])
    return torch.cat(coords), torch.cat(types), c.shape[0]


def _tab_inputs(case, seed):
    """Environment rows of one neighbor type as the table op gets them:
    neighbors uniform in the cutoff sphere (0.9 A to 6 A), nearest first, the
    last slots empty, normalised; and cotangents. FP64."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n, k = case["atoms"], case["neighbors"]

    def rand(*shape):
        return torch.rand(shape, generator=g, dtype=torch.float64, device="cuda")

    r = (0.9**3 + rand(n, k) * (RCUT**3 - 0.9**3)) ** (1 / 3)
    d = rand(n, k, 3) - 0.5
    vec = r.sort(1)[0][..., None] * d / d.norm(dim=-1, keepdim=True)
    full = (k * (0.6 + 0.4 * rand(n, 1))).long()
    nbr = torch.where(torch.arange(k, device="cuda") < full, 1, -1)
    e = _env(vec, nbr)
    avg, std = 0.06, 0.11
    em = torch.cat([(e[..., :1] - avg) / std, e[..., 1:] / std], -1)
    em = em.to(getattr(torch, case["dtype"])).double()

    def cot(*shape):
        return (rand(*shape) - 0.5).to(getattr(torch, case["dtype"])).double()

    return em, cot(n, 4, NEURON[-1]), cot(n, k), cot(n, k, 4), avg, std


# ---------------------------------------------------------------- prepare --
def prepare(case, seed):
    return {"md": _prepare_md, "batch": _prepare_batch, "plain": _prepare_plain,
            "train": _prepare_train, "engine": _prepare_engine, "tabulate": _prepare_tabulate,
            "ops": _prepare_ops}[case["kind"]](case, seed)


def _prepare_md(case, seed):
    coord, atype, edge = _frame(case, seed)
    ev = _package("model").SeAEvaluator(_params(_model(seed, _sel(case)), True), atype,
                                        _box(edge), skin=SKIN if case["form"] == "skin" else 0.0)
    ev.coord.copy_(torch.as_tensor(coord))
    ev.capture()
    host = torch.as_tensor(coord).pin_memory() if case["form"] == "host" else None
    return {"kind": "md", "form": case["form"], "ev": ev, "host": host,
            "buffer": torch.empty(ev.results.numel(), dtype=torch.float64).pin_memory()
            if host is not None else None, "coord": torch.as_tensor(coord, device="cuda")}


def _prepare_batch(case, seed):
    frames = _frames(case, np.random.default_rng([3, seed]))
    ev = _package("batch").BatchEvaluator(_params(_model(seed, _sel(case)), True),
                                          [(c, t, _box(L)) for c, t, L in frames])
    ev.capture()
    coord = torch.as_tensor(np.concatenate([f[0] for f in frames]), device="cuda")
    return {"kind": "batch", "ev": ev, "coord": coord}


def _prepare_plain(case, seed):
    coord, atype, edge = _frame(case, seed)
    ev = _package("model").SeAEvaluator(_params(_model(seed, _sel(case)), False), atype,
                                        _box(edge), mode="plain")
    ev.coord.copy_(torch.as_tensor(coord))
    ev.capture()
    return {"kind": "plain", "ev": ev, "coord": torch.as_tensor(coord, device="cuda")}


def _prepare_train(case, seed):
    train = _package("train")
    frames, labels = _train_inputs(case, seed)
    loss = train.EnergyStdLoss(LR, PREFS[0], PREFS[0], PREFS[1], PREFS[1], PREFS[2], PREFS[2])
    tr = train.SeATrainer(_params(_model(seed, _sel(case)), False),
                          [(c, t, _box(L)) for c, t, L in frames],
                          dtype=getattr(torch, case["dtype"]), loss=loss)
    tr.set_labels(*labels)
    tr.capture()
    return {"kind": "train", "tr": tr}


def _prepare_engine(case, seed):
    coord, atype, nloc = _extended(case, seed)
    i, j, _, _ = _pairs(coord, torch.zeros_like(atype), None, nloc, RCUT + SKIN)
    num = torch.bincount(i, minlength=nloc)
    width = int(num.max())
    rows = torch.full((nloc, width), -1, dtype=torch.int32, device="cuda")
    first = torch.cumsum(num, 0) - num
    rows[i, torch.arange(i.numel(), device="cuda") - first[i]] = j.int()
    fl = _package("engine").ForwardLower(_params(_model(seed, _sel(case)), True), nloc,
                                         coord.shape[0], max(512, width))
    ptrs = rows.data_ptr() + torch.arange(nloc, device="cuda") * (4 * width)
    atype = atype.int()
    fl(coord, atype, nloc, num.int(), ptrs, rebuilt=True)  # the engine has just re-neighbored
    return {"kind": "engine", "fl": fl, "rows": rows,
            "args": (coord, atype, nloc, num.int(), ptrs)}


def _prepare_tabulate(case, seed):
    table = _package("table")
    _package("ops")
    em, dy, gx, ge, avg, std = _tab_inputs(case, seed)
    dt = getattr(torch, case["dtype"])
    stat = np.tile(np.array([avg, 0, 0, 0.0]), (1, case["neighbors"]))
    dstd = np.full((1, 4 * case["neighbors"]), std)
    tab, info = table.build_tables_device(_model(seed, (46, 92))["emb"][:1], stat, dstd,
                                          (case["neighbors"],), 0.9, SMTH, RCUT)[0]
    em = em.to(dt)
    return {"kind": "tabulate", "second": case["second"], "table": tab.to(dt),
            "info": torch.as_tensor(info, dtype=dt), "em": em,
            "em_x": em[..., 0].contiguous(),
            "dy": dy.to(dt), "gx": gx.to(dt), "ge": ge.to(dt)}


def _prepare_ops(case, seed):
    m = _model(seed, _sel(case))
    coord, atype, edge = _dev(_frame(case, seed))
    dt = getattr(torch, case["dtype"])
    nn = int(sum(m["sel"]))
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    nd = torch.randn((coord.shape[0], nn * 4), generator=g, dtype=torch.float64, device="cuda")

    def stat(a):
        return torch.as_tensor(a.reshape(2, -1), dtype=dt, device="cuda")

    return {"kind": "ops", "coord": coord.to(dt), "atype": atype, "box": _box(edge).reshape(9),
            "avg": stat(m["avg"]), "std": stat(m["std"]), "nd": nd.to(dt),
            "sec": np.array([0, 46, 138], np.int32)}


# -------------------------------------------------------------------- run --
def run(s):
    kind = s["kind"]
    if kind == "md" and s["form"] == "host":
        e, f, v = s["ev"].compute(s["host"], s["buffer"])
        return {"energy": np.float32([e]), "force": f.astype(np.float32),
                "virial": v.astype(np.float32)}
    if kind in ("md", "batch", "plain"):
        ev = s["ev"]
        ev.coord.copy_(s["coord"])
        ev.replay()
        dt = torch.float64 if kind == "plain" else torch.float32
        return {"energy": ev.energy.to(dt), "force": ev.force.to(dt), "virial": ev.virial.to(dt)}
    if kind == "train":
        s["tr"].train_step(LR)
        return {"grads": s["tr"].named_grads(), "flat": s["tr"].flat.detach()}
    if kind == "engine":
        e, f, v = s["fl"](*s["args"])
        return {"energy": e.float(), "force": f.float(), "virial": v.float()}
    if kind == "tabulate":
        return _run_tabulate(s)
    return _run_ops(s)


def _run_tabulate(s):
    op = torch.ops.deepmd
    em, em_x, dy = s["em"].requires_grad_(), s["em_x"].requires_grad_(), s["dy"]
    out = op.tabulate_fusion_se_a(s["table"], s["info"], em_x, em, NEURON[-1])[0]
    if not s["second"]:
        dx, de = torch.autograd.grad(out, (em_x, em), dy)
        return {"out": out.detach(), "dx": dx, "de": de}
    dy = dy.requires_grad_()
    dx, de = torch.autograd.grad(out, (em_x, em), dy, create_graph=True)
    dz, = torch.autograd.grad((dx, de), dy, (s["gx"], s["ge"]))
    return {"out": out.detach(), "dx": dx.detach(), "de": de.detach(), "dz": dz}


def _run_ops(s):
    ops = _package("ops")
    c, t, owner = ops.copy_coord(s["coord"], s["atype"], RCUT, s["box"])
    nloc, nall = s["atype"].numel(), t.numel()
    il, num, rows, _ = ops.build_nlist(c, nloc, RCUT, t)
    em, emd, rij, nl = ops.prod_env_mat_a(c, t, il, num, rows, s["avg"], s["std"], nloc, RCUT,
                                          SMTH, s["sec"])
    force = ops.prod_force_a(s["nd"], emd, nl, nloc, nall)
    virial, atom = ops.prod_virial_a(s["nd"], emd, rij, nl, nloc, nall)
    owner = owner.long()  # the ghosts' shares go to the atoms they are images of
    force = torch.zeros_like(s["coord"]).index_add_(0, owner, force[0])
    atom = force.new_zeros((nloc, 9)).index_add_(0, owner, atom)
    return {"em": em, "em_deriv": emd, "rij": rij, "nlist": nl, "force": force,
            "virial": virial, "atom_virial": atom}


# ------------------------------------------------------------------- work --
def work(case):
    """Bytes of inputs and results, and operations of the model's formulas (a
    table row costs its polynomial, a network layer its products)."""
    kind, M = case["kind"], NEURON[-1]
    fit = sum(a * b for a, b in zip((M * AXIS,) + FITTING, FITTING))
    emb = sum(a * b for a, b in zip((1,) + NEURON, NEURON))
    weights = 2 * (fit + emb)
    if kind == "tabulate":
        n, k = case["atoms"], case["neighbors"]
        b = 4 if case["dtype"] == "float32" else 8
        passes = 3 if case["second"] else 2
        return {"bytes": b * (n * (10 * k + 8 * M) + (n * (5 * k + 4 * M) if passes == 3 else 0)),
                "flops": 2.0 * n * k * M * (14 + 18 + (18 if passes == 3 else 0))}
    if kind == "batch":
        mean = (case["atoms"] - 24) / math.log(case["atoms"] / 24)  # log-uniform sizes
        n, w = case["frames"] * mean, 1.5
    else:
        n, w = 3 * case["molecules"] * case.get("frames", 1), 1.0
    near = 90.0  # neighbors within the cutoff at this density
    if kind == "ops":
        b = 4 if case["dtype"] == "float32" else 8
        return {"bytes": n * (b * 138 * (4 + 12 + 3 + 4) + 4 * 138 + b * 3 * 6 * 3),
                "flops": n * near * 150.0}
    desc = near * M * (7 + 15) + 3 * 4 * M * AXIS
    if kind in ("md", "engine"):
        desc_b = 24 + 24 + 8 * (2 * 138 if case.get("form") == "skin" or kind == "engine" else 0)
        return {"bytes": n * desc_b + 4 * weights, "flops": n * 2.0 * (desc + 2 * fit)}
    if kind == "batch":
        return {"bytes": n * 48 + 4 * w * weights, "flops": n * 2.0 * (desc + 2 * fit)}
    if kind == "plain":
        return {"bytes": n * 48 + 8 * weights, "flops": n * 2.0 * (near * 3 * emb + 2 * fit)}
    b = 4 if case["dtype"] == "float32" else 8  # train
    return {"bytes": n * 72 + 6 * b * weights, "flops": n * 2.0 * (near * 9 * emb + 8 * fit)}


# ------------------------------------------------------------------ exact --
def _t(a, grad=False):
    return torch.tensor(np.asarray(a), dtype=torch.float64, device="cuda", requires_grad=grad)


def _weights(m, grad=False):
    """The model's networks as FP64 tensors: embedding [(W, b)] and fitting
    ([(W, b, idt)], (W, b)) per type."""
    emb = [[(_t(W, grad), _t(b, grad)) for W, b in net] for net in m["emb"]]
    fit = [([(_t(W, grad), _t(b, grad), None if d is None else _t(d, grad))
             for W, b, d in f["layers"]], (_t(f["out"][0], grad), _t(f["out"][1], grad)))
           for f in m["fit"]]
    return emb, fit


def _embed(net, x):
    for W, b in net:
        y = torch.tanh(x @ W + b)
        x = y + x if W.shape[0] == W.shape[1] else \
            y + torch.cat([x, x], -1) if W.shape[1] == 2 * W.shape[0] else y
    return x


def _energies(m, nets, em, t):
    """Atomic energies of centers of types ``t`` from normalised rows."""
    emb, fit = nets
    off, xyz = 0, 0.0
    for ty, k in enumerate(m["sel"]):
        e = em[:, off:off + k]
        xyz = xyz + e.transpose(1, 2) @ _embed(emb[ty], e[..., :1])
        off += k
    xyz = xyz / off
    D = (xyz.transpose(1, 2) @ xyz[:, :, :AXIS]).reshape(em.shape[0], -1)
    out = torch.zeros(em.shape[0], dtype=torch.float64, device="cuda")
    for ty, (layers, (Wo, bo)) in enumerate(fit):
        at = (t == ty).nonzero().view(-1)
        if at.numel():
            h = D[at]
            for W, b, d in layers:
                y = torch.tanh(h @ W + b)
                h = y if d is None else h + d * y
            out = out.index_add(0, at, (h @ Wo + bo).view(-1))
    return out


def _efv(m, nets, coord, atype, edge, centers, graph=False):
    """(energy, force on every atom, virial) in FP64."""
    vec, nbr = _slots(coord, atype, edge, centers, m["sel"])
    avg, std = _t(m["avg"]), _t(m["std"])
    step = centers if graph else 2048
    energy, force, virial = 0.0, torch.zeros_like(coord), 0.0
    for a in range(0, centers, step):
        b = min(centers, a + step)
        v = vec[a:b].clone().requires_grad_()
        t = atype[a:b].long()
        e = _energies(m, nets, (_env(v, nbr[a:b]) - avg[t]) / std[t], t).sum()
        q = -torch.autograd.grad(e, v, create_graph=graph)[0]
        on = nbr[a:b] >= 0
        q = q * on[..., None]
        force = force.index_add(0, nbr[a:b][on], q[on])
        force = force.index_add(0, torch.arange(a, b, device="cuda"), -q.sum(1))
        energy = energy + (e if graph else e.detach())
        virial = virial + torch.einsum("ijd,ije->de", q, v).reshape(9)
    return energy, force, virial


def exact(case, seed):
    kind = case["kind"]
    if kind == "tabulate":
        return _exact_tabulate(case, seed)
    if kind == "ops":
        return _exact_ops(case, seed)
    m = _model(seed, _sel(case))
    if kind == "train":
        return _exact_train(case, seed, m)
    nets = _weights(m)
    if kind == "engine":
        coord, atype, nloc = _extended(case, seed)
        e, f, v = _efv(m, nets, coord, atype, None, nloc)
        return {"energy": e.view(1), "force": f, "virial": v}
    if kind == "batch":
        frames = _frames(case, np.random.default_rng([3, seed]))
        r = [_efv(m, nets, *_dev(f), f[1].size) for f in frames]
        return {"energy": torch.stack([x[0] for x in r]), "force": torch.cat([x[1] for x in r]),
                "virial": torch.stack([x[2] for x in r])}
    frame = _frame(case, seed)
    e, f, v = _efv(m, nets, *_dev(frame), frame[1].size)
    return {"energy": e.view(1), "force": f, "virial": v}


def _exact_train(case, seed, m):
    emb, fit = nets = _weights(m, True)
    frames, (Eh, Fh, Vh) = _train_inputs(case, seed)
    names, ws = [], []
    for t, net in enumerate(emb):
        for k, pair in enumerate(net):
            key = f"atomic_model.descriptor.sea.filter_layers.networks.{t}.layers.{k}"
            names += [key + ".matrix", key + ".bias"]
            ws += list(pair)
    for t, (layers, out) in enumerate(fit):
        for k, tensors in enumerate(layers + [out]):
            key = f"atomic_model.fitting_net.filter_layers.networks.{t}.layers.{k}"
            for part, w in zip((".matrix", ".bias", ".idt"), tensors):
                if w is not None:
                    names.append(key + part)
                    ws.append(w)
    total = [torch.zeros_like(w) for w in ws]
    nf, na, at = len(frames), sum(f[1].size for f in frames), 0
    for k, f in enumerate(frames):
        n = f[1].size
        e, force, v = _efv(m, nets, *_dev(f), n, graph=True)
        loss = (PREFS[0] * (e - Eh[k]) ** 2 / n / nf
                + PREFS[1] * (force - _t(Fh[at:at + n])).square().sum() / (3 * na)
                + PREFS[2] * (v - _t(Vh[k])).square().mean() / n / nf)
        at += n
        for g, d in zip(total, torch.autograd.grad(loss, ws)):
            g += d
    # the first Adam step; every tensor starts at a multiple of 4 elements
    flat = []
    for w, g in zip(ws, total):
        new = (w.detach() - LR * g / (g.abs() + 1e-8)).reshape(-1)
        flat.append(torch.nn.functional.pad(new, (0, -new.numel() % 4)))
    return {"grads": dict(zip(names, total)), "flat": torch.cat(flat)}


def _fold(e, g):
    """The op's gradient of a row's empty slots, which are alike: their sum at
    the first of them, zero at the others (source/lib/src/tabulate.cc:178-204)."""
    empty = (e.detach()[..., 1:] == 0).all(-1)
    empty = empty if g.dim() == 2 else empty[..., None]
    first = empty & (torch.cumsum(empty, 1) == 1)
    return torch.where(empty, first * (g * empty).sum(1, keepdim=True), g)


def _exact_tabulate(case, seed):
    em, dy, gx, ge, _, _ = _tab_inputs(case, seed)
    net = _weights(_model(seed, (46, 92)))[0][0]
    dy = dy.requires_grad_()
    parts = []
    for a in range(0, em.shape[0], 1024):
        s = slice(a, a + 1024)
        x = em[s, :, 0].clone().requires_grad_()
        e = em[s].clone().requires_grad_()
        out = e.transpose(1, 2) @ _embed(net, x[..., None])
        dx, de = torch.autograd.grad(out, (x, e), dy[s], create_graph=case["second"])
        dx, de = _fold(e, dx), _fold(e, de)
        r = [out, dx, de]
        if case["second"]:
            r.append(torch.autograd.grad((dx, de), dy, (gx[s], ge[s]))[0][s])
        parts.append([v.detach() for v in r])
    return dict(zip(("out", "dx", "de", "dz"), (torch.cat(p) for p in zip(*parts))))


def _exact_ops(case, seed):
    m = _model(seed, _sel(case))
    s = _prepare_ops(case, seed)
    coord, atype, edge = s["coord"].double(), s["atype"], float(s["box"][0])
    n = coord.shape[0]
    vec, nbr = _slots(coord, atype, edge, n, m["sel"])
    t = atype.long()
    std = _t(m["std"])[t]
    v = vec.clone().requires_grad_()
    em = (_env(v, nbr) - _t(m["avg"])[t]) / std
    deriv = torch.stack([-torch.autograd.grad(em[..., a].sum(), v, retain_graph=a < 3)[0]
                         for a in range(4)], 2)
    deriv = deriv * (nbr >= 0)[..., None, None]
    q = torch.einsum("ija,ijad->ijd", s["nd"].double().view(n, -1, 4), deriv)
    on = nbr >= 0
    w = torch.einsum("ijd,ije->ijde", q, vec).reshape(n, -1, 9)
    force = torch.zeros_like(coord).index_add_(0, nbr[on], q[on]) - q.sum(1)
    return {"em": em.detach().reshape(n, -1), "em_deriv": deriv.reshape(n, -1),
            "rij": vec.reshape(n, -1), "nlist": None, "force": force,
            "virial": w.sum((0, 1)),
            "atom_virial": coord.new_zeros((n, 9)).index_add_(0, nbr[on], w[on])}
