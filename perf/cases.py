"""The work a program has this library do, as measurable cases.

Every case goes through the package's public entry points (Solver, LearnedNet,
kernel_dbcg_simple) the way the reference's driver, the learned workload and
the benchmark call them:

  step    one implicit theta step: element build, right-hand side, solve
  loop    several steps on the device (vdr_time_steps) with the mass integral
  block   K right-hand sides with one operator
  meshes  many independent meshes in one handle: build, right-hand side,
          segmented solve
  net     the learned preconditioner's network: forward pass, or loss and
          parameter gradients of one training step
  dropin  the reference's own host-array solve call, Jacobi BiCG

Inputs are made on the GPU from the seed; `exact` evaluates the same
quantities in 64 bits with plain torch.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import __graft_entry__ as _entry  # noqa: E402

vdr = _entry.package()
P = vdr.problems
DEV = "cuda"
F64 = torch.float64
COURANT = 10.0
GAUSS = 0.577350269189626
# local node signs of the reference cube
SX = (-1, 1, 1, -1, -1, 1, 1, -1)
SY = (-1, -1, 1, 1, -1, -1, 1, 1)
SZ = (-1, -1, -1, -1, 1, 1, 1, 1)


# ------------------------------------------------------------------- cases
# Every solve runs to 1e-10, as the small plain-method configuration does: the
# answers of two runs, whose sums are added in different orders, then agree to
# about that.
def listed():
    return [
        # the reference's recorded run: 7 x 20 x 20 nodes on stretched axes,
        # wind across, Robin ground, 20 implicit steps from a clean field
        {"name": "loop_recorded_6x19x19", "kind": "loop", "nex": 6, "ney": 19, "nez": 19,
         "flow": "channel", "variant": "vf", "steps": 20, "precision": "fp64", "tol": 1e-10},
        # a small steady solve (parameter studies)
        {"name": "step_steady_32x32x16", "kind": "step", "nex": 32, "ney": 32, "nez": 16,
         "flow": "constant", "variant": "ot", "precision": "fp64", "warm": False, "tol": 1e-10},
        # an ordinary ragged mesh, one step of a running field
        {"name": "step_67x45x31", "kind": "step", "nex": 67, "ney": 45, "nez": 31,
         "flow": "rotation", "variant": "vf", "precision": "fp64", "warm": True, "tol": 1e-10},
        # the mid-size grid of the batched and learned workloads
        {"name": "step_128x128x64", "kind": "step", "nex": 128, "ney": 128, "nez": 64,
         "flow": "rotation", "variant": "vf", "precision": "fp64", "warm": True, "tol": 1e-10},
        # the largest grid: the benchmark's step, from a clean field
        {"name": "step_256x256x128", "kind": "step", "nex": 256, "ney": 256, "nez": 128,
         "flow": "rotation", "variant": "vf", "precision": "fp64", "warm": False, "tol": 1e-10},
        # mixed precision, one step of a running field
        {"name": "step_mixed_97x83x61", "kind": "step", "nex": 97, "ney": 83, "nez": 61,
         "flow": "rotation", "variant": "vf", "precision": "mixed", "warm": True, "tol": 1e-10},
        # mixed precision, a large transient run on the device
        {"name": "loop_mixed_192x192x96", "kind": "loop", "nex": 192, "ney": 192, "nez": 96,
         "flow": "rotation", "variant": "vf", "steps": 3, "precision": "mixed", "tol": 1e-10},
        # 64 sources with one operator
        {"name": "block64_128x128x64", "kind": "block", "nex": 128, "ney": 128, "nez": 64,
         "K": 64, "tol": 1e-10},
        # many uneven meshes at once
        {"name": "meshes96_8to32", "kind": "meshes", "nmesh": 96, "nmin": 8, "nmax": 32,
         "tol": 1e-10},
        # the learned preconditioner's network on its workload's grid
        {"name": "net_forward_128x128x64", "kind": "net", "nex": 128, "ney": 128, "nez": 64,
         "train": False},
        # one training step's loss and gradients
        {"name": "net_train_64x64x32", "kind": "net", "nex": 64, "ney": 64, "nez": 32,
         "train": True},
        # the reference's solve call with host arrays
        {"name": "dropin_bicg_40x36x28", "kind": "dropin", "nex": 40, "ney": 36, "nez": 28,
         "tol": 1e-10},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _dims(rng, lo, hi):
    """Element counts per axis with about a log-uniform product."""
    n = _log_uniform(rng, lo, hi) ** (1.0 / 3.0)
    a, b = _log_uniform(rng, 0.6, 1.6), _log_uniform(rng, 0.6, 1.6)
    return (max(3, round(n * a)), max(3, round(n * b)), max(3, round(n / (a * b))))


def draw(rng):
    kind = rng.choice(["step"] * 5 + ["loop"] * 3 + ["block", "block", "meshes", "net", "net",
                                                     "dropin"])
    if kind == "step":
        flow = rng.choice(["rotation"] * 3 + ["constant"])
        nx, ny, nz = _dims(rng, 300, 3.0e6 if flow == "rotation" else 3.0e4)
        prec = rng.choice(["fp64", "fp64", "mixed"]) if flow == "rotation" else "fp64"
        return {"kind": "step", "nex": nx, "ney": ny, "nez": nz, "flow": flow,
                "variant": "vf" if flow == "rotation" else rng.choice(["ot", "gp"]),
                "precision": prec, "warm": flow == "rotation" and rng.random() < 0.6,
                "tol": 1e-10}
    if kind == "loop":
        prec = rng.choice(["fp64", "mixed"])
        flow = rng.choice(["channel", "rotation"]) if prec == "fp64" else "rotation"
        nx, ny, nz = _dims(rng, 300, 6.0e5)
        if flow == "channel":
            nx, ny, nz = rng.randint(4, 9), rng.randint(13, 25), rng.randint(13, 25)
        return {"kind": "loop", "nex": nx, "ney": ny, "nez": nz, "flow": flow, "variant": "vf",
                "steps": rng.randint(2, 12 if flow == "channel" else 5), "precision": prec,
                "tol": 1e-10}
    if kind == "block":
        K = rng.choice([16, 32, 64])
        nx, ny, nz = _dims(rng, 1000, 4.0e7 / K)
        return {"kind": "block", "nex": nx, "ney": ny, "nez": nz, "K": K, "tol": 1e-10}
    if kind == "meshes":
        lo = rng.randint(4, 12)
        return {"kind": "meshes", "nmesh": rng.randint(8, 96), "nmin": lo,
                "nmax": lo + rng.randint(2, 20), "tol": 1e-10}
    if kind == "net":
        train = rng.random() < 0.5
        nx, ny, nz = _dims(rng, 8000, 1.5e5 if train else 1.0e6)
        return {"kind": "net", "nex": nx, "ney": ny, "nez": nz, "train": train}
    nx, ny, nz = _dims(rng, 300, 5.0e4)
    return {"kind": "dropin", "nex": nx, "ney": ny, "nez": nz, "tol": 1e-10}


# ------------------------------------------------------------------ inputs
def _axis(n, length, power):
    """n + 1 coordinates on [-length, length], denser in the middle."""
    t = torch.linspace(-1.0, 1.0, n + 1, dtype=F64, device=DEV)
    return length * t.sign() * t.abs() ** power


def _grid(nex, ney, nez):
    """Zero-based connectivity [8, E], element indices (i, j, k)."""
    nax, pl = nex + 1, (nex + 1) * (ney + 1)
    k, j, i = torch.meshgrid(*(torch.arange(n, device=DEV) for n in (nez, ney, nex)),
                             indexing="ij")
    i, j, k = i.reshape(-1), j.reshape(-1), k.reshape(-1)
    base = i + nax * j + pl * k
    off = torch.tensor([0, 1, 1 + nax, nax, pl, 1 + pl, 1 + pl + nax, pl + nax], device=DEV)
    return base[None, :] + off[:, None], (i, j, k)


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, dtype=F64, device=DEV)


def _blobs(g, x, y, z, count):
    """`count` Gaussian blobs, centres in [0.2, 0.8]^3, sigma in [0.05, 0.1]."""
    out = torch.zeros_like(x)
    for c in _uniform(g, count, 4).cpu().tolist():
        s = 0.05 + 0.05 * c[3]
        out += torch.exp(-((x - 0.2 - 0.6 * c[0]) ** 2 + (y - 0.2 - 0.6 * c[1]) ** 2
                           + (z - 0.2 - 0.6 * c[2]) ** 2) / (2 * s * s))
    return out


def _inflow(nod, ijk, n, vel, N):
    """Nodes of the boundary faces whose element velocity points inwards."""
    bc = torch.zeros(N, dtype=torch.int32, device=DEV)
    faces = ((0, (0, 3, 4, 7), (1, 2, 5, 6)), (1, (0, 1, 4, 5), (2, 3, 6, 7)),
             (2, (0, 1, 2, 3), (4, 5, 6, 7)))
    for d, low, high in faces:
        for side, sign, loc in ((0, 1, low), (n[d] - 1, -1, high)):
            sel = (ijk[d] == side) & (sign * vel[d] > 0)
            for a in loc:
                bc[nod[a][sel]] = 1
    return bc


def _system(flow, nex, ney, nez, seed):
    """Mesh, fields, mask and a running field on the GPU, all from the seed."""
    g = torch.Generator(device=DEV).manual_seed(int(seed) * 2654435761 % (1 << 62) + 1)
    nod, ijk = _grid(nex, ney, nez)
    E, N = nod.shape[1], (nex + 1) * (ney + 1) * (nez + 1)
    if flow == "channel":  # stretched axes, metres; ground at x = 0
        ax = (torch.linspace(0.0, 1.0, nex + 1, dtype=F64, device=DEV) ** 1.8 * 420.0,
              _axis(ney, 4000.0, 2.4), _axis(nez, 4000.0, 2.4))
    else:
        ax = tuple(torch.linspace(0.0, 1.0, n + 1, dtype=F64, device=DEV)
                   for n in (nex, ney, nez))
    zz, yy, xx = (t.reshape(-1).clone() for t in torch.meshgrid(ax[2], ax[1], ax[0],
                                                                indexing="ij"))
    if flow != "channel":  # interior coordinates moved by up to a tenth of a cell
        for c, n in ((xx, nex), (yy, ney), (zz, nez)):
            d = (2.0 * _uniform(g, N) - 1.0) * (0.1 / n)
            c += torch.where((c > 0.25 / n) & (c < 1.0 - 0.25 / n), d, torch.zeros_like(d))
    cx, cy, cz = (c[nod].mean(0) for c in (xx, yy, zz))
    kod = torch.zeros((6, E), dtype=torch.int32, device=DEV)
    for f, sel in ((1, ijk[2] == 0), (2, ijk[2] == nez - 1), (3, ijk[0] == 0),
                   (4, ijk[0] == nex - 1), (5, ijk[1] == ney - 1), (6, ijk[1] == 0)):
        kod[f - 1][sel] = f
    pdec, alpha = torch.zeros(E, dtype=F64, device=DEV), 0.0
    u = _uniform(g, 6).cpu().tolist()
    if flow == "channel":
        # uniform wind and exchange, one emitting element, face-code mask
        speed, turn = 4.0 + 2.0 * u[0], 0.2 * (u[1] - 0.5)
        vel = torch.tensor([[0.0], [-speed * math.cos(turn)], [speed * math.sin(turn)]],
                           dtype=F64, device=DEV).expand(3, E).contiguous()
        lam = torch.full((E,), 30.0 + 20.0 * u[2], dtype=F64, device=DEV)
        pdec += 0.0007
        alpha = 0.01
        q = torch.zeros(E, dtype=F64, device=DEV)
        src = ((nez // 2 * ney) + ney // 2) * nex + min(nex - 1, int(3 * u[3]))
        q[src] = 0.5 + u[4]
        bc = torch.zeros(N, dtype=torch.int32, device=DEV)
        for f, loc in ((1, (0, 1, 2, 3)), (2, (4, 5, 6, 7)), (4, (1, 2, 6, 5)),
                       (5, (3, 2, 6, 7)), (6, (0, 1, 5, 4))):
            for a in loc:
                bc[nod[a][kod[f - 1] == f]] = 1
        told = torch.zeros(N, dtype=F64, device=DEV)
    else:
        if flow == "constant":
            v = torch.tensor([1.0, 0.4 + 0.2 * u[0], 0.2 + 0.1 * u[1]], dtype=F64, device=DEV)
            vel = (v / v.norm())[:, None].expand(3, E).contiguous()
            lam = torch.full((E,), 1e-3, dtype=F64, device=DEV)
        else:  # solid-body rotation with shear, lognormal diffusivity
            vel = torch.stack([-(cy - 0.45 - 0.1 * u[0]) + (0.2 + 0.2 * u[2]) * cz,
                               cx - 0.45 - 0.1 * u[1], torch.zeros_like(cx)])
            vel /= vel.square().sum(0).sqrt().max()
            lam = torch.exp(math.log(1e-4)
                            + torch.randn(E, generator=g, dtype=F64, device=DEV))
        q = _blobs(g, cx, cy, cz, 2) / E
        bc = _inflow(nod, ijk, (nex, ney, nez), vel, N)
        told = _blobs(g, xx, yy, zz, 3) * (bc == 0)
    return dict(dims=(nex, ney, nez), nod=nod, kod=kod, xyz=(xx, yy, zz), vel=vel, lam=lam,
                pdec=pdec, q=q, bc=bc, alpha=alpha, told=told, gen=g)


def _host(t):
    return t.reshape(-1).cpu().numpy()


def _problem(S, variant, tol):
    nax, nay, naz = (n + 1 for n in S["dims"])
    mesh = P.Mesh(nax, nay, naz, *(_host(c) for c in S["xyz"]),
                  _host((S["nod"] + 1).to(torch.int32)), _host(S["kod"]))
    return P.Problem("case", mesh, _host(S["vel"]), _host(S["lam"]), _host(S["pdec"]),
                     _host(S["q"]), _host(S["bc"]), S["alpha"],
                     {"ot": P.DR_OT, "gp": P.DR_GP, "vf": P.DR_VF}[variant], tol)


def _coefficients(case):
    """(aH, aM, cf, rM) of the theta scheme, or of the steady problem."""
    if case.get("flow") == "constant":
        return 1.0, 0.0, 1.0, 0.0
    if case.get("flow") == "channel":
        dt = 100.0
    elif case["kind"] == "meshes":
        dt = COURANT / 32.0
    else:
        dt = COURANT / max(case["nex"], case["ney"], case["nez"])
    return 2.0, 3.0 / dt, 3.0, 3.0 / dt


def _of(case, seed):
    return _system(case.get("flow", "rotation"), case["nex"], case["ney"], case["nez"], seed)


def _sources(S, K):
    """K per-element source fields, one Gaussian blob each."""
    cx, cy, cz = (c[S["nod"]].mean(0) for c in S["xyz"])
    return torch.stack([_blobs(S["gen"], cx, cy, cz, 1) / cx.numel() for _ in range(K)])


def _cubes(case, seed):
    lo, span = case["nmin"], case["nmax"] - case["nmin"] + 1
    sizes = [lo + (m * 29 + 7) % span for m in range(case["nmesh"])]
    return [_system("rotation", n, n, n, int(seed) * 1000 + m) for m, n in enumerate(sizes)]


def _union(systems):
    """The block-diagonal system of several meshes."""
    off = np.cumsum([0] + [s["xyz"][0].numel() for s in systems])
    cat = lambda k, d=-1: torch.cat([s[k] for s in systems], dim=d)  # noqa: E731
    U = dict(nod=torch.cat([s["nod"] + int(o) for s, o in zip(systems, off)], dim=1),
             kod=cat("kod"), xyz=tuple(torch.cat([s["xyz"][d] for s in systems])
                                       for d in range(3)),
             vel=cat("vel"), lam=cat("lam"), pdec=cat("pdec"), q=cat("q"), bc=cat("bc"),
             alpha=0.0, told=cat("told"))
    U["off"] = off
    return U


# channels (skip, upsampled, out) of the network's 3x3x3 layers, in the order
# of its flat parameter array; the head (16 weights, one bias) is last
LAYERS = ((16, 0, 16), (16, 0, 16), (16, 0, 32), (32, 0, 32), (32, 0, 64), (64, 0, 64),
          (32, 64, 32), (32, 0, 32), (16, 32, 16), (16, 0, 16))


def _parameters(g):
    """Weights of a trained network's scale: He-scaled normals, small biases,
    every layer starting at a multiple of 8 floats."""
    parts = []
    for ws, co, fan in [(27 * co * (a + b), co, 27 * (a + b)) for a, b, co in LAYERS] + \
            [(16, 1, 16)]:
        w = torch.randn(ws, generator=g, dtype=F64, device=DEV) * math.sqrt(2.0 / fan)
        b = 0.1 * torch.randn(co, generator=g, dtype=F64, device=DEV)
        parts += [w, b, torch.zeros(-(ws + co) % 8, dtype=F64, device=DEV)]
    return torch.cat(parts).to(torch.float32)


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    aH, aM, cf, rM = _coefficients(case)
    st = dict(kind=kind, aH=aH, aM=aM, cf=cf, rM=rM, tol=case.get("tol"))
    if kind == "meshes":
        U = _union(_cubes(case, seed))
        off = U["off"].astype(np.int64)
        mesh = P.MeshUnion(0, 0, 0, *(_host(c) for c in U["xyz"]),
                           _host((U["nod"] + 1).to(torch.int32)), _host(U["kod"]),
                           n_node=int(off[-1]), n_elem=U["nod"].shape[1], node_off=off)
        prob = P.Problem("cubes", mesh, _host(U["vel"]), _host(U["lam"]), _host(U["pdec"]),
                         _host(U["q"]), _host(U["bc"]), 0.0, P.DR_VF, case["tol"])
        st["s"] = s = vdr.Solver(prob, vdr.Options(), aH=aH, aM=aM)
        s.set_segments(off)
        st["b"] = torch.empty(int(off[-1]), dtype=F64, device=DEV)
        st["x"] = torch.empty_like(st["b"])
        return st
    S = _of(case, seed)
    prob = _problem(S, case.get("variant", "vf"), case.get("tol", 1e-8))
    s = vdr.Solver(prob, vdr.Options(precision=case.get("precision", "fp64")), aH=aH, aM=aM)
    N = s.N
    if kind == "dropin":
        m = prob.mesh
        b = s.assemble_rhs(cf, rM, _host(S["told"]))
        b[prob.bc == 1] = 0.0
        st["args"] = (N, b, _host(S["told"]), case["tol"], 2000, s.element_matrices(), m.iss,
                      s.diag(), m.nax, m.nay, m.naz, prob.bc)
        s.close()
        return st
    st["s"] = s
    if kind == "step":
        st["told"] = S["told"] if case["warm"] else None
        st["b"], st["x"] = (torch.empty(N, dtype=F64, device=DEV) for _ in range(2))
    elif kind == "loop":
        st["told"], st["steps"] = S["told"], case["steps"]
        st["x"] = torch.empty(N, dtype=F64, device=DEV)
    elif kind == "block":
        st["Q"] = _sources(S, case["K"])
        st["B"], st["X"] = (torch.empty((N, case["K"]), dtype=F64, device=DEV)
                            for _ in range(2))
    elif kind == "net":
        st["net"] = net = vdr.LearnedNet(s, seed=1)
        st["train"] = case["train"]
        net.set_params(_parameters(S["gen"]).cpu().numpy())
        net.update_features()
        st["r"] = torch.randn(N, generator=S["gen"], dtype=torch.float32, device=DEV)
        st["out"] = torch.empty_like(st["r"])
    return st


# --------------------------------------------------------------------- run
def run(state):
    kind, st = state["kind"], state
    if kind == "dropin":
        return vdr.kernel_dbcg_simple(*st["args"])[0]
    s = st["s"]
    if kind == "step":
        # new fields or a new step size mark the operator stale; the step
        # builds it with the right-hand side and solves from the old field
        s.set_operator(st["aH"], st["aM"])
        s.assemble_rhs_device(st["b"], st["cf"], st["rM"], st["told"])
        if st["told"] is None:
            st["x"].zero_()
        else:
            st["x"].copy_(st["told"])
        status = s.solve_device(st["b"], st["x"], tol=st["tol"], itmax=5000)[2]
        if status != 0:
            raise RuntimeError("solve status %d" % status)
        return {"b": st["b"], "x": st["x"]}
    if kind == "loop":
        s.set_operator(st["aH"], st["aM"])
        st["x"].copy_(st["told"])
        masses, _, _, status, _ = s.time_steps_device(st["x"], st["steps"], st["cf"],
                                                      st["rM"], tol=st["tol"], itmax=5000)
        if status != 0:
            raise RuntimeError("time loop status %d" % status)
        return {"x": st["x"], "masses": masses}
    if kind == "block":
        s.assemble_rhs_block_device(st["Q"], st["B"], st["cf"])
        st["X"].zero_()
        status = s.solve_block_device(st["B"], st["X"], tol=st["tol"], inner_tol=1e-4)[3]
        if status != 0:
            raise RuntimeError("block solve status %d" % status)
        return {"B": st["B"], "X": st["X"]}
    if kind == "meshes":
        s.set_operator(st["aH"], st["aM"])
        s.assemble_rhs_device(st["b"], st["cf"], st["rM"], None)
        st["x"].zero_()
        status = s.solve_segmented_device(st["b"], st["x"], tol=st["tol"], itmax=5000)[3]
        if status != 0:
            raise RuntimeError("segmented solve status %d" % status)
        return {"b": st["b"], "x": st["x"]}
    if st["train"]:
        loss = st["net"].residual_loss_grad(st["r"])
        return {"loss": loss, "grad": st["net"].get_grads()}
    st["net"].forward(st["r"], st["out"])
    return st["out"]


# -------------------------------------------------------------------- work
# iterations that the solves of each kind take, to the nearest few
ITERATIONS = {"step": 33, "loop": 25, "block": 45, "meshes": 30, "dropin": 60}


def work(case):
    kind = case["kind"]
    if kind == "meshes":
        lo, span = case["nmin"], case["nmax"] - case["nmin"] + 1
        sizes = [lo + (m * 29 + 7) % span for m in range(case["nmesh"])]
        E, N = sum(n ** 3 for n in sizes), sum((n + 1) ** 3 for n in sizes)
    else:
        E = case["nex"] * case["ney"] * case["nez"]
        N = (case["nex"] + 1) * (case["ney"] + 1) * (case["nez"] + 1)
    mesh = 24 * N + 32 * E
    if kind == "net":
        n1 = [(v + 2) // 2 for v in (case["nex"], case["ney"], case["nez"])]
        n2 = [(v + 1) // 2 for v in n1]
        vox = (N, math.prod(n1), math.prod(n2))
        level = (0, 0, 1, 1, 2, 2, 1, 1, 0, 0)
        flops = sum(2 * vox[lv] * 27 * (a + b) * co
                    for lv, (a, b, co) in zip(level, LAYERS)) + 32 * N
        return {"bytes": 24 * N if not case["train"] else 24 * N + 544 * E,
                "flops": flops * (3 if case["train"] else 1)}
    if kind == "dropin":
        return {"bytes": 512 * E + 32 * E + 36 * N, "flops": 2 * 128 * E * ITERATIONS[kind]}
    if kind == "block":
        K = case["K"]
        return {"bytes": 8 * K * E + 16 * K * N + mesh, "flops": 2 * 128 * E * K * 45}
    steps = case.get("steps", 1)
    return {"bytes": mesh + 48 * E + 24 * N,
            "flops": 4500 * E + steps * ITERATIONS[kind] * 2 * (128 * E + 20 * N)}


# ------------------------------------------------- the same in 64 bits, torch
def _shape(xi, eta, zeta):
    t = lambda s: torch.tensor(s, dtype=F64, device=DEV)  # noqa: E731
    sx, sy, sz = t(SX), t(SY), t(SZ)
    n = 0.125 * (1 + sx * xi) * (1 + sy * eta) * (1 + sz * zeta)
    dn = torch.stack([0.125 * sx * (1 + sy * eta) * (1 + sz * zeta),
                      0.125 * sy * (1 + sx * xi) * (1 + sz * zeta),
                      0.125 * sz * (1 + sx * xi) * (1 + sy * eta)])
    return n, dn


def _tau(variant, X, inv, lam, v):
    vm = v.square().sum(1).sqrt()
    if variant == "ot":
        dl = torch.stack([X[:, 0, 1] - X[:, 0, 0], X[:, 1, 3] - X[:, 1, 0],
                          X[:, 2, 4] - X[:, 2, 0]], 1).abs()
        h = 2.0 / ((v.abs() / dl).sum(1) + 1e-14)
    else:
        h = 2.0 / torch.einsum("eab,eb->ea", inv, v / vm[:, None].clamp_min(1e-300)).norm(dim=1)
    pe = vm * h / (2.0 * lam)
    beta = 1.0 / torch.tanh(pe) - 1.0 / pe
    small = pe < (1e-3 if variant == "vf" else 1e-2)
    beta = torch.where(small, pe / 3 - pe ** 3 / 45 + 2 * pe ** 5 / 945, beta)
    tau = 0.5 * h / vm * beta
    return torch.where((vm > 1e-14) & (pe > 1e-12), tau, torch.zeros_like(tau))


def _elements(S, variant, lo, hi):
    """H, M [e, 8, 8] and the source weights f_i / q [e, 8] of elements lo..hi."""
    nod = S["nod"][:, lo:hi].T
    X = torch.stack([c[nod] for c in S["xyz"]], 1)  # [e, 3, 8]
    v, lam = S["vel"][:, lo:hi].T, S["lam"][lo:hi]
    H = torch.zeros(nod.shape[0], 8, 8, dtype=F64, device=DEV)
    M, f = torch.zeros_like(H), torch.zeros(nod.shape[0], 8, dtype=F64, device=DEV)
    vol = torch.zeros_like(lam)

    def point(xi, eta, zeta):
        n, dn = _shape(xi, eta, zeta)
        J = torch.einsum("ecn,dn->ecd", X, dn)
        inv = torch.linalg.inv(J)
        tau = _tau(variant, X, inv, lam, v)
        a = torch.einsum("ecd,ed,cn->en", inv, v, dn)
        return n, dn, torch.linalg.det(J), inv, a, n + tau[:, None] * a

    for q in range(8):
        n, dn, det, inv, a, w = point(GAUSS * SX[q], GAUSS * SY[q], GAUSS * SZ[q])
        grad = torch.einsum("ecd,cn->edn", inv, dn)
        wd = w * det[:, None]
        H += torch.einsum("edi,edj->eij", grad * (lam * det)[:, None, None], grad)
        H += wd[:, :, None] * (a + S["pdec"][lo:hi, None] * n)[:, None, :]
        M += wd[:, :, None] * n
        f += wd
        vol += det
    if S["alpha"]:  # third-kind term on the face xi = -1
        on = (S["kod"][2, lo:hi] == 3).to(F64) * S["alpha"]
        face = X[:, :, [0, 3, 7, 4]]
        for r in (-GAUSS, GAUSS):
            for s in (-GAUSS, GAUSS):
                dr = torch.tensor([s - 1, 1 - s, 1 + s, -1 - s], dtype=F64, device=DEV) / 4
                ds = torch.tensor([r - 1, -1 - r, 1 + r, 1 - r], dtype=F64, device=DEV) / 4
                area = torch.linalg.cross(face @ dr, face @ ds).norm(dim=1)
                n, _, _, _, _, w = point(-1.0, r, s)
                H += (on * area)[:, None, None] * w[:, :, None] * n
    return H, M, f / vol[:, None]


def _assemble(S, variant, co, told=None, keep_mass=False):
    """A [E, 8, 8], b (zero on Dirichlet rows), diag, source weights and
    (asked for) M."""
    aH, aM, cf, rM = co
    E, N = S["nod"].shape[1], S["xyz"][0].numel()
    A = torch.empty(E, 8, 8, dtype=F64, device=DEV)
    M = torch.empty(E, 8, 8, dtype=F64, device=DEV) if keep_mass else None
    phi = torch.empty(E, 8, dtype=F64, device=DEV)
    b = torch.zeros(N, dtype=F64, device=DEV)
    diag = torch.zeros_like(b)
    for lo in range(0, E, 1 << 18):
        hi = min(E, lo + (1 << 18))
        h, m, f = _elements(S, variant, lo, hi)
        A[lo:hi], phi[lo:hi] = aH * h + aM * m, f
        nod = S["nod"][:, lo:hi].T
        be = cf * f * S["q"][lo:hi, None]
        if told is not None:
            be = be - ((h - rM * m) @ told[nod][:, :, None])[:, :, 0]
        b.index_add_(0, nod.reshape(-1), be.reshape(-1))
        diag.index_add_(0, nod.reshape(-1), torch.diagonal(A[lo:hi], dim1=1, dim2=2).reshape(-1))
        if keep_mass:
            M[lo:hi] = m
    free = S["bc"] == 0
    return A, b * free, torch.where(free, diag, torch.ones_like(diag)), phi, M


def _apply(S, A, x):
    """sum_e A_e x for x [N, K]."""
    y = torch.zeros_like(x)
    E, step = A.shape[0], max(1, (1 << 27) // (8 * x.shape[1]))
    for lo in range(0, E, step):
        nod = S["nod"][:, lo:lo + step].T
        ye = torch.bmm(A[lo:lo + step], x[nod])
        y.index_add_(0, nod.reshape(-1), ye.reshape(-1, x.shape[1]))
    return y


def _solve(S, A, diag, b, x0=None):
    """Jacobi-BiCGStab on P A P, columns of b at once, restarted on its own
    residual until that no longer falls."""
    one = b.dim() == 1
    b = b[:, None] if one else b
    free = (S["bc"] == 0).to(F64)[:, None]
    b, dinv = b * free, (1.0 / diag)[:, None]
    op = lambda x: free * _apply(S, A, x)  # noqa: E731
    norm = b.norm(dim=0).clamp_min(1e-300)
    x = torch.zeros_like(b) if x0 is None else (x0[:, None] if one else x0) * free
    best = math.inf
    safe = lambda t: torch.where(t == 0, torch.ones_like(t), t)  # noqa: E731
    for _ in range(4):
        r = b - op(x)
        rel = float((r.norm(dim=0) / norm).max())
        if rel < 2e-15 or rel > 0.3 * best:
            break
        best = rel
        scale = r.norm(dim=0).clamp_min(1e-300)
        rh, p, rho, y = r, r, (r * r).sum(0), torch.zeros_like(x)
        for _ in range(3000):
            v = op(dinv * p)
            al = rho / safe((rh * v).sum(0))
            s = r - al * v
            t = op(dinv * s)
            om = (t * s).sum(0) / safe((t * t).sum(0))
            y = y + dinv * (al * p + om * s)
            r = s - om * t
            if float((r.norm(dim=0) / scale).max()) < 1e-10:
                break
            new = (rh * r).sum(0)
            p = r + (new / safe(rho) * al / safe(om)) * (p - om * v)
            rho = new
        x = x + y
    return x[:, 0] if one else x


def _conv(x, w, bias):
    """3x3x3 convolution with zero padding and ReLU; x [D, H, W, C], w
    [27, out, C]."""
    D, Hh, W, C = x.shape
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    y = bias.expand(D * Hh * W, -1)
    for t in range(27):
        dz, dy, dx = t // 9, t // 3 % 3, t % 3
        y = y + xp[dz:dz + D, dy:dy + Hh, dx:dx + W].reshape(-1, C) @ w[t].T
    return torch.relu(y).reshape(D, Hh, W, -1)


def _pool(x):
    D, Hh, W, C = x.shape
    pad = (0, 0, 0, W % 2, 0, Hh % 2, 0, D % 2)
    s, n = (torch.nn.functional.pad(t, pad) for t in (x, torch.ones_like(x[..., :1])))
    f = lambda t: t.reshape((t.shape[0] // 2, 2, t.shape[1] // 2, 2,  # noqa: E731
                             t.shape[2] // 2, 2, t.shape[3])).sum(dim=(1, 3, 5))
    return f(s) / f(n)


def _up(x, like):
    for d in range(3):
        x = x.repeat_interleave(2, dim=d)
    return x[:like.shape[0], :like.shape[1], :like.shape[2]]


def _network(S, theta, r):
    nex, ney, nez = S["dims"]
    shape = (nez + 1, ney + 1, nex + 1)
    N, nod = r.numel(), S["nod"]
    acc, cnt = torch.zeros(N, 4, dtype=F64, device=DEV), torch.zeros(N, 1, dtype=F64, device=DEV)
    fe = torch.cat([S["vel"], (S["lam"].log() - math.log(1e-4))[None]]).T
    for a in range(8):
        acc.index_add_(0, nod[a], fe)
        cnt.index_add_(0, nod[a], torch.ones_like(fe[:, :1]))
    x = torch.zeros(N, 16, dtype=F64, device=DEV)
    x[:, 0], x[:, 1:5] = r, acc / cnt
    x = x.reshape(*shape, 16)
    ws, at = [], 0
    for a, b, co in LAYERS:
        n = 27 * co * (a + b)
        ws.append((theta[at:at + n].reshape(27, co, a + b), theta[at + n:at + n + co]))
        at += n + co + -(n + co) % 8
    head, bias = theta[at:at + 16], theta[at + 16]
    s0 = _conv(_conv(x, *ws[0]), *ws[1])
    s1 = _conv(_conv(_pool(s0), *ws[2]), *ws[3])
    b2 = _conv(_conv(_pool(s1), *ws[4]), *ws[5])
    u1 = _conv(_conv(torch.cat([s1, _up(b2, s1)], -1), *ws[6]), *ws[7])
    u0 = _conv(_conv(torch.cat([s0, _up(u1, s0)], -1), *ws[8]), *ws[9])
    return u0.reshape(N, 16) @ head + bias


def exact(case, seed):
    kind, co = case["kind"], _coefficients(case)
    variant = case.get("variant", "vf")
    if kind == "meshes":
        U = _union(_cubes(case, seed))
        A, b, diag, _, _ = _assemble(U, variant, co)
        return {"b": b, "x": _solve(U, A, diag, b)}
    S = _of(case, seed)
    if kind == "step":
        told = S["told"] if case["warm"] else None
        A, b, diag, _, _ = _assemble(S, variant, co, told)
        return {"b": b, "x": _solve(S, A, diag, b, told)}
    if kind == "dropin":
        A, b, diag, _, _ = _assemble(S, variant, co, S["told"])
        return _solve(S, A, diag, b, S["told"]).cpu().numpy()
    if kind == "block":
        Q = _sources(S, case["K"])
        A, _, diag, phi, _ = _assemble(S, variant, co)
        B = torch.zeros(diag.numel(), case["K"], dtype=F64, device=DEV)
        for lo in range(0, Q.shape[1], 1 << 18):
            nod = S["nod"][:, lo:lo + (1 << 18)].T
            w = co[2] * phi[lo:lo + (1 << 18), :, None] * Q[:, lo:lo + (1 << 18)].T[:, None, :]
            B.index_add_(0, nod.reshape(-1), w.reshape(-1, case["K"]))
        B *= (S["bc"] == 0).to(F64)[:, None]
        return {"B": B, "X": _solve(S, A, diag, B)}
    if kind == "loop":
        aH, aM, cf, rM = co
        A, F, diag, _, M = _assemble(S, variant, co, None, keep_mass=True)
        t, masses = S["told"].clone(), []
        one = torch.ones_like(t)
        # detJ-weighted shape integrals from M's trial side: sum_i M_ij is
        # int N_j plus the test function's streamline part, so the mass
        # integral is taken from an unstabilised copy
        plain = dict(S, vel=torch.zeros_like(S["vel"]))
        for _ in range(case["steps"]):
            ht = (_apply(S, A, t[:, None]) - aM * _apply(S, M, t[:, None]))[:, 0] / aH
            b = F - (ht - rM * _apply(S, M, t[:, None])[:, 0])
            t = _solve(S, A, diag, b, t)
            m = 0.0
            for lo in range(0, A.shape[0], 1 << 18):
                hi = min(A.shape[0], lo + (1 << 18))
                nod = S["nod"][:, lo:hi].T
                mm = _elements(plain, "vf", lo, hi)[1]
                m += float((one[nod][:, None, :] @ mm @ t[nod][:, :, None]).sum())
            masses.append(m)
        return {"x": t, "masses": np.array(masses)}
    theta = _parameters(S["gen"]).to(F64)
    r = torch.randn(S["xyz"][0].numel(), generator=S["gen"], dtype=torch.float32,
                    device=DEV).to(F64)
    if not case["train"]:
        return _network(S, theta, r)
    theta.requires_grad_(True)
    A, _, diag, _, _ = _assemble(S, variant, co)
    free = (S["bc"] == 0).to(F64)
    dbar = (diag * free).sum() / free.sum()
    z = free * (r / diag + _network(S, theta, r) / dbar)
    rho = free * r - free * _apply(S, A, z[:, None])[:, 0]
    loss = rho.square().sum() / (free * r).square().sum()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": theta.grad.to(torch.float32).cpu().numpy()}

