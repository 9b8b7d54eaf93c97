"""Performance cases: the work a user of this package has it do, over the sizes it is used at.

Each case calls the package through the bindings of its C ABI (``andosim_b200.abi``): whole
frames in both semantics and with both preconditioners, a batch of small scenes, and the single
stages a program calls on their own (the contact query, the broad phase, the Newton system, the
learned preconditioner's evaluation and its training gradient, the PCG on a caller's system).
Scenes come from ``andosim_b200.scenes``; the sizes are those of its configurations and of the
tests, and odd ones between them.

A frame case sets the scene's state and steps it once, so every pass does the same work. The
solver's tolerances are 1e-3 to 1e-4 and its vectors are single precision, so a frame's positions
and velocities are handed on in single precision, as a cache or a renderer takes them.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from andosim_b200 import abi, learned, scenes

GRAVITY = np.array([0.0, 0.0, -9.81])


# ------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # the module's default semantics on its smallest configuration: launches and latency
        {"name": "frame_reference_32", "kind": "frame_reference", "n": 32},
        # many small scenes at once (a parameter sweep, training data): 16 uneven cloths
        {"name": "frame_batch_16_scenes", "kind": "frame_batch", "scenes": 16, "lo": 16, "hi": 128},
        # a stack of sheets lying on one another: contacts at nearly every vertex
        {"name": "frame_stack_4x96", "kind": "frame_stack", "n": 96, "sheets": 4},
        # driven curtains, block Jacobi, an odd size between the tests' and the benchmark's
        {"name": "frame_curtains_2x151", "kind": "frame_curtains", "n": 151, "precond": "block_jacobi"},
        # the benchmark's curtains with the learned preconditioner (the largest frame)
        {"name": "frame_curtains_2x256_learned", "kind": "frame_curtains", "n": 256, "precond": "learned"},
        # a host with its own system: one small cloth's, and the tablecloth's 512 x 512
        {"name": "pcg_32x32", "kind": "pcg", "nx": 32, "ny": 32, "tol": 1e-4},
        {"name": "pcg_512x512", "kind": "pcg", "nx": 512, "ny": 512, "tol": 1e-4},
        # the validator's contact list of the stack
        {"name": "contacts_4x96", "kind": "contacts", "n": 96, "sheets": 4},
        # candidate pairs, as a host with its own narrow phase takes them
        {"name": "broad_phase_3x127", "kind": "broad_phase", "n": 127, "sheets": 3, "query": 1},
        # gradient and Hessian of a hanging cloth, read back (solver dump)
        {"name": "newton_system_97", "kind": "newton_system", "n": 97},
        # the preconditioner evaluated on a frame's first system and read back
        {"name": "precond_eval_2x128", "kind": "precond_eval", "n": 128},
        # forward and backward of one training system
        {"name": "train_gradient_2x64", "kind": "train_gradient", "n": 64},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["frame_reference", "frame_batch", "frame_stack", "frame_curtains", "frame_curtains", "pcg", "pcg",
                       "contacts", "broad_phase", "newton_system", "precond_eval", "train_gradient"])
    if kind == "frame_reference":
        return {"kind": kind, "n": logint(8, 256)}
    if kind == "frame_batch":
        lo = logint(8, 48)
        return {"kind": kind, "scenes": rng.randint(2, 16), "lo": lo, "hi": rng.randint(lo + 1, 128)}
    if kind in ("frame_stack", "contacts"):
        return {"kind": kind, "n": logint(12, 96), "sheets": rng.randint(2, 4)}
    if kind == "frame_curtains":
        return {"kind": kind, "n": logint(16, 230), "precond": rng.choice(["block_jacobi", "learned"])}
    if kind == "pcg":
        return {"kind": kind, "nx": logint(5, 500), "ny": logint(5, 500), "tol": rng.choice([1e-3, 1e-4, 1e-5])}
    if kind == "broad_phase":
        return {"kind": kind, "n": logint(12, 110), "sheets": rng.randint(2, 4), "query": rng.randint(0, 1)}
    if kind == "newton_system":
        return {"kind": kind, "n": logint(9, 200)}
    return {"kind": kind, "n": logint(12, 128 if kind == "precond_eval" else 80)}


# ------------------------------------------------------------------------------------------ scenes
def stack(n, sheets, seed):
    """Sheets of scenes.c2 (each turned by its own angle) lying 0.7 mm over one another on one wavy ground, falling slowly."""
    sc = scenes.c2(seed=seed, n=n, sheets=sheets, wave=0.0)
    rng = np.random.default_rng(seed + 1)
    x = sc.vertices
    h = np.zeros(len(x))
    for _ in range(3):
        th, lam, ph = rng.uniform(0, 2 * math.pi), rng.uniform(0.3, 0.6), rng.uniform(0, 2 * math.pi)
        h += np.sin(2 * math.pi * (x[:, 0] * math.cos(th) + x[:, 1] * math.sin(th)) / lam + ph)
    x[:, 2] = 0.004 + 0.002 * h / 3.0 + 0.0007 * np.repeat(np.arange(sheets), n * n) + rng.uniform(-2e-5, 2e-5, len(x))
    v = rng.normal(0.0, 2e-3, x.shape)
    v[:, 2] -= 0.02
    return sc, x, v


def curtains(n, seed):
    """scenes.c4 at an early frame of its drive: the pins one frame ahead, the cloth moving with them."""
    size = 2.0 * (n - 1) / 255.0        # the 256 x 256 configuration's edge length
    sc = scenes.c4(seed=seed, n=n, size=max(size, 0.05))
    rng = np.random.default_rng(seed + 1)
    v = rng.normal(0.0, 2e-3, sc.vertices.shape)
    return sc, sc.vertices, v, sc.pins_at(5)


def hanging(n, seed):
    """scenes.c1 sagging between its pinned corners, moving."""
    sc = scenes.c1(seed=seed, n=n)
    rng = np.random.default_rng(seed + 1)
    x = sc.vertices.copy()
    bump = np.sin(math.pi * x[:, 0]) * np.sin(math.pi * x[:, 1])
    x[:, 2] -= rng.uniform(0.02, 0.04) * bump
    x += rng.normal(0.0, 1e-3 / n, x.shape)
    v = rng.normal(0.0, 1e-2, x.shape)
    v[:, 2] -= 0.3 * bump
    return sc, x, v


def scene(sc):
    return abi.Scene(sc.vertices, sc.triangles, sc.material)


def grid_system(nx, ny, seed, device, dtype):
    """A cloth-like SPD system on an nx by ny vertex grid with the scenes' triangulation: a mass term, and per mesh edge
    a stiffness block a I + b n n^T with b / a and the stiffness spread as in a stretched sheet. Block offsets of a row and, per
    offset, the blocks (zero where the neighbour does not exist)."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    V = nx * ny
    steps = {(1, 0): 1, (0, 1): nx, (-1, 1): nx - 1}    # edges along x, along y, and the diagonal split
    idx = torch.arange(V)
    ix, iy = idx % nx, idx // nx
    rand = torch.rand(len(steps), V, 2, generator=g)
    nrm = torch.randn(len(steps), V, 3, generator=g)
    rhs = torch.randn(V, 3, generator=g)
    rand, nrm, rhs, ix, iy = (t.to(device) for t in (rand, nrm, rhs, ix, iy))
    nrm = (nrm / nrm.norm(dim=2, keepdim=True)).float()
    k = (20.0 * torch.exp(rand[..., 0] - 0.5)).float()
    eye = torch.eye(3, device=device)
    diag = torch.eye(3, device=device).repeat(V, 1, 1)
    off = {}
    for e, ((dx, dy), st) in enumerate(steps.items()):
        ok = (ix + dx >= 0) & (ix + dx < nx) & (iy + dy < ny)
        B = k[e][:, None, None] * (0.2 * eye + rand[e, :, 1][:, None, None] * nrm[e][:, :, None] * nrm[e][:, None, :])
        B = torch.where(ok[:, None, None], B, torch.zeros_like(B))
        down = torch.zeros_like(B)
        down[st:] = B[:V - st]
        diag = diag + B + down
        off[st], off[-st] = -B, -down
    off[0] = diag
    order = sorted(off)
    there = torch.stack([(off[o].abs().amax(dim=(1, 2)) > 0) for o in order], dim=1)      # V x 7
    blocks = torch.stack([off[o] for o in order], dim=1).to(torch.float32)                # V x 7 x 3 x 3
    return order, there, blocks, rhs.to(torch.float32).contiguous()


# ----------------------------------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "frame_reference":
        sc, x, v = hanging(case["n"], seed)
        S = scene(sc)
        p = abi.make_params(sc.params, semantics="reference")
        s.update(S=S, p=p, x=x, v=v, pins=abi.pin_array(sc.pins), walls=sc.walls)
    elif kind == "frame_stack":
        sc, x, v = stack(case["n"], case["sheets"], seed)
        s.update(S=scene(sc), p=abi.make_params(sc.params, semantics="corrected"), x=x, v=v, pins=(), walls=sc.walls)
    elif kind == "frame_curtains":
        sc, x, v, pins = curtains(case["n"], seed)
        S = scene(sc)
        refresh = 8
        if case["precond"] == "learned":
            S.set_precond_weights(learned.load_weights())
        p = abi.make_params(sc.params, semantics="corrected", precond=case["precond"], precond_refresh=refresh)
        s.update(S=S, p=p, x=x, v=v, pins=abi.pin_array(pins), walls=sc.walls)
    elif kind == "frame_batch":
        rng = np.random.default_rng(seed)
        items = []
        for k in range(case["scenes"]):
            n = case["lo"] + (k * 37) % (case["hi"] - case["lo"] + 1)      # uneven sizes, the same for every seed
            sc, x, v = hanging(n, seed * 64 + k)
            sc.material["youngs_modulus"] = float(10 ** rng.uniform(4, 6))
            p = abi.make_params(dict(sc.params, enable_strain_limiting=False), semantics="corrected")
            items.append((scene(sc), p, x, v, abi.pin_array(sc.pins), sc.walls))
        s.update(items=items)
    elif kind == "pcg":
        dev = torch.device("cuda")
        order, there, blocks, rhs = grid_system(case["nx"], case["ny"], seed, dev, torch.float32)
        V = case["nx"] * case["ny"]
        cols = (torch.arange(V, device=dev)[:, None] + torch.tensor(order, device=dev)[None, :])[there].to(torch.int32).contiguous()
        rowptr = torch.zeros(V + 1, dtype=torch.int32, device=dev)
        rowptr[1:] = there.sum(dim=1).cumsum(0).to(torch.int32)
        s.update(V=V, rowptr=rowptr, cols=cols, vals=blocks[there].contiguous(), rhs=rhs, tol=case["tol"],
                 x=torch.empty(3 * V, device=dev), work=torch.empty(24 * V, device=dev))
    elif kind == "contacts":
        sc, x, v = stack(case["n"], case["sheets"], seed)
        s.update(S=scene(sc), x=x, v=v, buf=np.zeros(16 * len(x), CONTACT))
    elif kind == "broad_phase":
        sc, x, v = stack(case["n"], case["sheets"], seed)
        s.update(S=scene(sc), x=x, query=case["query"], buf=np.zeros((96 * len(x), 2), np.int32))
    elif kind == "newton_system":
        sc, x, v = hanging(case["n"], seed)
        s.update(S=scene(sc), p=abi.make_params(sc.params, semantics="corrected"), x=x, v=v, pins=abi.pin_array(sc.pins), walls=sc.walls)
    elif kind in ("precond_eval", "train_gradient"):
        sc, x, v, pins = curtains(case["n"], seed)
        S = scene(sc)
        p = abi.make_params(sc.params, semantics="corrected")
        pins = abi.pin_array(pins)
        w = learned.load_weights()
        if kind == "precond_eval":
            S.set_precond_weights(w)
            s.update(S=S, p=p, x=x, v=v, pins=pins, walls=sc.walls)
        else:
            T = abi.Trainer(w)
            S.upload(x, v)
            S.eval_system(p, pins, sc.walls)
            T.add_system(S, max_probes=4, tol=1e-6)
            s.update(T=T, S=S)
    else:
        raise ValueError(kind)
    if kind.startswith("frame"):
        run(s)      # the frame before: launch shapes chosen, buffers at their sizes, as in any run of more than one frame
    return s


# --------------------------------------------------------------------------------------------- run
def run(s):
    kind = s["kind"]
    if kind == "frame_batch":
        for S, p, x, v, _, _ in s["items"]:
            S.upload(x, v)
            S.apply_gravity(GRAVITY, p.dt)
        it = s["items"]
        abi.step_batch([i[0] for i in it], [i[1] for i in it], [i[4] for i in it], [i[5] for i in it])
        return [tuple(a.astype(np.float32) for a in i[0].download()) for i in it]
    if kind.startswith("frame"):
        S = s["S"]
        S.upload(s["x"], s["v"], s["x"])
        S.apply_gravity(GRAVITY, s["p"].dt)
        S.step(s["p"], s["pins"], s["walls"])
        x, v = S.download()
        return x.astype(np.float32), v.astype(np.float32)
    if kind == "pcg":
        it, status, rel = C.c_int32(), C.c_int32(), C.c_double()
        L = abi.lib()
        rc = L.ando_pcg_solve_noalloc(
            0, C.c_void_p(torch.cuda.current_stream().cuda_stream), s["V"], s["rowptr"].data_ptr(), s["cols"].data_ptr(),
            s["vals"].data_ptr(), s["rhs"].data_ptr(), s["x"].data_ptr(), s["work"].data_ptr(), s["work"].numel(), s["tol"], 1000,
            C.byref(it), C.byref(status), C.byref(rel))
        if rc or status.value:
            raise RuntimeError(f"pcg: {rc} {status.value} {L.ando_last_error().decode()}")
        return s["x"]
    S = s["S"]
    if kind == "contacts":
        S.upload(s["x"], s["v"])
        n = C.c_int32()
        c = s["buf"]
        rc = abi.lib().ando_compute_contacts_corrected(S.ctx, 1e-3, None, 0, c.ctypes.data_as(C.POINTER(abi.Contact)), len(c), C.byref(n))
        if rc:
            raise RuntimeError(f"contacts: {rc} {abi.lib().ando_last_error().decode()}")
        return {"n": n.value, **{name: c[name] for name in CONTACT.names}}
    if kind == "broad_phase":
        S.upload(s["x"])
        n = C.c_int32()
        rc = abi.lib().ando_broad_phase(S.ctx, s["query"], 5e-4, s["buf"].ctypes.data_as(C.POINTER(C.c_int32)), len(s["buf"]), C.byref(n))
        if rc:
            raise RuntimeError(f"broad phase: {rc} {abi.lib().ando_last_error().decode()}")
        return {"n": n.value, "pairs": s["buf"]}
    if kind == "newton_system":
        S.upload(s["x"], s["v"])
        S.eval_system(s["p"], s["pins"], s["walls"])
        rowptr, cols, vals, rhs, _ = S.last_system()
        return {"gradient": S.last_gradient(), "rowptr": rowptr, "cols": cols, "vals": vals, "rhs": rhs}
    if kind == "precond_eval":
        S.upload(s["x"], s["v"])
        S.eval_system(s["p"], s["pins"], s["walls"])
        return S.precond_eval()
    loss, grad = s["T"].loss(0, grad=True)
    return {"loss": loss, "gradient": grad}


# type, four vertex indices, body, count | gap, normal, witnesses, barycentric, weights (abi.Contact)
CONTACT = np.dtype([("ids", "<i4", (8,)), ("gap", "<f8"), ("normal", "<f8", (3,)), ("witness", "<f8", (6,)), ("bary", "<f8", (3,)),
                    ("weights", "<f8", (4,))])
assert CONTACT.itemsize == C.sizeof(abi.Contact)


# ------------------------------------------------------------------------------------------- exact
def exact(case, seed):
    """The PCG's solution and the hanging cloth's gradient and Hessian in 64 bits; the other outputs are whole frames, lists
    or a network's outputs, which have no value independent of this code."""
    if case["kind"] == "pcg":
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        order, there, blocks, rhs = grid_system(case["nx"], case["ny"], seed, dev, torch.float32)
        V = case["nx"] * case["ny"]
        A, b = blocks.double(), rhs.double()
        cols = (torch.arange(V, device=dev)[:, None] + torch.tensor(order, device=dev)[None, :]).clamp(0, V - 1)
        P = torch.linalg.inv(A[:, order.index(0)])

        def mul(p):
            return torch.einsum("vkab,vkb->va", A, p[cols])

        x = torch.zeros_like(b)
        r = b.clone()
        z = torch.einsum("vab,vb->va", P, r)
        p, rz = z.clone(), (r * z).sum()
        for it in range(2000):
            q = mul(p)
            a = rz / (p * q).sum()
            x += a * p
            r -= a * q
            if it % 10 == 9 and float(r.abs().max()) < 1e-13 * float(b.abs().max()):
                break
            z = torch.einsum("vab,vb->va", P, r)
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
        return x.reshape(-1).cpu().numpy()
    if case["kind"] != "newton_system":
        return None
    # hanging cloth, no contact, no strain limit reached: inertia, membrane k |F - R|^2, pin springs
    sc, x, v = hanging(case["n"], seed)
    m = sc.material
    dt = sc.params["dt"]
    area, dm = abi.rest_state(sc.vertices, sc.triangles)
    mass = abi.lumped_masses(len(x), sc.triangles, area, m["thickness"], m["density"])
    mu = m["youngs_modulus"] / (2.0 * (1.0 + m["poisson_ratio"]))
    k = area * m["thickness"] * mu
    T = sc.triangles.astype(np.int64)
    D = np.stack([x[T[:, 1]] - x[T[:, 0]], x[T[:, 2]] - x[T[:, 0]]], axis=2)      # T x 3 x 2
    Dm = dm.reshape(-1, 2, 2)
    F = D @ Dm
    U, sig, Vt = np.linalg.svd(F, full_matrices=False)
    assert sig.max() < 1.0 + sc.params["strain_tau"]
    P = 2.0 * k[:, None, None] * (F - U @ Vt)
    G = np.concatenate([-(Dm[:, :1] + Dm[:, 1:]), Dm], axis=1)                    # T x 3 x 2: rows of vertices 0, 1, 2
    g = np.zeros_like(x)
    diag = mass / dt ** 2
    H = 2.0 * k[:, None, None] * (G @ G.transpose(0, 2, 1))
    el = np.zeros(len(x))
    for a in range(3):
        np.add.at(g, T[:, a], np.einsum("tij,tj->ti", P, G[:, a]))
        np.add.at(el, T[:, a], H[:, a, a])
    g += (mass / dt ** 2)[:, None] * (x - (x + dt * v))
    pin = np.zeros(len(x))
    for i, t in sc.pins:
        kp = 100.0 * (mass[i] / dt ** 2 + el[i])
        g[i] += kp * (x[i] - np.asarray(t))
        pin[i] += kp
    V = len(x)
    key = (T[:, :, None] * V + T[:, None, :]).reshape(-1)
    uniq, inv = np.unique(np.concatenate([key, np.arange(V) * (V + 1)]), return_inverse=True)
    c = np.zeros(len(uniq))
    np.add.at(c, inv, np.concatenate([H.reshape(-1), diag + pin]))
    return {"gradient": g.reshape(-1), "rowptr": None, "cols": None, "vals": c[:, None, None] * np.eye(3), "rhs": -g.reshape(-1)}


# -------------------------------------------------------------------------------------------- work
# Newton iterations of a frame and PCG iterations of one, as measured on scenes of these kinds: a frame's least work depends
# on them
NEWTON, PCG = 6, 70


def work(case):
    """Bytes that a pass cannot do without: its inputs and outputs once; for a solve the matrix once (later iterations may
    find it on the chip) and the vectors' updates; for a frame that many Newton systems, solves and contact passes."""
    kind = case["kind"]
    if kind == "pcg":
        V = case["nx"] * case["ny"]
        return {"bytes": 40.0 * 7 * V + 24.0 * V, "flops": 60.0 * (18.0 * 7 * V + 30.0 * V)}
    if kind == "frame_batch":
        n = 0.5 * (case["lo"] + case["hi"])
        V = case["scenes"] * n * n
    else:
        V = case["n"] ** 2 * {"frame_stack": case.get("sheets", 1), "contacts": case.get("sheets", 1), "frame_curtains": 2,
                              "broad_phase": case.get("sheets", 1), "precond_eval": 2, "train_gradient": 2}.get(kind, 1)
    system = V * (7 * 36 + 7 * 16 + 72 + 48)                     # blocks out, elastic constants, diagonal terms, factors
    if kind == "frame_reference":
        return {"bytes": float(V * 144 + 2 * system), "flops": float(2 * V * 7 * 40)}
    if kind.startswith("frame"):
        return {"bytes": float(V * 144 + NEWTON * (system + V * 300)), "flops": float(NEWTON * (PCG * V * 156 + V * 2000))}
    if kind == "contacts":
        return {"bytes": float(V * 48 + 6 * V * 208), "flops": float(6 * V * 200)}
    if kind == "broad_phase":
        return {"bytes": float(V * 24 + 3 * V * (8 + 4 * 8)), "flops": float(3 * V * 4 * 20)}
    if kind == "newton_system":
        return {"bytes": float(system + V * 100), "flops": float(V * 2000)}
    dense = 2.0 * V * (8 * 64 + 3 * (64 * 64 + 128 * 64) + 3 * 6 * 64 * 10)
    if kind == "precond_eval":
        return {"bytes": float(2 * system + V * 7 * 36), "flops": dense}
    return {"bytes": float(V * 7 * 80 + V * 64 * 4 * 14), "flops": 3.0 * dense}
