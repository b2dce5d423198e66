"""Performance cases of the projective-dynamics step, its adjoint and the learned warm start.

Each case is a plain dict.  `prepare` builds what a program holds before the call (the deformable with its factor on
the GPU, the state, the network), `run` makes one pass through the public entry points, `work` counts the bytes and
operations that pass cannot do without and `exact` gives the 64-bit values where they have a closed form.

Kinds (the field "kind"):
  mlp_infer   warm-start network inference over the nodes of a mesh (`WarmStartMLP.forward`), BF16 in, FP32 out
  mlp_train   one AdamW step on a mini-batch (`WarmStartMLP.train_step`), FP32 weights and moments updated in place
  ainv        x = A^-1 b through the allocation-free C entry point, FP64 or FP32
  host_step   `PyForward` then `PyBackward` on host arrays with the reference's options (what `EnvBase.simulate` calls)
  forward     one `forward_device` step without contact
  adjoint     one `backward_device` step without contact (conjugate gradients)
  contact     one `forward_device` step of a block that touches the ground, and with "adjoint" its `backward_device`
  rollout     `Rollout.apply` over a few steps and its backward pass: gradients for q0, v0, parameters and forces

Meshes, materials and step sizes are those of `diffphd_b200.scenes`.  The states are seeded smooth deformations and
velocities of the rest shape (a body in motion), or the block's first contact with the ground.  A program in mixed
precision ("precision": "mixed", the option fp32_bulk) keeps its states and gradients as FP32 tensors.
"""
import ctypes as C
import math

import numpy as np
import torch

from diffphd_b200 import core, scenes
from diffphd_b200.autograd import DiffSim, Rollout
from diffphd_b200.warmstart import WarmStartMLP

METHOD = "pd_eigen_alg_phd"
N_IN, N_HID, N_OUT, N_USED = 16, 128, 8, 4
MLP_STEP, MLP_LR, MLP_DECAY = 1000, 1e-3, 1e-5


def listed():
    return [
        # one frame's inference on the cantilever's 425 nodes: a call in a real-time loop, where launches count
        {"name": "mlp_infer_425", "kind": "mlp_infer", "rows": 425},
        # one frame's inference on the 64^3 block's 274,625 nodes
        {"name": "mlp_infer_274625", "kind": "mlp_infer", "rows": 274625},
        # one step of `warmstart.fit` at its default batch
        {"name": "mlp_train_65536", "kind": "mlp_train", "rows": 65536},
        # the solve inside a caller's own time-stepping loop on the tet block, in the solver's double precision
        {"name": "ainv_tet_32x16x16", "kind": "ainv", "scene": "tet", "cells": "32x16x16", "precision": "f64"},
        # a step and its gradient on host vectors with the reference's defaults: the drop-in use on its small scene
        {"name": "host_step_cantilever_16x4x4", "kind": "host_step", "scene": "cantilever", "cells": "16x4x4"},
        # forward simulation of the heterogeneous Neo-Hookean block, gate tightened below the default
        {"name": "forward_tet_32x16x16", "kind": "forward", "scene": "tet", "cells": "32x16x16", "precision": "f64"},
        # a refined cantilever in mixed precision at the default gate, started from rest
        {"name": "forward_cantilever_48x24x24_mixed", "kind": "forward", "scene": "cantilever", "cells": "48x24x24",
         "precision": "mixed"},
        # a reverse-sweep step of a training loop on the tet block, mixed precision
        {"name": "adjoint_tet_32x16x16_mixed", "kind": "adjoint", "scene": "tet", "cells": "32x16x16",
         "precision": "mixed"},
        # the largest contact-free mesh: a factor of 224 M values, far beyond the L2 cache
        {"name": "adjoint_cantilever_64x32x32", "kind": "adjoint", "scene": "cantilever", "cells": "64x32x32",
         "precision": "f64"},
        # a rotated block meeting the ground with Coulomb friction, every node a contact candidate
        {"name": "contact_drop_16", "kind": "contact", "scene": "drop", "cells": "16x16x16", "precision": "f64",
         "adjoint": False},
        # the same at the configured 24^3, a step and its contact-aware gradient in mixed precision
        {"name": "contact_drop_24_mixed_grad", "kind": "contact", "scene": "drop", "cells": "24x24x24",
         "precision": "mixed", "adjoint": True},
        # a training pass through the differentiable rollout on the small scene, recomputed from a checkpoint
        {"name": "rollout_cantilever_16x4x4", "kind": "rollout", "scene": "cantilever", "cells": "16x4x4",
         "steps": 3, "checkpoint": 2},
    ]


def draw(rng):
    kind = rng.choice(["mlp_infer", "mlp_train", "ainv", "host_step", "forward", "forward", "adjoint", "adjoint",
                       "contact", "rollout"])
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    if kind == "mlp_infer":
        return {"kind": kind, "rows": log(64, 274625)}
    if kind == "mlp_train":
        return {"kind": kind, "rows": log(1000, 65536)}
    if kind == "contact":
        c = log(6, 20)
        return {"kind": kind, "scene": "drop", "cells": "%dx%dx%d" % (c, c + rng.randint(-1, 1), c),
                "precision": rng.choice(["f64", "mixed"]), "adjoint": rng.random() < 0.5}
    if kind in ("host_step", "rollout"):
        case = {"kind": kind, "scene": "cantilever", "cells": "%dx%dx%d" % (log(6, 16), log(2, 5), log(2, 5))}
        return dict(case, steps=rng.randint(1, 2), checkpoint=rng.randint(1, 2)) if kind == "rollout" else case
    scene = rng.choice(["tet", "cantilever"])
    if scene == "tet" or kind == "ainv":
        cells = (log(8, 32), log(4, 16), log(4, 16))
    else:
        cells = (log(16, 60), log(6, 30), log(6, 30))
    precision = rng.choice(["f64", "mixed"])
    if kind == "forward" and scene == "tet":
        precision = "f64"
    return {"kind": kind, "scene": scene, "cells": "%dx%dx%d" % cells, "precision": precision}


def _cells(case):
    return tuple(int(c) for c in case["cells"].split("x"))


def _scene(case, seed):
    if case["scene"] == "tet":
        return scenes.nh_tet_block(cells=_cells(case), seed=seed)
    if case["scene"] == "drop":
        return scenes.contact_drop(cells=_cells(case), seed=seed, height=0.0)
    return scenes.cantilever(cells=_cells(case), seed=seed, heterogeneous=True)


def _smooth(verts, rng, amplitude):
    """A smooth random vector field over the body: a few sine waves of about its own length."""
    x = verts - verts.min(axis=0)
    u = np.zeros_like(verts)
    for _ in range(4):
        k, phase, a = 2.0 / x.max() * rng.normal(size=3), rng.uniform(0, 2 * math.pi), rng.normal(size=3)
        u += np.sin(x @ k + phase)[:, None] * a
    return amplitude * u / 4


def _state(scene, seed, at_rest=False):
    """Positions and velocities of the body in motion (zero motion at a clamped end)."""
    rng = np.random.default_rng(seed)
    q, v = scene.q0.reshape(-1, 3).copy(), np.zeros((scene.n, 3))
    if scene.plane is not None:
        v[:, 2] = -rng.uniform(0.3, 0.6)
    elif not at_rest:
        x = scene.verts[:, :1] - scene.verts[:, :1].min()
        q += _smooth(scene.verts, rng, 0.0005) * x / x.max()
        v = _smooth(scene.verts, rng, 0.1) * x / x.max()
    return q.ravel(), v.ravel()


def _options(case, scene):
    """The scene's own options (1e-6 gate, Anderson window 5); what a case adds to them."""
    o = dict(scene.options, verbose=-1)
    if case.get("precision") == "mixed":
        o["fp32_bulk"] = 1
    if case["kind"] == "adjoint":
        o.update(alg_phd_bwd_solver=1, rel_tol=1e-11 if case["precision"] == "f64" else 1e-8, abs_tol=1e-14)
    elif case["kind"] == "contact":
        o.update(alg_phd_bwd_solver=1, rel_tol=1e-8 if case["adjoint"] else 1e-7)
    elif case["kind"] == "forward" and case["precision"] == "f64":
        o.update(rel_tol=1e-8)
    return o


def _gpu(a):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _mlp_weights(seed):
    """Flat FP32 weights (W1, W2, W3, biases) of a network in mid-training."""
    g = torch.Generator().manual_seed(seed)
    n = lambda *s: torch.randn(*s, generator=g, dtype=torch.float64)
    w1, w2, w3 = n(N_IN, N_HID) * (2 / N_IN) ** 0.5, n(N_HID, N_HID) * (2 / N_HID) ** 0.5, n(N_HID, N_OUT) * 0.03
    w1[15:], w3[:, N_USED:] = 0, 0
    return torch.cat([w1.ravel(), w2.ravel(), w3.ravel(), 0.05 * n(2 * N_HID), torch.zeros(N_OUT)]).float()


def _mlp_rows(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = 0.5 * torch.randn(case["rows"], N_IN, generator=g, device="cuda")
    x[:, 15] = 0
    y = 0.1 * torch.randn(case["rows"], N_USED, generator=g, device="cuda")
    return x.to(torch.bfloat16), y


def _moments(seed):
    g = torch.Generator().manual_seed(seed + 1)
    n = _mlp_weights(seed).numel()
    return 1e-4 * torch.randn(n, generator=g), 1e-6 * (0.5 + torch.rand(n, generator=g))


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("mlp_infer", "mlp_train"):
        mlp = WarmStartMLP("cuda", seed=seed)
        mlp.load_master(_mlp_weights(seed))
        x, y = _mlp_rows(case, seed)
        if kind == "mlp_train":
            m, v = _moments(seed)
            mlp.m.copy_(m)
            mlp.v.copy_(v)
            mlp.step_count = MLP_STEP
        return {"case": case, "mlp": mlp, "x": x, "y": y}
    scene = _scene(case, seed)
    options = _options(case, scene)
    at_rest = kind == "forward" and case["precision"] == "mixed"
    q, v = _state(scene, seed, at_rest)
    rng = np.random.default_rng(seed + 2)
    gq, gv = rng.standard_normal(scene.dofs), 0.01 * rng.standard_normal(scene.dofs)
    s = {"case": case, "dt": scene.dt, "options": options}
    if kind == "rollout":
        s["sim"] = DiffSim(scene, options)
        s["params"] = s["sim"].default_params().to("cuda")
        d = s["sim"].deformable(s["params"].cpu().numpy())
    else:
        d = core.from_scene(scene)
    s["d"] = d
    if kind == "host_step":
        f = np.zeros(scene.dofs)
        s.update(q=q, v=v, f=f, gq=gq, gv=gv, scene=scene)
        d.PyForward(METHOD, q, v, [], f, scene.dt, dict(options, max_pd_iter=1), q.copy(), v.copy(), [])
        return s
    s.update(q=_gpu(q), v=_gpu(v), f=torch.zeros(scene.dofs, dtype=torch.float64, device="cuda"), gq=_gpu(gq),
             gv=_gpu(gv), b=_gpu(rng.standard_normal(scene.dofs)))
    # the handle of a running simulation: its factor, buffers and captured loops exist
    out = [torch.empty_like(s["q"]) for _ in range(3)]
    d.forward_device(METHOD, s["q"], s["v"], s["f"], scene.dt, dict(options, max_pd_iter=1), out[0], out[1],
                     stream=_stream())
    if kind == "adjoint":
        d.backward_device(METHOD, s["q"], s["gq"], s["gv"], scene.dt, dict(options, max_pd_iter=1), *out,
                          stream=_stream())
        d.reset_warm_start()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "mlp_infer":
        return s["mlp"].forward(s["x"])
    if kind == "mlp_train":
        mlp = s["mlp"]
        loss = mlp.train_step(s["x"], s["y"], MLP_LR, weight_decay=MLP_DECAY)
        return {"loss": loss, "weights": mlp.master, "m": mlp.m, "v": mlp.v, "packed": mlp.packed}
    d, dt, options = s["d"], s["dt"], s["options"]
    f32 = case.get("precision") == "mixed"
    as_kept = (lambda ts: [t.to(torch.float32) for t in ts]) if f32 else list
    if kind == "ainv":
        x = torch.empty_like(s["b"])
        lib = core.load_library()
        core.Deformable._check(lib.dphd_ainv_noalloc(d._h, dt, C.c_void_p(s["b"].data_ptr()),
                                                     C.c_void_p(x.data_ptr()), int(f32), C.c_void_p(_stream())))
        return as_kept([x])
    if kind == "host_step":
        n = s["q"].size
        qn, vn, active = np.zeros(n), np.zeros(n), []
        d.PyForward(METHOD, s["q"], s["v"], [], s["f"], dt, options, qn, vn, active)
        dq, dv, df = np.zeros(n), np.zeros(n), np.zeros(n)
        dw, dp = np.zeros(d.NumOfPdElementEnergies()), np.zeros(d.NumOfStateForceParameters())
        d.PyBackward(METHOD, s["q"], s["v"], [], s["f"], dt, qn, vn, active, s["gq"], s["gv"], options, dq, dv, [],
                     df, dw, [], dp)
        return [qn, vn, dq, dv, df, dw, dp]
    if kind == "rollout":
        leaves = [s[k].detach().requires_grad_(True) for k in ("q", "v", "params", "f")]
        q, v = Rollout.apply(s["sim"], *leaves, case["steps"], case["checkpoint"])
        ((q * s["gq"]).sum() + (v * s["gv"]).sum()).backward()
        return [q.detach(), v.detach()] + [t.grad for t in leaves]
    stream = _stream()
    new = lambda: torch.empty_like(s["q"])
    q_next, v_next = new(), new()
    out = []
    if kind in ("forward", "contact"):
        d.reset_warm_start()  # a new rollout from this state
        d.forward_device(METHOD, s["q"], s["v"], s["f"], dt, options, q_next, v_next, stream=stream)
        out = [q_next, v_next]
    if kind == "adjoint" or case.get("adjoint"):
        dq, dv, df = new(), new(), new()
        dp = torch.empty(d.NumOfPdParams(), dtype=torch.float64, device="cuda")
        d.backward_device(METHOD, out[0] if out else s["q"], s["gq"], s["gv"], dt, options, dq, dv, df,
                          dl_dparams=dp, stream=stream)
        out += [dq, dv, df, dp]
    return as_kept(out)


def work(case):
    """Inputs, outputs and the mesh once; for the solves one read of the sparse-inverse factor and one local step."""
    kind = case["kind"]
    if kind in ("mlp_infer", "mlp_train"):
        rows = case["rows"]
        macs = N_IN * N_HID + N_HID * N_HID + N_HID * N_USED
        if kind == "mlp_infer":
            return {"bytes": rows * (2 * N_IN + 4 * N_OUT) + 2 * macs, "flops": 2.0 * macs * rows}
        return {"bytes": rows * (2 * N_IN + 4 * N_USED) + 26.0 * macs, "flops": 6.0 * macs * rows}
    a, b, c = _cells(case)
    n, m, tet = (a + 1) * (b + 1) * (c + 1), a * b * c, case["scene"] == "tet"
    m, k, samples = (5 * m, 4, 1) if tet else (m, 8, 8)
    item = 4 if case.get("precision") == "mixed" else 8
    factor = 1.3 * n ** 1.7  # values of the nested-dissection factor of a box of n nodes
    vectors = {"ainv": 2, "host_step": 10, "forward": 5, "adjoint": 6, "contact": 11 if case.get("adjoint") else 5,
               "rollout": 9}[kind] * 3 * n * 8
    passes = 2 if kind in ("host_step", "rollout") or case.get("adjoint") else 1
    elements = 0 if kind == "ainv" else m * (4 * k + 24)
    local = 0 if kind == "ainv" else 600.0 * m * samples
    steps = case.get("steps", 1)
    return {"bytes": steps * (vectors + passes * (elements + factor * item)),
            "flops": steps * passes * (local + 12 * factor)}


# ---- 64-bit values --------------------------------------------------------------------------------------------
def _mlp_parts(flat):
    sizes = [N_IN * N_HID, N_HID * N_HID, N_HID * N_OUT, N_HID, N_HID, N_OUT]
    w1, w2, w3, b1, b2, b3 = torch.split(flat, sizes)
    return w1.view(N_IN, N_HID), w2.view(N_HID, N_HID), w3.view(N_HID, N_OUT), b1, b2, b3


def _mlp_forward(x, w1, w2, w3, b1, b2, b3):
    gelu = torch.nn.functional.gelu
    return gelu(gelu(x @ w1 + b1) @ w2 + b2) @ w3 + b3


def _exact_mlp(case, seed):
    flat = _mlp_weights(seed).to("cuda")
    x, y = _mlp_rows(case, seed)
    x, y, weights = x.double(), y.double(), flat.double()
    parts = [p.clone().requires_grad_(True) if i > 2 else p.to(torch.bfloat16).double().requires_grad_(True)
             for i, p in enumerate(_mlp_parts(weights))]  # the matrices are BF16 operands
    out = _mlp_forward(x, *parts)
    if case["kind"] == "mlp_infer":
        return out.detach()
    loss = ((out[:, :N_USED] - y) ** 2).sum() / case["rows"]
    loss.backward()
    used = [torch.ones_like(p) for p in parts]
    used[0][15:], used[2][:, N_USED:], used[5][N_USED:] = 0, 0, 0
    grad = torch.cat([(p.grad * u).ravel() for p, u in zip(parts, used)])
    used = torch.cat([u.ravel() for u in used]) > 0
    m0, v0 = (t.to("cuda").double() for t in _moments(seed))
    m, v = torch.where(used, 0.9 * m0 + 0.1 * grad, m0), torch.where(used, 0.999 * v0 + 0.001 * grad ** 2, v0)
    step = MLP_STEP + 1
    decay = torch.arange(weights.numel(), device="cuda") < N_IN * N_HID + N_HID * N_HID + N_HID * N_OUT
    new = weights * torch.where(decay, 1 - MLP_LR * MLP_DECAY, 1.0)
    new = new - MLP_LR * (m / (1 - 0.9 ** step)) / ((v / (1 - 0.999 ** step)).sqrt() + 1e-8)
    return {"loss": loss.detach().reshape(1), "weights": torch.where(used, new, weights), "m": m, "v": v,
            "packed": None}


def _exact_ainv(case, seed):
    """Dense Cholesky solve with A = diag(m/h^2, 1 on clamped nodes) + sum_e w_e V/s sum_s G_s G_s^T."""
    scene = _scene(case, seed)
    verts, elems = _gpu(scene.verts), torch.as_tensor(scene.elems, device="cuda").long()
    corner = verts[elems]
    edges = corner[:, [1, 2, 3] if case["scene"] == "tet" else [1, 2, 4]] - corner[:, :1]
    volume = (torch.linalg.det(edges).abs() / (6 if case["scene"] == "tet" else 1)).mean()
    if case["scene"] == "tet":
        inv = torch.linalg.inv(edges.transpose(1, 2))
        grads = torch.cat([-inv.sum(dim=1, keepdim=True), inv], dim=1)[None]  # one sample: (1, m, 4, 3)
        stiffness = _gpu(scene.energies[0][1]).view(-1, 2)[:, 0] * 2
    else:
        h = float(volume) ** (1 / 3)
        g = torch.zeros(8, 8, 3, dtype=torch.float64)
        for s in range(8):
            p = [((s >> 2 - d & 1) - 0.5) / math.sqrt(3) + 0.5 for d in range(3)]
            for a in range(8):
                bit = [a >> 2 - d & 1 for d in range(3)]
                lin = [p[d] if bit[d] else 1 - p[d] for d in range(3)]
                for d in range(3):
                    g[s, a, d] = (1 if bit[d] else -1) / h * math.prod(lin[e] for e in range(3) if e != d)
        grads = g.to("cuda")[:, None]  # the same for every element
        stiffness = sum(_gpu(p) for _, p, _ in scene.energies)
    block = torch.einsum("smad,smbd->mab", grads, grads) * (stiffness * volume / grads.shape[0])[:, None, None]
    n = scene.n
    A = torch.zeros(n * n, dtype=torch.float64, device="cuda")
    rows = (elems[:, :, None] * n + elems[:, None, :]).ravel()
    A.index_add_(0, rows, block.expand(len(elems), -1, -1).ravel())
    A = A.view(n, n)
    A.diagonal().add_(scene.density * volume / scene.dt ** 2)
    fixed = torch.as_tensor(np.unique(scene.dirichlet_dofs // 3), device="cuda")
    A[fixed], A[:, fixed] = 0, 0
    A[fixed, fixed] = 1
    rng = np.random.default_rng(seed + 2)
    rng.standard_normal(scene.dofs), rng.standard_normal(scene.dofs)
    b = _gpu(rng.standard_normal(scene.dofs)).view(n, 3)
    b[fixed] = 0
    return [torch.cholesky_solve(b, torch.linalg.cholesky(A)).ravel()]


def exact(case, seed):
    if case["kind"] in ("mlp_infer", "mlp_train"):
        return _exact_mlp(case, seed)
    if case["kind"] == "ainv":
        return _exact_ainv(case, seed)
    return None  # the steps stop at their gate, not at a solution with a closed form
