"""The work a user of d2ic_gb300 has it do, as timed cases through the package's public entry points.

A case is a dict of plain values: its ``kind`` names the entry point, the rest its sizes and options.

* ``frame``      one frame through ``DICMeshBased.run`` (global CG, strain, results on the host)
* ``objective``  ``GlobalCGSolver.objective_and_gradient``: one value and gradient, for a caller's own optimiser
* ``sequence``   ``BatchMeshBased.sequence`` with chained local refinement and constant-velocity warm starts
* ``batch``      ``solve_batch``: independent frames of uneven size in one launch
* ``serve``      ``DICServer``: frames of several sequences, continuous batching
* ``init``       ``DICInitMotion.run``: ZNCC at the element centres, projected onto the nodes
* ``refine``     ``DICMeshBased.run`` with ``LocalGaussNewtonSolver`` and the discrepancy map
* ``jvp``        noise propagation: ``ImplicitAdjoint.jvp`` of K images and the strain sensitivity
* ``vjp``        ``ImplicitAdjoint.vjp`` of K nodal cotangents (image-space sensitivity maps)
* ``step``       ``DifferentiableSolve``: forward solve and backward pass of one image

Images are seeded Gaussian-dot speckle (dots at about one per 12 pixels, grey levels 20 to 230, camera
noise) under a random affine map per seed; mesh and mask are fixed by the case.  ``exact`` restates
each path in 64-bit torch.
"""
from __future__ import annotations

import math
from dataclasses import replace

import numpy as np
import torch

import d2ic_gb300 as d2
from d2ic_gb300.adjoint import DifferentiableSolve, ImplicitAdjoint, strain_jvp
from d2ic_gb300.engine import FrameLayout, FrameSlot
from d2ic_gb300.pixel_assets import build_pixel_assets_device
from d2ic_gb300.serving import DICServer, Request, ServeConfig, solve_batch
from d2ic_gb300.synthetic import Affine, speckle_sequence_device

DEV = "cuda"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # a single small frame from zero motion: the smallest solve, bound by the latency of a CG round
        dict(name="frame_512_cold", kind="frame", height=512, width=512, element=16, mask="rect", interp="cubic",
             pixels="f32", start="cold", max_iters=200, tol=1e-3, reg=0.1),
        # the plate-with-hole sequence's frame, warm-started from the frame before (the headline benchmark)
        dict(name="frame_2048_plate", kind="frame", height=2048, width=2048, element=16, mask="plate", interp="cubic",
             pixels="f32", start="warm", max_iters=200, tol=1e-3, reg=0.1),
        # the largest camera frames at the finest mesh: 8-bit pixels, 8-px elements, the default iteration cap
        dict(name="frame_4096_fine_u8", kind="frame", height=4096, width=4096, element=8, mask="ellipse",
             interp="cubic", pixels="u8", start="warm", max_iters=50, tol=1e-3, reg=0.1),
        # one evaluation for a caller's own optimiser, bilinear option, odd image and element sizes
        dict(name="objective_linear_odd", kind="objective", height=737, width=1111, element=23, mask="ellipse",
             interp="linear", reg=0.1),
        # the reference's published benchmark: 11 frames of 1040 x 400, 15-px elements, CG at tol 1e-2
        # and reg 0.5, three local refinement sweeps per frame, constant-velocity warm start
        dict(name="sequence_1040x400", kind="sequence", height=400, width=1040, element=15, mask="plate",
             interp="cubic", frames=11, sweeps=3, max_iters=400, tol=1e-2, reg=0.5),
        # independent frames of uneven size, element size and mask in one launch
        dict(name="batch_12_uneven", kind="batch", frames=12, low=512, high=2048, mix=2, interp="cubic", max_iters=200,
             tol=1e-3, reg=0.1),
        # requests of several small sequences, each started by ZNCC, then warm-started
        dict(name="serve_8x3_small", kind="serve", sequences=8, frames=3, low=384, high=768, mix=4, interp="cubic",
             max_iters=200, tol=1e-3, reg=0.1),
        # initial motion of a first frame with the configuration's default window and search range
        dict(name="init_1536_default", kind="init", height=1536, width=1536, element=16, mask="plate", win=41,
             search=24, reach=20),
        # local refinement of a converged frame and its discrepancy map
        dict(name="refine_2048", kind="refine", height=2048, width=2048, element=16, mask="plate", interp="cubic",
             sweeps=3, reg=0.1),
        # uncertainty propagation: 64 noise images at once, displacement and strain sensitivities
        dict(name="jvp_1024_64", kind="jvp", height=1024, width=1024, element=12, mask="rect", images=64, reg=0.1),
        # image-space sensitivity maps of six nodal functionals, odd sizes
        dict(name="vjp_777x901_6", kind="vjp", height=777, width=901, element=13, mask="ellipse", images=6, reg=0.1),
        # one forward and backward pass of the solve as a differentiable function
        dict(name="step_512", kind="step", height=512, width=512, element=16, mask="rect", max_iters=200, tol=1e-3,
             reg=0.1, polish=3),
    ]


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "objective", "sequence", "batch", "serve", "init", "refine", "jvp",
                       "vjp", "step"])

    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def image(lo, hi):
        h = log_int(lo, hi)
        return dict(height=h, width=min(hi, max(lo, int(round(h * rng.uniform(0.6, 1.6))))),
                    mask=rng.choice(["rect", "plate", "ellipse"]))

    interp = rng.choice(["cubic", "cubic", "cubic", "linear"])
    if kind == "frame":
        return dict(kind=kind, **image(320, 2800), element=rng.randint(8, 32), interp=interp,
                    pixels=rng.choice(["f32", "u8"]), start=rng.choice(["cold", "warm"]),
                    max_iters=rng.choice([50, 200]) if interp == "cubic" else 50, tol=1e-3, reg=0.1)
    if kind == "objective":
        return dict(kind=kind, **image(192, 4000), element=rng.randint(7, 40), interp=interp, reg=0.1)
    if kind == "sequence":
        return dict(kind=kind, **image(320, 1200), element=rng.randint(10, 24), interp=interp,
                    frames=rng.randint(3, 11), sweeps=rng.randint(1, 4), max_iters=400, tol=1e-2, reg=0.5)
    if kind == "batch":
        return dict(kind=kind, frames=rng.randint(2, 12), low=400, high=log_int(512, 2048), mix=rng.randint(10, 10 ** 6),
                    interp="cubic", max_iters=200, tol=1e-3, reg=0.1)
    if kind == "serve":
        return dict(kind=kind, sequences=rng.randint(2, 8), frames=rng.randint(1, 3), low=320, high=log_int(400, 768),
                    mix=rng.randint(10, 10 ** 6), interp="cubic", max_iters=200, tol=1e-3, reg=0.1)
    if kind == "init":
        search = rng.randint(4, 24)
        return dict(kind=kind, **image(256, 1200), element=rng.randint(12, 40), win=2 * rng.randint(5, 20) + 1,
                    search=search, reach=search - 2)
    if kind == "refine":
        return dict(kind=kind, **image(256, 2048), element=rng.randint(8, 32), interp=interp, sweeps=rng.randint(1, 5),
                    reg=rng.choice([0.1, 0.5]))
    if kind == "jvp":
        return dict(kind=kind, **image(256, 1024), element=rng.randint(10, 24), images=log_int(1, 64), reg=0.1)
    if kind == "vjp":
        return dict(kind=kind, **image(256, 900), element=rng.randint(10, 24), images=rng.randint(1, 6), reg=0.1)
    return dict(kind="step", **image(256, 640), element=rng.randint(12, 24), max_iters=200, tol=1e-3, reg=0.1,
                polish=rng.randint(1, 3))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _mask(height, width, shape):
    """Region of interest: a centred rectangle, the same with a central hole, or an ellipse."""
    y = (np.arange(height)[:, None] + 0.5 - height / 2) / height
    x = (np.arange(width)[None, :] + 0.5 - width / 2) / width
    if shape == "ellipse":
        return (x / 0.47) ** 2 + (y / 0.43) ** 2 <= 1.0
    inside = (np.abs(x) <= 0.44) & (np.abs(y) <= 0.44)
    if shape == "plate":
        side = min(height, width)
        inside &= (x * width) ** 2 + (y * height) ** 2 >= (0.146 * side) ** 2
    return inside


def _geometry(case):
    """Mesh and assets of a case's image size, element size and mask."""
    H, W = case["height"], case["width"]
    mesh, assets = d2.mask_to_mesh_assets(_mask(H, W, case["mask"]), case["element"])
    return mesh, replace(assets, pixel_data=build_pixel_assets_device(mesh, np.empty((H, W), np.uint8), 1.0,
                                                                      assets.roi_mask))


def _motion(height, width, seed, frames):
    """Affine maps of ``frames`` consecutive frames: strains to 1%, rotation to 0.5 degrees (less on
    large images) and a translation to 3 px are reached over 20 frames; the first one shown is frame 12 of
    that load path.  Also returns the map of the frame before."""
    r = np.random.default_rng(seed)
    side = max(height, width)
    exx, eyy, exy = r.uniform(-0.01, 0.01, 3) * min(1.0, 2048 / side)
    th = math.radians(r.uniform(-0.5, 0.5)) * min(1.0, 1024 / side)
    A = np.array([[exx, exy - th], [exy + th, eyy]])
    t = r.uniform(-3.0, 3.0, 2)
    x0 = [width / 2, height / 2]
    return [Affine(A * k / 20.0, t * k / 20.0, x0) for k in range(12, 12 + frames)], Affine(A * 11 / 20, t * 11 / 20, x0)


def _approach(height, width, seed, frames, reach):
    """Maps of a specimen that is shifted as a whole by up to ``reach`` pixels before its first frame and
    strained a little more from frame to frame (a fixture takes up its play, then the load comes on)."""
    r = np.random.default_rng(seed)
    A = r.uniform(-1.5e-3, 1.5e-3, (2, 2)) * min(1.0, 512 / max(height, width))
    t = r.integers(-reach, reach + 1, 2) + r.uniform(-0.15, 0.15, 2)
    return [Affine(A * (k + 1), t, [width / 2, height / 2]) for k in range(frames)]


def _images(height, width, warps, seed, pixels, noise=1.0):
    ref, frames = speckle_sequence_device(height, width, warps, seed=seed, noise_seeds=[1000 * seed + k for k in
                                          range(len(warps) + 1)], noise_sigma=noise, device=DEV, u8=pixels == "u8")
    return ref, frames


def _nodal(warp, nodes):
    """The map's displacement at the nodes, (Nn, 2) float32: what the previous frame's solve left."""
    xy = torch.as_tensor(np.asarray(nodes, np.float64))
    return warp.displacement(xy).to(torch.float32).numpy()


def _cold_warp(height, width, seed):
    """A first frame's small motion: subpixel translation, strains to 0.3% of a 512-px image's."""
    r = np.random.default_rng(seed)
    A = r.uniform(-0.003, 0.003, (2, 2)) * min(1.0, 512 / max(height, width))
    return Affine(A, r.uniform(-0.7, 0.7, 2), [width / 2, height / 2])


def _config(case, **kw):
    return d2.MeshDICConfig(max_iters=case.get("max_iters", 1), tol=case.get("tol", 1e-3), reg_strength=case["reg"],
                            **kw)


def _mix(case, count):
    """Image side, element size and mask of each member of a batch or stream, fixed by the case."""
    r = np.random.default_rng(case["mix"])
    out = []
    for _ in range(count):
        h, w = (int(round(math.exp(r.uniform(math.log(case["low"]), math.log(case["high"]))))) for _ in range(2))
        w = int(min(case["high"], max(case["low"], w, 0.6 * h)))
        out.append(dict(height=h, width=w, element=int(r.choice([8, 12, 16, 24, 32])),
                        mask=str(r.choice(["ellipse", "ellipse", "plate"]))))
    return out


def _inputs(case, seed):
    """Images, mesh and starting displacement of a single-image case."""
    H, W = case["height"], case["width"]
    mesh, assets = _geometry(case)
    if case.get("start") == "cold":
        warps, before = [_cold_warp(H, W, seed)], None
    elif "reach" in case:
        warps, before = _approach(H, W, seed, case.get("frames", 1), case["reach"]), None
    else:
        warps, before = _motion(H, W, seed, case.get("frames", 1))
    ref, frames = _images(H, W, warps, seed, case.get("pixels", "f32"))
    u0 = None if before is None else _nodal(before, mesh.nodes_xy)
    return dict(mesh=mesh, assets=assets, ref=ref, frames=frames, u0=u0, warps=warps)


def _linearisation_point(p, seed):
    """A converged solution's stand-in: the true displacement plus noise of a solve's size."""
    u = _nodal(p["warps"][0], p["mesh"].nodes_xy)
    return u + np.random.default_rng(seed + 77).normal(0.0, 0.01, u.shape).astype(np.float32)


def _noise_images(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + 5)
    return 2.0 * torch.randn((case["images"], case["height"], case["width"]), generator=g, device=DEV)


def _cotangents(n_nodes, count, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + 6)
    return torch.randn((count, n_nodes, 2), generator=g, device=DEV)


# ---------------------------------------------------------------------------
# what a user's program has in hand, and one pass
# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind)
    if kind == "batch":
        frames = []
        for i, m in enumerate(_mix(case, case["frames"])):
            p = _inputs(m, 100 * seed + i)
            layout = FrameLayout(p["assets"].pixel_data, p["mesh"].nodes_xy.shape[0], p["ref"], case["interp"])
            frames.append((layout, p["frames"][0], torch.as_tensor(p["u0"], device=DEV), _config(case)))
        s["frames"] = frames
        return s
    if kind == "serve":
        server = DICServer(config=ServeConfig(max_slots=16), interpolation=case["interp"])
        s["images"] = []
        for i, m in enumerate(_mix(case, case["sequences"])):
            p = _inputs(dict(m, pixels="u8", frames=case["frames"], reach=1), 100 * seed + i)
            server.add_sequence(i, p["ref"], p["mesh"], p["assets"], _config(case),
                                init=d2.InitMotionConfig(win=17, search=8, score_min=0.2))
            s["images"].append(p["frames"])
        s["server"] = server
        return s
    if kind == "init":
        p = _inputs(case, seed)
        cfg = d2.InitMotionConfig(win=case["win"], search=case["search"])
        s["dic"] = d2.DICInitMotion(cfg, d2.TranslationZNCCSolver(cfg))
        s["dic"].prepare(p["ref"], p["assets"])
        s["image"] = p["frames"][0]
        return s
    p = _inputs(case, seed)
    mesh, assets = p["mesh"], p["assets"]
    s.update(image=p["frames"][0], u0=p["u0"])
    if kind == "sequence":
        idx, deg = d2.mesh_assets.build_node_neighbor_tables(mesh)
        assets = replace(assets, node_neighbor_index=idx, node_neighbor_degree=deg)
        cg = d2.DICMeshBased(mesh, d2.GlobalCGSolver(interpolation=case["interp"]), _config(case))
        local = d2.DICMeshBased(mesh, d2.LocalGaussNewtonSolver(interpolation=case["interp"]),
                                replace(_config(case), max_iters=case["sweeps"]))
        s["batch"] = d2.BatchMeshBased(p["ref"], assets, cg, d2.BatchConfig(), dic_local=local,
                                       propagator=d2.ConstantVelocityPropagator())
        s["batch"].before(p["frames"])
        s["cg"], s["images"] = cg, p["frames"]
    elif kind in ("frame", "objective", "step"):
        dic = d2.DICMeshBased(mesh, d2.GlobalCGSolver(interpolation=case.get("interp", "cubic")), _config(case))
        dic.prepare(p["ref"], assets)
        s["dic"] = dic
        if kind == "objective":
            s["u"] = p["u0"]
        if kind == "step":
            s["solve"] = DifferentiableSolve(dic.solver, dic.state, u0=p["u0"], polish=case["polish"])
            s["cotangent"] = _cotangents(mesh.nodes_xy.shape[0], 1, seed)[0]
    elif kind == "refine":
        s["dic"] = d2.DICMeshBased(mesh, d2.LocalGaussNewtonSolver(interpolation=case["interp"]),
                                   replace(_config(case), max_iters=case["sweeps"], compute_discrepancy_map=True))
        s["dic"].prepare(p["ref"], assets)
        s["u"] = _linearisation_point(p, seed)
    else:   # jvp, vjp
        layout = FrameLayout(assets.pixel_data, mesh.nodes_xy.shape[0], p["ref"], "cubic")
        slot = FrameSlot(layout, 1)
        slot.load_image(s["image"])
        s["u"] = torch.as_tensor(_linearisation_point(p, seed), device=DEV)
        s["adjoint"] = ImplicitAdjoint(slot, s["u"], case["reg"])
        if kind == "jvp":
            s["noise"] = _noise_images(case, seed)
            s["nodes"] = mesh.nodes_xy
            s["neighbours"] = d2.mesh_assets.build_node_neighbor_tables(mesh)
        else:
            s["cotangents"] = _cotangents(mesh.nodes_xy.shape[0], case["images"], seed)
    return s


def _frame_outputs(res):
    return dict(u=res.u_nodal, strain=res.strain, history=res.history, n_iters=res.diagnostics.info["n_iters"])


def run(s):
    kind = s["kind"]
    if kind == "frame":
        s["dic"].set_initial_guess(s["u0"])
        return _frame_outputs(s["dic"].run(s["image"]))
    if kind == "objective":
        J, g = s["dic"].solver.objective_and_gradient(s["dic"].state, s["image"], s["u"])
        return dict(J=J, g=g)
    if kind == "sequence":
        s["cg"].set_initial_guess(s["u0"])
        res = s["batch"].sequence(s["images"]).results
        return dict(u=[r.u_nodal for r in res], strain=[r.strain for r in res])
    if kind == "batch":
        res = solve_batch(s["frames"])
        return dict(u=[r[0] for r in res], history=[r[3] for r in res], n_iters=np.array([r[1] for r in res]))
    if kind == "serve":
        server = s["server"]
        server.reset_sequences()
        for k in range(len(s["images"][0])):
            for i, frames in enumerate(s["images"]):
                server.submit(Request(seq_id=i, frame_index=k, image=frames[k]))
        done = sorted(server.run_until_idle(), key=lambda r: (r.seq_id, r.frame_index))
        return dict(u=[r.u for r in done], strain=[r.strain for r in done], n_iters=np.array([r.n_iters for r in done]))
    if kind == "init":
        res = s["dic"].run(s["image"])
        return dict(u=res.u_nodal, matches=res.diagnostics.info["matches"])
    if kind == "refine":
        s["dic"].set_initial_guess(s["u"])
        res = s["dic"].run(s["image"])
        return dict(u=res.u_nodal, strain=res.strain, history=res.history, discrepancy=res.pixel_maps["discrepancy_ref"],
                    rms=res.diagnostics.info["discrepancy_rms"])
    if kind == "jvp":
        # kept in single precision, which is what the FP32 image terms carry
        du = s["adjoint"].jvp(s["noise"])
        strain = strain_jvp(s["u"], du, s["nodes"], *s["neighbours"])
        return dict(du=du.to(torch.float32), strain=strain.to(torch.float32))
    if kind == "vjp":
        return s["adjoint"].vjp(s["cotangents"])
    image = s["image"].detach().requires_grad_(True)
    u = s["solve"](image)
    (grad,) = torch.autograd.grad(u, image, s["cotangent"])
    return dict(u=u, grad=grad)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

SAMPLE_FLOPS = 110   # per pixel: 16 taps (value and two derivatives) and the weights (bicubic), the residual,
                     # the interpolated displacement and the four nodal partials


def _size(case):
    """Region-of-interest pixels, nodes and image bytes of a single-image case."""
    H, W, e = case["height"], case["width"], case["element"]
    np_ = int(_mask(H, W, case["mask"]).sum())
    nn = (math.ceil(H / e) + 1) * (math.ceil(W / e) + 1)
    return np_, nn, H * W * (1 if case.get("pixels") == "u8" else 4)


def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        parts = _mix(case, case.get("sequences", case["frames"]))
        n = case["frames"] if kind == "serve" else 1
        w = [work(dict(m, kind="frame", max_iters=case["max_iters"], pixels="u8" if kind == "serve" else "f32"))
             for m in parts]
        return dict(bytes=n * sum(x["bytes"] for x in w), flops=n * sum(x["flops"] for x in w))
    npx, nn, img = _size(case)
    records = 16 * npx                                   # position, reference value and local coordinates
    if kind in ("frame", "sequence"):
        n = case.get("frames", 1)
        iters = case["max_iters"] if kind == "frame" else 30 + case["sweeps"]
        return dict(bytes=n * (img + records + 40 * nn), flops=n * iters * SAMPLE_FLOPS * npx)
    if kind == "objective":
        return dict(bytes=img + records + 32 * nn, flops=SAMPLE_FLOPS * npx)
    if kind == "init":
        centres = npx / case["element"] ** 2
        offsets = (2 * case["search"] + 1) ** 2
        return dict(bytes=2 * img + 24 * nn, flops=centres * (2 * offsets * case["win"] ** 2 + 6 * nn))
    if kind == "refine":
        return dict(bytes=2 * img + records + 4 * case["height"] * case["width"] + 40 * nn,
                    flops=(2 * case["sweeps"] + 1) * SAMPLE_FLOPS * npx)
    if kind == "jvp":
        return dict(bytes=case["images"] * (img + 36 * nn) + records,
                    flops=case["images"] * (SAMPLE_FLOPS * npx + 25 * 100 * nn))
    if kind == "vjp":
        return dict(bytes=case["images"] * (img + 16 * nn) + records + img,
                    flops=case["images"] * (SAMPLE_FLOPS * npx + 25 * 100 * nn))
    return dict(bytes=2 * img + records + 40 * nn, flops=(60 + 4 * case["polish"] + 2) * SAMPLE_FLOPS * npx)


# ---------------------------------------------------------------------------
# the same paths in 64 bits (plain torch)
# ---------------------------------------------------------------------------

F64 = torch.float64
HALO = 40       # rows and columns of edge-extended coefficients around the image; |pole|^40 < 1e-22


def _coefficients(img):
    """Interpolating cubic B-spline coefficients of the edge-extended image, with a HALO border: the
    separable inverse of (1, 4, 1)/6, whose impulse response is sqrt(3) (sqrt(3) - 2)^|k|."""
    c = torch.nn.functional.pad(img.to(F64)[None, None], (2 * HALO,) * 4, mode="replicate")[0, 0]
    for dim in (0, 1):
        n = c.shape[dim] - 2 * HALO
        out = torch.zeros_like(c.narrow(dim, 0, n))
        for k in range(-HALO, HALO + 1):
            out = out + math.sqrt(3.0) * (math.sqrt(3.0) - 2.0) ** abs(k) * c.narrow(dim, HALO + k, n)
        c = out
    return c


def _weights(t):
    o = 1 - t
    return ([o ** 3 / 6, (3 * t ** 3 - 6 * t ** 2 + 4) / 6, (-3 * t ** 3 + 3 * t ** 2 + 3 * t + 1) / 6, t ** 3 / 6],
            [-o * o / 2, 1.5 * t * t - 2 * t, -1.5 * t * t + t + 0.5, t * t / 2],
            [o, 3 * t - 2, 1 - 3 * t, t])


def _cubic(c, x, y, second=False):
    """Value, d/dx, d/dy (and with ``second`` the Hessian) of the spline at index coordinates (x, y)."""
    ix, iy = torch.floor(x), torch.floor(y)
    wx, dx, ddx = _weights(x - ix)
    wy, dy, ddy = _weights(y - iy)
    flat, pitch = c.reshape(-1), c.shape[1]
    base = (iy.long() + HALO - 1) * pitch + ix.long() + HALO - 1
    out = [0.0] * (6 if second else 3)
    for a in range(4):
        taps = [flat[base + (a * pitch + b)] for b in range(4)]
        rv = sum(w * t for w, t in zip(wx, taps))
        rd = sum(w * t for w, t in zip(dx, taps))
        out[0], out[1], out[2] = out[0] + wy[a] * rv, out[1] + wy[a] * rd, out[2] + dy[a] * rv
        if second:
            rdd = sum(w * t for w, t in zip(ddx, taps))
            out[3], out[4], out[5] = out[3] + wy[a] * rdd, out[4] + dy[a] * rd, out[5] + ddy[a] * rv
    return out


def _linear(img, x, y):
    """Bilinear value and derivatives, indices clamped into the image."""
    H, W = img.shape
    ix, iy = torch.floor(x), torch.floor(y)
    tx, ty = x - ix, y - iy
    x0, x1 = ix.long().clamp(0, W - 1), (ix.long() + 1).clamp(0, W - 1)
    y0, y1 = iy.long().clamp(0, H - 1), (iy.long() + 1).clamp(0, H - 1)
    a, b, c, d = img[y0, x0], img[y0, x1], img[y1, x0], img[y1, x1]
    return [(1 - tx) * (1 - ty) * a + tx * (1 - ty) * b + (1 - tx) * ty * c + tx * ty * d,
            (1 - ty) * (b - a) + ty * (d - c), (1 - tx) * (c - a) + tx * (d - b)]


class _Problem:
    """The FE-DIC objective of one mesh and reference image in 64 bits."""

    def __init__(self, mesh, roi, ref, interp):
        self.interp = interp
        nodes, elements = np.asarray(mesh.nodes_xy, np.float64), np.asarray(mesh.elements, np.int64)
        gx, gy = np.unique(nodes[:, 0]), np.unique(nodes[:, 1])
        cell = np.full((gy.size - 1, gx.size - 1), -1, np.int64)
        cell[elements[:, 0] // gx.size, elements[:, 0] % gx.size] = np.arange(elements.shape[0])
        row, col = np.nonzero(roi)
        cx, cy = np.searchsorted(gx, col + 0.5) - 1, np.searchsorted(gy, row + 0.5) - 1
        ok = (cx >= 0) & (cy >= 0) & (cx < gx.size - 1) & (cy < gy.size - 1)
        row, col, cx, cy = row[ok], col[ok], cx[ok], cy[ok]
        ok = cell[cy, cx] >= 0
        row, col, cx, cy = row[ok], col[ok], cx[ok], cy[ok]
        T = lambda a: torch.as_tensor(a, device=DEV)  # noqa: E731
        xi = T(2 * (col + 0.5 - gx[cx]) / (gx[cx + 1] - gx[cx]) - 1)
        eta = T(2 * (row + 0.5 - gy[cy]) / (gy[cy + 1] - gy[cy]) - 1)
        self.shape = [(1 - xi) * (1 - eta) / 4, (1 + xi) * (1 - eta) / 4, (1 + xi) * (1 + eta) / 4,
                      (1 - xi) * (1 + eta) / 4]
        self.col, self.row = T(col).to(F64), T(row).to(F64)
        self.element = T(cell[cy, cx])
        self.el = T(elements)
        self.n, self.n_pix = nodes.shape[0], int(row.size)
        self.nodes = T(nodes)
        self.ref = ref.to(F64)
        self.i1 = self.ref[T(row), T(col)]
        pairs = np.unique(np.concatenate([elements[:, [a, b]] for a in range(4) for b in range(4) if a != b]), axis=0)
        self.src, self.dst = T(pairs[:, 0]), T(pairs[:, 1])
        self.w = 1 / (torch.linalg.norm(self.nodes[self.dst] - self.nodes[self.src], dim=1) + 1e-6)
        self.used = torch.zeros(self.n, dtype=torch.bool, device=DEV)
        self.used[self.el.reshape(-1)] = True

    def load(self, img):
        self.img = img.to(F64)
        self.samples = _coefficients(img) if self.interp == "cubic" else self.img

    def position(self, u):
        ue = u[self.el][self.element]
        dx = sum(n * ue[:, a, 0] for a, n in enumerate(self.shape))
        dy = sum(n * ue[:, a, 1] for a, n in enumerate(self.shape))
        return self.col + dx, self.row + dy

    def sample(self, c, u):
        x, y = self.position(u)
        return _cubic(c, x, y) if self.interp == "cubic" else _linear(c, x, y)

    def to_nodes(self, values):
        """Per local node a and value v: sum of N_a v over the pixels of each node, (Nn, len(values))."""
        out = torch.zeros((self.n, len(values)), dtype=F64, device=DEV)
        for a, n in enumerate(self.shape):
            per = torch.zeros((self.el.shape[0], len(values)), dtype=F64, device=DEV)
            per.index_add_(0, self.element, torch.stack([n * v for v in values], dim=1))
            out.index_add_(0, self.el[:, a], per)
        return out

    def springs(self, u):
        d = u[self.src] - u[self.dst]
        return (0.25 * (self.w * (d * d).sum(dim=1)).sum(),
                torch.zeros_like(u).index_add_(0, self.src, self.w[:, None] * d))

    def value_and_grad(self, u, alpha):
        v, gx, gy = self.sample(self.samples, u)
        r = v - self.i1
        energy, pull = self.springs(u)
        J = 0.5 * (r * r).sum() / max(self.n_pix, 1) + alpha * energy
        return J, self.to_nodes([r * gx, r * gy]) / max(self.n_pix, 1) + alpha * pull

    def cg(self, u, alpha, max_iters, tol):
        """Polak-Ribiere+ nonlinear CG with Armijo backtracking (10 halvings, then the step is taken)."""
        hist = torch.full((max_iters, 3), float("nan"), dtype=F64)
        J, g = self.value_and_grad(u, alpha)
        d, g_prev, k = torch.zeros_like(u), torch.zeros_like(u), 0
        while k < max_iters:
            gn = float(g.norm())
            if gn < tol:
                hist[k] = torch.tensor([float(J), gn, 0.0])
                break
            beta = max(float((g * (g - g_prev)).sum() / ((g_prev * g_prev).sum() + 1e-16)), 0.0) if k else 0.0
            d = -g + beta * d
            gd = float((g * d).sum())
            if gd >= 0:
                d, gd = -g, -gn * gn
            a = 1.0
            for _ in range(10):
                Jc, gc = self.value_and_grad(u + a * d, alpha)
                if float(Jc) <= float(J) + 1e-4 * a * gd:
                    break
                a *= 0.5
            else:
                last = Jc
                Jc, gc = self.value_and_grad(u + a * d, alpha)
                hist[k] = torch.tensor([float(last), gn, a], dtype=F64)
            if math.isnan(float(hist[k, 0])):
                hist[k] = torch.tensor([float(Jc), gn, a], dtype=F64)
            u, g_prev, g, J = u + a * d, g, gc, Jc
            k += 1
        return u, hist, k

    def hessian(self, u, alpha):
        """Dense Hessian over the used nodes' degrees of freedom, and their indices."""
        x, y = self.position(u)
        v, gx, gy, xx, xy, yy = _cubic(self.samples, x, y, second=True)
        r = (v - self.i1) / max(self.n_pix, 1)
        block = [[gx * gx / max(self.n_pix, 1) + r * xx, gx * gy / max(self.n_pix, 1) + r * xy],
                 [None, gy * gy / max(self.n_pix, 1) + r * yy]]
        block[1][0] = block[0][1]
        H = torch.zeros((2 * self.n, 2 * self.n), dtype=F64, device=DEV)
        for a in range(4):
            for b in range(4):
                for i in range(2):
                    for j in range(2):
                        per = torch.zeros(self.el.shape[0], dtype=F64, device=DEV)
                        per.index_add_(0, self.element, self.shape[a] * self.shape[b] * block[i][j])
                        H.index_put_((2 * self.el[:, a] + i, 2 * self.el[:, b] + j), per, accumulate=True)
        for i in range(2):
            H.index_put_((2 * self.src + i, 2 * self.src + i), alpha * self.w, accumulate=True)
            H.index_put_((2 * self.src + i, 2 * self.dst + i), -alpha * self.w, accumulate=True)
        dof = torch.nonzero(self.used.repeat_interleave(2)).reshape(-1)
        return H[dof][:, dof], dof

    def solve(self, u, alpha, B):
        """H^-1 B for right-hand sides B (Nn, 2, K); zero at unused nodes."""
        H, dof = self.hessian(u, alpha)
        X = torch.zeros((2 * self.n, B.shape[2]), dtype=F64, device=DEV)
        X[dof] = torch.linalg.solve(H, B.reshape(2 * self.n, -1)[dof])
        return X.reshape(self.n, 2, -1)

    def mixed(self, u, dI):
        """Derivative of the gradient at ``u`` along the image direction dI."""
        x, y = self.position(u)
        v, gx, gy = _cubic(self.samples, x, y)
        dv, dgx, dgy = _cubic(_coefficients(dI), x, y)
        r = v - self.i1
        return self.to_nodes([dv * gx + r * dgx, dv * gy + r * dgy]) / max(self.n_pix, 1)

    def mixed_transposed(self, u, lam):
        """Image-space adjoint of ``mixed`` for a nodal field lam (Nn, 2)."""
        dI = torch.zeros_like(self.img, requires_grad=True)
        (grad,) = torch.autograd.grad((self.mixed(u, dI) * lam).sum(), dI)
        return grad

    def neighbours(self):
        """Dense (src, dst) pairs of nodes sharing an element: the strain fit's neighbourhoods."""
        return self.src, self.dst

    def strain(self, u, du=None, eps=1e-8):
        """Green-Lagrange strain (Voigt) by least squares over the neighbours, or its derivative along du."""
        dX = self.nodes[self.dst] - self.nodes[self.src]
        fit = torch.zeros((self.n, 2, 2), dtype=F64, device=DEV).index_add_(0, self.src, dX[:, :, None] * dX[:, None, :])
        fit = torch.linalg.inv(fit + eps * torch.eye(2, dtype=F64, device=DEV))

        def gradient(v):
            b = torch.zeros((self.n, 2, 2), dtype=F64, device=DEV).index_add_(
                0, self.src, dX[:, :, None] * (v[self.dst] - v[self.src])[:, None, :])
            return (fit @ b).transpose(1, 2)

        Fm = torch.eye(2, dtype=F64, device=DEV) + gradient(u)
        E = (Fm.transpose(1, 2) @ Fm - torch.eye(2, dtype=F64, device=DEV)) / 2
        if du is not None:
            P = gradient(du).transpose(1, 2) @ Fm
            E = (P + P.transpose(1, 2)) / 2
        return torch.stack([E[:, 0, 0], E[:, 1, 1], E[:, 0, 1]], dim=1)

    def refine(self, u, alpha, sweeps, lam=1e-3, max_step=0.2, omega=0.5):
        """Relaxed nodal Gauss-Newton sweeps; gradient images by central differences, zero on the border."""
        gx, gy = torch.zeros_like(self.img), torch.zeros_like(self.img)
        gx[:, 1:-1] = (self.img[:, 2:] - self.img[:, :-2]) / 2
        gy[1:-1] = (self.img[2:] - self.img[:-2]) / 2
        fields = [_coefficients(f) if self.interp == "cubic" else f for f in (gx, gy)]
        has = torch.zeros(self.n, dtype=torch.bool, device=DEV)
        has[self.el[torch.unique(self.element)].reshape(-1)] = True
        sw = torch.zeros(self.n, dtype=F64, device=DEV).index_add_(0, self.src, self.w)
        hist = torch.full((sweeps, 2), float("nan"), dtype=F64)
        for k in range(sweeps):
            r = self.sample(self.samples, u)[0] - self.i1
            gx, gy = (self.sample(c, u)[0] for c in fields)
            b = self.to_nodes([r * gx, r * gy])
            A = torch.zeros((self.n, 3), dtype=F64, device=DEV)
            for a, n in enumerate(self.shape):
                per = torch.zeros((self.el.shape[0], 3), dtype=F64, device=DEV)
                per.index_add_(0, self.element, (n * n)[:, None] * torch.stack([gx * gx, gx * gy, gy * gy], dim=1))
                A.index_add_(0, self.el[:, a], per)
            b = b + alpha * self.springs(u)[1]
            add = lam * (A[:, 0] + A[:, 2] + 1e-12) + alpha * sw + 1e-8
            a11, a22, a12 = A[:, 0] + add, A[:, 2] + add, A[:, 1]
            step = -torch.stack([a22 * b[:, 0] - a12 * b[:, 1], a11 * b[:, 1] - a12 * b[:, 0]], 1) / (
                a11 * a22 - a12 * a12)[:, None]
            step = torch.where((has | ((sw > 0) if alpha else has))[:, None], step, 0.0)
            step = omega * step * torch.clamp(max_step / (step.norm(dim=1) + 1e-12), max=1.0)[:, None]
            hist[k] = torch.stack([(r * r).mean().sqrt(), (step * step).mean().sqrt()]).cpu()
            u = u + step
        return u, hist

    def discrepancy(self, u):
        """Bilinear I2(x + u) - I1(x) at the region's pixels (NaN elsewhere), and its RMS."""
        x, y = self.position(u)
        H, W = self.img.shape
        ok = (x >= 0) & (y >= 0) & (torch.floor(x) < W - 1) & (torch.floor(y) < H - 1)
        ok &= (self.col < W - 1) & (self.row < H - 1)
        r = torch.where(ok, _linear(self.img, x, y)[0] - self.i1, float("nan"))
        out = torch.full((H, W), float("nan"), dtype=F64, device=DEV)
        out[self.row.long(), self.col.long()] = r
        return out, float((r[ok] ** 2).sum().div(max(int(ok.sum()), 1)).sqrt())


def _zncc(ref, img, centres, win, search):
    """Best integer shift and score per centre, first maximum in row-major order of the offsets."""
    ref, img = ref.to(F64), img.to(F64)
    H, W = ref.shape
    r, ps, n = win // 2, win + 2 * search, win * win
    c = torch.round(torch.as_tensor(np.asarray(centres, np.float32), device=DEV).to(F64)).long()
    reach = r + search
    ok = ((c >= reach).all(dim=1)) & (c[:, 0] + reach < W) & (c[:, 1] + reach < H)
    u = torch.zeros((c.shape[0], 2), dtype=F64, device=DEV)
    score = torch.full((c.shape[0],), float("nan"), dtype=F64, device=DEV)
    size = 1 << (ps - 1).bit_length()
    where = torch.nonzero(ok).reshape(-1)
    for part in torch.split(where, 512):
        x, y = c[part, 0], c[part, 1]
        k = torch.arange(win, device=DEV)
        t = ref[(y[:, None] - r + k)[:, :, None], (x[:, None] - r + k)[:, None, :]]
        t = t - t.mean(dim=(1, 2), keepdim=True)
        t = t / (t.square().mean(dim=(1, 2), keepdim=True).sqrt() + 1e-12)
        k = torch.arange(ps, device=DEV)
        p = img[(y[:, None] - reach + k)[:, :, None], (x[:, None] - reach + k)[:, None, :]]
        p = p - p.mean(dim=(1, 2), keepdim=True)

        def boxes(v):
            s = torch.nn.functional.pad(v.cumsum(1).cumsum(2), (1, 0, 1, 0))
            return s[:, win:, win:] - s[:, :-win, win:] - s[:, win:, :-win] + s[:, :-win, :-win]

        mean = boxes(p) / n
        std = (boxes(p * p) / n - mean * mean).clamp(min=0).sqrt()
        cross = torch.fft.irfft2(torch.fft.rfft2(p, s=(size, size)) * torch.fft.rfft2(t, s=(size, size)).conj(),
                                 s=(size, size))[:, :2 * search + 1, :2 * search + 1]
        s = (cross / n / (std + 1e-12)).reshape(part.numel(), -1)
        best = s.argmax(dim=1)
        score[part] = s.gather(1, best[:, None])[:, 0]
        u[part] = torch.stack([best % (2 * search + 1) - search, best // (2 * search + 1) - search], 1).to(F64)
    return u, score


def _init_motion(p, win, search, score_min, img):
    centres = np.asarray(p["assets"].element_centers_xy, np.float32)
    u, score = _zncc(p["ref"], img, centres, win, search)
    keep = score >= score_min
    u = torch.where(keep[:, None], u, 0.0)
    nodes = torch.as_tensor(np.asarray(p["mesh"].nodes_xy, np.float32), device=DEV).to(F64)
    at = torch.as_tensor(centres, device=DEV).to(F64)
    out = torch.empty_like(nodes)
    for part in torch.split(torch.arange(nodes.shape[0], device=DEV), 1024):
        d2_ = (nodes[part][:, None, :] - at[None]).square().sum(dim=2)
        w = 1 / d2_.clamp(min=1e-300)
        near, which = d2_.min(dim=1)
        out[part] = torch.where((near < 1e-12)[:, None], u[which], (w @ u) / w.sum(dim=1, keepdim=True))
    return out, int(keep.sum())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        u, strain, hist, n = [], [], [], []
        for i, m in enumerate(_mix(case, case.get("sequences", case["frames"]))):
            extra = dict(pixels="u8", frames=case["frames"], reach=1) if kind == "serve" else {}
            p = _inputs(dict(m, **extra), 100 * seed + i)
            pb = _Problem(p["mesh"], p["assets"].roi_mask, p["ref"], case["interp"])
            at = (torch.as_tensor(p["u0"], device=DEV).to(F64) if kind == "batch"
                  else _init_motion(p, 17, 8, 0.2, p["frames"][0])[0])
            for img in p["frames"]:
                pb.load(img)
                at, h, k = pb.cg(at, case["reg"], case["max_iters"], case["tol"])
                u.append(at)
                hist.append(h)
                strain.append(pb.strain(at))
                n.append(k)
        if kind == "batch":
            return dict(u=u, history=hist, n_iters=np.array(n))
        return dict(u=u, strain=strain, n_iters=np.array(n))
    p = _inputs(case, seed)
    if kind == "init":
        u, matches = _init_motion(p, case["win"], case["search"], 0.2, p["frames"][0])
        return dict(u=u, matches=matches)
    pb = _Problem(p["mesh"], p["assets"].roi_mask, p["ref"], case.get("interp", "cubic"))
    T = lambda a: torch.as_tensor(a, device=DEV).to(F64)  # noqa: E731
    u0 = torch.zeros((pb.n, 2), dtype=F64, device=DEV) if p["u0"] is None else T(p["u0"])
    alpha = case["reg"]
    pb.load(p["frames"][0])
    if kind == "frame":
        u, hist, k = pb.cg(u0, alpha, case["max_iters"], case["tol"])
        return dict(u=u, strain=pb.strain(u), history=hist, n_iters=k)
    if kind == "sequence":
        out, before, u = dict(u=[], strain=[]), None, None
        for k, img in enumerate(p["frames"]):
            pb.load(img)
            start = u0 if u is None else (u if before is None else 2 * u - before)
            before = u
            u, _, _ = pb.cg(start, alpha, case["max_iters"], case["tol"])
            u, _ = pb.refine(u, alpha, case["sweeps"])
            out["u"].append(u)
            out["strain"].append(pb.strain(u))
        return out
    if kind == "step":
        u, _, _ = pb.cg(u0, alpha, case["max_iters"], case["tol"])
        for _ in range(6):
            u = u - pb.solve(u, alpha, pb.value_and_grad(u, alpha)[1][:, :, None])[:, :, 0]
        lam = pb.solve(u, alpha, _cotangents(pb.n, 1, seed)[0].to(F64)[:, :, None])[:, :, 0]
        return dict(u=u, grad=-pb.mixed_transposed(u, lam))
    if kind == "objective":
        J, g = pb.value_and_grad(u0, alpha)
        return dict(J=float(J), g=g)
    u = T(_linearisation_point(p, seed))
    if kind == "refine":
        u, hist = pb.refine(u, alpha, case["sweeps"])
        disc, rms = pb.discrepancy(u)
        return dict(u=u, strain=pb.strain(u), history=hist, discrepancy=disc, rms=rms)
    if kind == "jvp":
        B = torch.stack([pb.mixed(u, dI) for dI in _noise_images(case, seed)], dim=2)
        du = -pb.solve(u, alpha, B).permute(2, 0, 1)
        return dict(du=du, strain=torch.stack([pb.strain(u, d) for d in du]))
    lam = pb.solve(u, alpha, _cotangents(pb.n, case["images"], seed).to(F64).permute(1, 2, 0))
    return torch.stack([-pb.mixed_transposed(u, lam[:, :, k]) for k in range(case["images"])])
