"""The work a user has the fitting library do, as cases of a performance measurement.

Every case goes through the package's public entry points (``Batch.fit_frames``,
``Batch.landmark_init``, ``Batch.render``, ``render_loss`` and its backward pass,
``Batch.set_video_frames``, ``tdi_raster_noalloc``). The models are the ones the package's
workloads use: 53,490 vertices (the full-size face mesh), 19,830 (the size of the fitted
model the reference ships with) and 5,000. Frames follow the package's video workload: AR(1)
expressions, random-walk head angles, face boxes of 120-600 px at 1080p rescaled to the
reference face size and cropped to 256x256. They are generated here (batched on the GPU) so
that a batch of a thousand frames takes seconds.

Kinds of case and their ranges (what ``draw`` draws from):

fit_frame   one to four frames per call, host arrays in and out: interactive use, latency.
fit_batch   a video's frames fitted together, exact arithmetic (the default): 16 to 1,024.
fit_tensor  the same with both contractions on the tensor cores: 16 to 512.
window      what the drop-in program does with a window of frames on the shipped model size:
            landmark initialisation on the device, then the reference's two-stage illumination
            sequence and the expression finetune, up to 100 iterations: 8 to 96 frames.
landmarks   landmark initialisation alone (a start for every frame of a video): 1 to 1,024.
render      images and owner-triangle maps of fitted states: 1 to 64 frames.
loss_grad   the differentiable loss and its gradients (forward and backward): 1 to 96 frames.
crops       decoded video frames to crops, read back: 1 to 24 frames of 720p or 1080p.
visibility  one frame's visible fragments from device arrays, no allocation: the smallest call.
"""
import ctypes as C
import functools
import importlib
import math

import numpy as np
import torch

tdi = importlib.import_module("3di_b200")
synth = importlib.import_module("3di_b200.synth")
autograd = importlib.import_module("3di_b200.autograd")

NL, DIM, NPIX = 51, 256, 65536
FOCAL, WIDTH, HEIGHT = 800.0, 1920, 1080
BOUND, MARGIN = 0.08, 0.03
TRIANGLES = {53490: 106466, 19830: 39053, 5000: 9800}
# Raster passes and Gauss-Newton evaluations of one frame of the video workload capped at 20
# outer iterations, and visible fragments of a face of the reference size: what the counts in
# work() stand on.
RENDERS, EVALS, FRAGMENTS = 22, 9, 3900


def listed():
    return [
        # one frame of a live stream: the smallest fit, all latency and launches
        {"name": "fit_frame_1", "kind": "fit_frame", "V": 53490, "F": 1},
        # an ordinary chunk of a video, a ragged count
        {"name": "fit_batch_77", "kind": "fit_batch", "V": 53490, "F": 77},
        # the throughput batch of the benchmark
        {"name": "fit_batch_1024", "kind": "fit_batch", "V": 53490, "F": 1024},
        # the mixed-precision mode on a mid-size batch
        {"name": "fit_tensor_300", "kind": "fit_tensor", "V": 53490, "F": 300},
        # a window of the drop-in program on the shipped model's size
        {"name": "window_48", "kind": "window", "V": 19830, "F": 48},
        # starts for a video's frames
        {"name": "landmarks_500", "kind": "landmarks", "V": 53490, "F": 500},
        # one frame's start (every live frame begins with it)
        {"name": "landmarks_1", "kind": "landmarks", "V": 19830, "F": 1},
        # overlays of a fitted clip
        {"name": "render_24", "kind": "render", "V": 19830, "F": 24},
        # a training step through the loss on the full mesh, and a single small one
        {"name": "loss_grad_96", "kind": "loss_grad", "V": 53490, "F": 96},
        {"name": "loss_grad_2", "kind": "loss_grad", "V": 5000, "F": 2},
        # a clip's decoded frames to crops
        {"name": "crops_13_1080p", "kind": "crops", "W": 1920, "H": 1080, "F": 13},
        # visibility from device arrays
        {"name": "visibility_1", "kind": "visibility", "V": 53490, "F": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit_frame", "fit_batch", "fit_batch", "fit_tensor", "window", "landmarks", "render",
                       "loss_grad", "crops", "visibility"])
    c = {"kind": kind, "V": rng.choice([5000, 19830, 53490])}
    if kind == "fit_frame":
        c["F"] = rng.randint(1, 4)
    elif kind == "fit_batch":
        c["F"] = _log(rng, 16, 1024)
    elif kind == "fit_tensor":
        c["F"] = _log(rng, 16, 512)
    elif kind == "window":
        c["F"] = _log(rng, 8, 96)
    elif kind == "landmarks":
        c["F"] = _log(rng, 1, 1024)
    elif kind == "render":
        c["F"] = _log(rng, 1, 64)
    elif kind == "loss_grad":
        c["F"] = _log(rng, 1, 96)
    elif kind == "crops":
        del c["V"]
        c["W"], c["H"] = rng.choice([(1280, 720), (1920, 1080), (1279, 719)])
        c["F"] = _log(rng, 1, 24)
    else:
        c["F"] = 1
    return c


# ------------------------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=None)
def _mesh(V):
    """The subject's model: one per size, as a program fits one subject."""
    return synth.make_model(V, TRIANGLES[V], config_id=1, n_id=24, n_tex=24)


def _dev(a):
    return torch.as_tensor(np.asarray(a)).to("cuda", torch.float64)


def _rodrigues(u):
    th = torch.linalg.norm(u, dim=1)[:, None, None]
    n = u / th[:, :, 0]
    z = torch.zeros_like(n[:, 0])
    S = torch.stack([z, -n[:, 2], n[:, 1], n[:, 2], z, -n[:, 0], -n[:, 1], n[:, 0], z], 1).reshape(-1, 3, 3)
    return torch.eye(3, dtype=u.dtype, device=u.device) + torch.sin(th) * S + (1 - torch.cos(th)) * (S @ S)


def _axis_angles(ang_deg):
    return np.stack([synth.euler_to_axis_angle(*np.deg2rad(a)) for a in ang_deg])


def _points(mean, E, eps, u, tau):
    """Camera points [F][3][n] of the vertices mean [3][n], E [n][3][K] at the given states."""
    n, K = E.shape[0], E.shape[2]
    P = mean[None] + (eps @ E.reshape(n * 3, K).T).reshape(-1, n, 3).transpose(1, 2)
    return P, _rodrigues(u) @ P + tau[:, :, None]


def _make_frames(V, F, seed, want_targets=True, pinned=False):
    """Frames of a video (synth.Frames) and their targets: a point-sampled rendering of the mesh
    at the true states (nearest of the triangles' sample points per pixel) with noise."""
    m = _mesh(V)
    rng = np.random.Generator(np.random.PCG64([seed, V, F]))
    K = m.n_expr
    eps, ang = np.empty((F, K)), np.empty((F, 3))
    e, a = rng.normal(size=K), rng.uniform(-20, 20, size=3)
    for f in range(F):
        if f:
            e = 0.95 * e + math.sqrt(1 - 0.95 ** 2) * rng.normal(size=K)
            a = np.clip(a + rng.normal(0.0, 1.5, size=3), -40.0, 40.0)
        eps[f], ang[f] = np.clip(e, -3.5, 3.5), a
    mean, E = _dev(m.mean), _dev(m.E)
    lis = torch.as_tensor(m.lis.astype(np.int64)).cuda()
    extent = float(max(np.ptp(m.mean[0, m.lis].astype(np.float64)), np.ptp(m.mean[1, m.lis].astype(np.float64))))
    tz = FOCAL * extent / rng.uniform(120, 600, F)
    half = FOCAL * extent / tz * 0.75
    px = half + (WIDTH - 2 * half) * rng.uniform(size=F)
    py = half + np.maximum(HEIGHT - 2 * half, 0.0) * rng.uniform(size=F)
    tau = np.stack([(px - WIDTH / 2) * tz / FOCAL, (py - HEIGHT / 2) * tz / FOCAL, tz], 1)
    noise = rng.normal(0.0, 1.5, (2, F, NL))
    lam_true = synth.LAMBDA_INIT + rng.normal(0.0, 0.02, (F, 3)) / synth.UNIT_M
    d_ang, d_tau, d_eps = rng.normal(0, 2.0, (F, 3)), rng.normal(0, 0.003, (F, 3)) / synth.UNIT_M, rng.normal(0, 0.3, (F, K))
    tri = torch.as_tensor(m.tl.astype(np.int64)).cuda()
    S = max(1, 100000 // m.n_triangles)
    w = np.random.Generator(np.random.PCG64(7)).dirichlet([1.0, 1.0, 1.0], S)
    w[0] = 1.0 / 3.0
    tex = _dev(m.tex)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed * 1000003 + F)
    targets = None
    if want_targets:
        targets = torch.empty((F, NPIX), dtype=torch.float32, pin_memory=pinned)
    fr = synth.Frames(xl=np.empty((F, NL), np.float32), yl=np.empty((F, NL), np.float32),
                      bounds=np.empty((F, 4, NL), np.float32), face_size=np.empty(F, np.float32),
                      cam=np.empty((F, 4), np.float32), x0y0=np.empty((F, 2), np.int32),
                      state_true=np.empty((F, K + 6), np.float32), state_init=np.empty((F, K + 6), np.float32),
                      lam_true=lam_true.astype(np.float32),
                      target=targets.numpy() if want_targets else np.zeros((F, 1), np.float32))
    bl, bu = -BOUND - MARGIN * 2 * BOUND, BOUND + MARGIN * 2 * BOUND
    fr.bounds[:, :2], fr.bounds[:, 2:] = bl, bu
    for f0 in range(0, F, 64):
        f1 = min(F, f0 + 64)
        n = f1 - f0
        for shrink in range(6):         # a face that leaves the crop gets a milder pose and expression
            sc = 0.6 ** shrink
            u = _axis_angles(ang[f0:f1] * sc)
            P, X = _points(mean, E, _dev(eps[f0:f1] * sc), _dev(u), _dev(tau[f0:f1]))
            xv, yv = FOCAL * X[:, 0] / X[:, 2] + WIDTH / 2, FOCAL * X[:, 1] / X[:, 2] + HEIGHT / 2
            lo = torch.stack([xv.min(1).values, yv.min(1).values], 1).cpu().numpy()
            hi = torch.stack([xv.max(1).values, yv.max(1).values], 1).cpu().numpy()
            xo, yo = xv[:, lis].cpu().numpy() + noise[0, f0:f1], yv[:, lis].cpu().numpy() + noise[1, f0:f1]
            ok = True
            for i in range(n):
                f = f0 + i
                box = max(int(xo[i].max()) - int(xo[i].min()), int(yo[i].max()) - int(yo[i].min()))
                rc = synth.REF_FACE_SIZE / box
                need = synth.REF_FACE_SIZE / 1.5 + 16.0
                shx = max(0.0, need - xo[i].min() * rc, 8.0 - lo[i, 0] * rc)
                shy = max(0.0, need - yo[i].min() * rc, 8.0 - lo[i, 1] * rc)
                fr.xl[f], fr.yl[f] = xo[i] * rc + shx, yo[i] * rc + shy
                fr.cam[f] = [FOCAL * rc, FOCAL * rc, WIDTH / 2 * rc + shx, HEIGHT / 2 * rc + shy]
                fr.face_size[f] = synth.face_size(fr.xl[f], fr.yl[f])
                fr.x0y0[f] = synth.crop_origin(fr.xl[f], fr.yl[f])
                ox, oy = fr.x0y0[f]
                ok &= (lo[i, 0] * rc + shx - ox >= 2 and hi[i, 0] * rc + shx - ox <= DIM - 3
                       and lo[i, 1] * rc + shy - oy >= 2 and hi[i, 1] * rc + shy - oy <= DIM - 3)
            if ok:
                break
        fr.state_true[f0:f1, :K], fr.state_true[f0:f1, K:K + 3] = eps[f0:f1] * sc, tau[f0:f1]
        fr.state_true[f0:f1, K + 3:] = u
        if want_targets:
            cam = _dev(fr.cam[f0:f1])
            R = _rodrigues(_dev(u))
            lamt = _dev(lam_true[f0:f1])
            q = torch.einsum("fji,fj->fi", R, lamt - _dev(tau[f0:f1]))
            b, c, a3 = P[:, :, tri[0]], P[:, :, tri[1]], P[:, :, tri[2]]
            nr = torch.cross(b - a3, c - a3, dim=1)
            nr = nr / torch.linalg.norm(nr, dim=1, keepdim=True)
            key = torch.full((n, NPIX), 2 ** 62, dtype=torch.int64, device="cuda")
            val = []
            for s in range(S):
                w0, w1, w2 = (float(x) for x in w[s])
                p = w0 * b + w1 * c + w2 * a3
                t = w0 * tex[tri[0]] + w1 * tex[tri[1]] + w2 * tex[tri[2]]
                Id = torch.einsum("fct,fc->ft", nr, q) - (nr * p).sum(1)
                val.append(t + float(synth.L_INTENSITY) * t * Id)
                pc = R @ p + _dev(tau[f0:f1])[:, :, None]
                ix = torch.round(cam[:, 0:1] * pc[:, 0] / pc[:, 2] + cam[:, 2:3]).long() - torch.as_tensor(fr.x0y0[f0:f1, 0:1].astype(np.int64)).cuda()
                iy = torch.round(cam[:, 1:2] * pc[:, 1] / pc[:, 2] + cam[:, 3:4]).long() - torch.as_tensor(fr.x0y0[f0:f1, 1:2].astype(np.int64)).cuda()
                pix = (ix.clamp(0, DIM - 1) * DIM + iy.clamp(0, DIM - 1))
                kk = (pc[:, 2] * 4096.0).long() * (1 << 24) + (s * m.n_triangles + torch.arange(m.n_triangles, device="cuda"))
                key.scatter_reduce_(1, pix, kk, "amin")
            hit = key < 2 ** 62
            img = torch.gather(torch.cat(val, 1), 1, torch.where(hit, key % (1 << 24), 0)) * hit
            img = img + 0.02 * torch.randn(img.shape, generator=gen, device="cuda", dtype=torch.float64)
            targets[f0:f1].copy_(img.float())
            del b, c, a3, nr, val, key, img
        # a start near the truth whose landmarks lie strictly inside their boxes
        scale, done = np.ones(n), np.zeros(n, bool)
        lm_mean, lm_E = mean[:, lis], E[lis]
        for _ in range(12):
            u0 = _axis_angles(ang[f0:f1] * sc + d_ang[f0:f1] * scale[:, None])
            t0 = tau[f0:f1] + d_tau[f0:f1] * scale[:, None]
            e0 = np.clip(eps[f0:f1] * sc + d_eps[f0:f1] * scale[:, None], -3.5, 3.5)
            X = _points(lm_mean, lm_E, _dev(e0), _dev(u0), _dev(t0))[1].cpu().numpy()
            xp = fr.cam[f0:f1, 0:1] * X[:, 0] / X[:, 2] + fr.cam[f0:f1, 2:3]
            yp = fr.cam[f0:f1, 1:2] * X[:, 1] / X[:, 2] + fr.cam[f0:f1, 3:4]
            fs = fr.face_size[f0:f1, None]
            g = np.concatenate([xp - (fr.xl[f0:f1] + bl * fs), yp - (fr.yl[f0:f1] + bl * fs),
                                (fr.xl[f0:f1] + bu * fs) - xp, (fr.yl[f0:f1] + bu * fs) - yp], 1)
            done = g.min(1) > 0.5
            if done.all():
                break
            scale[~done] *= 0.5
        fr.state_init[f0:f1, :K], fr.state_init[f0:f1, K:K + 3], fr.state_init[f0:f1, K + 3:] = e0, t0, u0
    return m, fr


def _light(F):
    return np.tile(synth.LAMBDA_INIT, (F, 1)).astype(np.float32), np.full(F, synth.L_INTENSITY, np.float32)


def _video(c, seed):
    """Decoded BGR frames (smooth shading with texture), landmarks of a face in each."""
    rng = np.random.Generator(np.random.PCG64([seed, c["W"], c["F"]]))
    F, W, H = c["F"], c["W"], c["H"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed * 7919 + F)
    low = torch.rand((F, 3, H // 16 + 2, W // 16 + 2), generator=gen, device="cuda")
    img = torch.nn.functional.interpolate(low, size=(H, W), mode="bilinear", align_corners=False) * 235.0
    img = (img + 20.0 * torch.rand((F, 1, H, W), generator=gen, device="cuda")).to(torch.uint8)
    bgr = img.permute(0, 2, 3, 1).contiguous().cpu().numpy()
    face = rng.uniform(120, 0.55 * H, F).astype(np.float32)
    t = rng.uniform(-0.5, 0.5, (2, F, NL))
    t[:, :, 0], t[:, :, 1] = -0.5, 0.5
    cx, cy = rng.uniform(0.3, 0.7, F) * W, rng.uniform(0.35, 0.65, F) * H
    xp = (cx[:, None] + t[0] * face[:, None]).astype(np.float32)
    yp = (cy[:, None] + t[1] * face[:, None]).astype(np.float32)
    cam = np.tile(np.array([FOCAL, FOCAL, W / 2, H / 2], np.float32), (F, 1))
    bounds = np.empty((F, 4, NL), np.float32)
    bounds[:, :2], bounds[:, 2:] = -BOUND, BOUND
    return dict(bgr=bgr, xp=xp, yp=yp, bounds=bounds, face_size=face, cam=cam,
                ref_face_size=float(synth.REF_FACE_SIZE))


def prepare(case, seed):
    kind, F = case["kind"], case["F"]
    st = {"kind": kind}
    if kind == "crops":
        st["video"] = _video(case, seed)
        st["model"] = tdi.Model(_mesh(5000))
        st["batch"] = tdi.Batch(st["model"], F)
        return st
    if kind == "visibility":
        m, fr = _make_frames(case["V"], 1, seed, want_targets=False)
        xp, yp, zc = _project(m, fr, 0)
        st["proj"] = tuple(p.float().contiguous() for p in (xp, yp, zc))
        st["tl"] = torch.as_tensor(m.tl).cuda()
        st["size"] = (m.n_vertices, m.n_triangles, int(fr.x0y0[0, 0]), int(fr.x0y0[0, 1]))
        st["out"] = torch.zeros((32768, 4), dtype=torch.int32, device="cuda")
        st["count"] = torch.zeros(1, dtype=torch.int32, device="cuda")
        st["flags"] = torch.zeros(1, dtype=torch.int32, device="cuda")
        return st
    # the throughput batch is uploaded from pinned memory, as a program that streams video does
    m, fr = _make_frames(case["V"], F, seed, want_targets=kind not in ("landmarks", "render"),
                         pinned=kind in ("fit_batch", "fit_tensor"))
    if kind in ("landmarks", "render"):
        fr.target = np.zeros((F, NPIX), np.float32)
    st["fr"], st["model"] = fr, tdi.Model(m)
    st["batch"] = tdi.Batch(st["model"], F)
    st["lam"], st["L"] = _light(F)
    if kind in ("fit_frame", "fit_batch"):
        st["cfg"] = tdi.default_config(max_iters_rigid=20)
    elif kind == "fit_tensor":
        st["cfg"] = tdi.default_config(max_iters_rigid=20, normal_eq=tdi.NORMAL_EQ_TENSOR,
                                       vertex_stage=tdi.VERTEX_TENSOR)
    elif kind in ("window", "landmarks"):
        st["p0L"] = np.ascontiguousarray(m.mean[:, m.lis].astype(np.float32))
        st["cfg"] = tdi.default_config(twostage_illum=1, finetune=1)
        if kind == "landmarks":
            st["batch"].set_frames(fr)
            st["batch"].set_state(fr.state_init, st["lam"], st["L"])
    elif kind == "render":
        st["batch"].set_frames(fr)
        st["batch"].set_state(fr.state_true, fr.lam_true, st["L"])
    elif kind == "loss_grad":
        st["batch"].set_frames(fr)
        st["cfg"] = tdi.default_config()
        st["leaf"] = [torch.as_tensor(a).cuda().requires_grad_(True) for a in (fr.state_init, st["lam"], st["L"])]
    return st


def _reports(rep):
    return np.array([[r.flags, r.n_fragments, r.iters_rigid, r.iters_finetune, r.iters_lambda, r.renders]
                     for r in rep], np.int64), np.array([r.objective for r in rep], np.float32)


def run(st):
    kind = st["kind"]
    if kind in ("fit_frame", "fit_batch", "fit_tensor"):
        x, lam, rep = st["batch"].fit_frames(st["fr"], st["fr"].state_init, st["lam"], st["L"], st["cfg"])
        return (x, lam) + _reports(rep)
    if kind == "window":
        b = st["batch"]
        b.set_frames(st["fr"])
        ok, slack, it = b.landmark_init(st["p0L"])
        b.set_state(None, st["lam"], st["L"])
        b.fit(st["cfg"])
        x, lam, rep = b.get_state()
        return (ok, slack, it, x, lam) + _reports(rep)
    if kind == "landmarks":
        ok, slack, it = st["batch"].landmark_init(st["p0L"])
        x, _, _ = st["batch"].get_state()
        return ok, slack, it, x
    if kind == "render":
        return st["batch"].render(want_images=True, want_tri_map=True)
    if kind == "loss_grad":
        for t in st["leaf"]:
            t.grad = None
        loss = autograd.render_loss(st["batch"], *st["leaf"], st["cfg"])
        loss.sum().backward()
        return [loss.detach()] + [t.grad for t in st["leaf"]]
    if kind == "crops":
        b = st["batch"]
        b.set_video_frames(**st["video"])
        return [b.read(f, tdi.READ_CROP) for f in range(b.n)]
    V, T, x0, y0 = st["size"]
    p = [C.c_void_p(t.data_ptr()) for t in st["proj"] + (st["tl"],)]
    s = tdi.load_library().tdi_raster_noalloc(
        *p, V, T, x0, y0, C.c_void_p(st["out"].data_ptr()), st["out"].shape[0], C.c_void_p(st["count"].data_ptr()),
        C.c_void_p(st["flags"].data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    if s != 0:
        raise RuntimeError("tdi_raster_noalloc: status %d" % s)
    return st["out"], st["count"], st["flags"]


def work(case):
    kind, F = case["kind"], case["F"]
    if kind == "crops":
        # every decoded byte in; crops out; the few operations of gray and bilinear per crop pixel
        return {"bytes": float(F * (3 * case["W"] * case["H"] + 4 * NPIX)), "flops": 40.0 * F * NPIX}
    V, T, K = case["V"], TRIANGLES[case["V"]], 79
    mesh = 4.0 * V * (3 + 1 + 3 * K) + 12.0 * T
    raster = 60.0 * T                                     # box, denominator and one sample per triangle
    vertex = 2.0 * 3 * V * K + 21.0 * V
    pixels = FRAGMENTS * (40.0 + 2 * 15 * 2 * 2)          # shading, blur of render and target
    normal = 2.0 * FRAGMENTS * ((K + 6) * (K + 7)) + FRAGMENTS * (K + 6) * 60.0
    if kind in ("fit_frame", "fit_batch", "fit_tensor", "window"):
        turns = 3 if kind == "window" else 1              # two-stage illumination repeats both fits
        per = turns * (RENDERS * (vertex + raster + pixels) + EVALS * normal)
        return {"bytes": mesh + F * (4.0 * NPIX + 4.0 * (NL * 6 + 8 + 2 * (K + 9)) + 28.0), "flops": F * per}
    if kind == "landmarks":
        n = K + 7                                         # three Newton steps at least, each a 204-row system
        return {"bytes": 4.0 * NL * 3 * (K + 1) + F * 4.0 * (NL * 6 + 8 + K + 6),
                "flops": F * 3.0 * (204.0 * n * n + n ** 3 / 3.0)}
    if kind == "render":
        return {"bytes": mesh + F * (4.0 * (K + 9) + 8.0 * NPIX), "flops": F * (vertex + raster + FRAGMENTS * 40.0)}
    if kind == "loss_grad":
        return {"bytes": mesh + F * (4.0 * NPIX + 3.0 * 4 * (K + 10)),
                "flops": F * (3 * vertex + raster + 3 * pixels)}
    return {"bytes": 12.0 * V + 12.0 * T + 16.0 * FRAGMENTS, "flops": raster}


# ------------------------------------------------------------- values in 64 bits (plain torch)

def _project(m, fr, f):
    """FP64 projections (xp, yp, camera Z) of a frame's vertices at its true state."""
    K = m.n_expr
    x = _dev(fr.state_true[f:f + 1])
    _, X = _points(_dev(m.mean), _dev(m.E), x[:, :K], x[:, K + 3:], x[:, K:K + 3])
    cam = _dev(fr.cam[f])
    return cam[0] * X[0, 0] / X[0, 2] + cam[2], cam[1] * X[0, 1] / X[0, 2] + cam[3], X[0, 2]


def _rotation32(u):
    """The path's FP32 rotation: sin and cos in FP64 rounded to FP32, products in FP32."""
    f = np.float32
    u = [f(v) for v in u]
    th = np.sqrt(f(f(u[0] * u[0] + u[1] * u[1]) + u[2] * u[2]))
    n = [f(v / th) for v in u]
    S = np.array([0, n[2], -n[1], -n[2], 0, n[0], n[1], -n[0], 0], f)
    S2 = np.empty(9, f)
    for j in range(3):
        for i in range(3):
            S2[3 * j + i] = f(f(S[i] * S[3 * j] + S[3 + i] * S[3 * j + 1]) + S[6 + i] * S[3 * j + 2])
    st, ci = f(math.sin(float(th))), f(f(1) - f(math.cos(float(th))))
    return [f(f(ci * S2[i] + f(1 if i % 4 == 0 else 0)) + st * S[i]) if i % 4 == 0 else f(ci * S2[i] + st * S[i])
            for i in range(9)]


def _fragments(m, mean32, E, tri, x, cam, x0, y0):
    """Visible samples of a frame. Visibility is a decision the path defines on FP32 values (which
    triangle is sampled at which pixel), so the projections and tests are FP32 here too; everything
    computed from it is FP64. Returns (triangle, pixel, owner) of the surviving samples."""
    K = m.n_expr
    acc = torch.zeros(E.shape[:2], dtype=torch.float32, device="cuda")
    for k in range(K):                                    # fused multiply-add: exact product, one rounding
        acc = (E[:, :, k] * float(x[k]) + acc.double()).float()
    P = mean32 + acc.T
    R, tau = _rotation32(x[K + 3:]), [np.float32(v) for v in x[K:K + 3]]
    X = [((float(R[i]) * P[0] + float(R[3 + i]) * P[1]) + float(R[6 + i]) * P[2]) + float(tau[i]) for i in range(3)]
    xp, yp = (float(cam[0]) * X[0]) / X[2] + float(cam[2]), (float(cam[1]) * X[1]) / X[2] + float(cam[3])
    b, c, a = tri
    bx, by, cx, cy, ax, ay = xp[b], yp[b], xp[c], yp[c], xp[a], yp[a]
    xlo, ylo = torch.floor(torch.minimum(torch.minimum(bx, cx), ax)), torch.floor(torch.minimum(torch.minimum(by, cy), ay))
    xhi, yhi = torch.ceil(torch.maximum(torch.maximum(bx, cx), ax)), torch.ceil(torch.maximum(torch.maximum(by, cy), ay))
    v0x, v1x, v0y, v1y = bx - ax, cx - ax, by - ay, cy - ay
    d00, d01, d11 = v0x * v0x + v0y * v0y, v0x * v1x + v0y * v1y, v1x * v1x + v1y * v1y
    den = d00 * d11 - d01 * d01
    zb = X[2][b].view(torch.int32).long()
    ids = torch.arange(m.n_triangles, device="cuda")
    row = torch.zeros_like(ids)
    out = []
    for i in range(int((xhi - xlo).max().item())):
        for j in range(int((yhi - ylo).max().item())):
            sx, sy = xlo + i, ylo + j
            v2x, v2y = sx - ax, sy - ay
            d20, d21 = v0x * v2x + v0y * v2y, v1x * v2x + v1y * v2y
            al, be = (d11 * d20 - d01 * d21) / den, (d00 * d21 - d01 * d20) / den
            ok = (sx < xhi) & (sy < yhi) & (al > 0) & (be > 0) & (al + be <= 1) & (row < 4)
            t = ids[ok]
            pix = ((sy[ok].long() - y0) + (sx[ok].long() - x0) * DIM) & 0xFFFF
            out.append(torch.stack([t, pix, row[ok]]))
            row = row + ok
    t, pix, r = torch.cat(out, 1)
    z = torch.full((NPIX,), 2 ** 62, dtype=torch.int64, device="cuda")
    key = zb[t] * (1 << 20) + t
    z.scatter_reduce_(0, pix, key, "amin")
    keep = (z[pix] >> 20 == zb[t]) & ~((t == 0) & (r == 0))
    return t[keep], pix[keep], (z[pix] == key)[keep]


def _image(tri, tex, frag, P, Rm, tau, lam, L, cam, x0, y0):
    """FP64 unblurred image over the given fragments (differentiable)."""
    t, pix, own = frag
    X = Rm @ P + tau[:, None]
    xp, yp = cam[0] * X[0] / X[2] + cam[2], cam[1] * X[1] / X[2] + cam[3]
    t, pix = t[own], pix[own]
    b, c, a = tri[0][t], tri[1][t], tri[2][t]
    sx, sy = (x0 + (pix >> 8)).double(), (y0 + (pix & 255)).double()
    v0x, v0y, v1x, v1y = xp[b] - xp[a], yp[b] - yp[a], xp[c] - xp[a], yp[c] - yp[a]
    v2x, v2y = sx - xp[a], sy - yp[a]
    D = v0x * v1y - v0y * v1x
    al, be = (v2x * v1y - v2y * v1x) / D, (v0x * v2y - v0y * v2x) / D
    ga = 1 - al - be
    nr = torch.linalg.cross((P[:, b] - P[:, a]).T, (P[:, c] - P[:, a]).T)
    nh = nr / torch.linalg.norm(nr, dim=1, keepdim=True)
    Id = nh @ (Rm.T @ (lam - tau)) - (nh * (P[:, b] * al + P[:, c] * be + P[:, a] * ga).T).sum(1)
    tt = tex[b] * al + tex[c] * be + tex[a] * ga
    return torch.zeros(NPIX, dtype=torch.float64, device="cuda").index_put((pix,), tt + L * tt * Id)


def _rotmat(u):
    th = torch.linalg.norm(u)
    n = u / th
    z = torch.zeros_like(n[0])
    S = torch.stack([z, -n[2], n[1], n[2], z, -n[0], -n[1], n[0], z]).reshape(3, 3)
    return torch.eye(3, dtype=u.dtype, device=u.device) + torch.sin(th) * S + (1 - torch.cos(th)) * (S @ S)


def _loss(img, target, pix, taps):
    k = taps.reshape(1, 1, 1, -1)

    def blur(a):
        a = torch.nn.functional.conv2d(a.reshape(1, 1, DIM, DIM), k, padding=(0, 7))
        return torch.nn.functional.conv2d(a, k.transpose(2, 3), padding=(7, 0)).reshape(-1)

    def grads(A):
        xx, yy = pix >> 8, pix & 255
        kr, kl = torch.where(xx < DIM - 1, pix + DIM, 0), torch.where(xx > 0, pix - DIM, 0)
        kd, ku = torch.where(yy < DIM - 1, pix + 1, 0), torch.where(yy > 0, pix - 1, 0)
        gx, gy = 0.5 * (A[kr] - A[kl]), 0.5 * (A[kd] - A[ku])
        s = 4 * gx * gx + 4 * gy * gy
        h = 1e-16 + torch.where(s > 0, torch.sqrt(torch.where(s > 0, s, 1.0)), 0.0)
        return 2 * gx / h, 2 * gy / h

    gx, gy = grads(blur(img))
    tx, ty = grads(blur(target))
    return -(gx * tx + gy * ty).sum()


def exact(case, seed):
    kind, F = case["kind"], case["F"]
    if kind == "crops":
        v = _video(case, seed)
        out = []
        for f in range(F):
            ref = np.float32(v["ref_face_size"]) / v["face_size"][f]
            c = float(ref)
            B, G, R = (v["bgr"][f, :, :, q].astype(np.int64) for q in range(3))
            gray = ((3735 * B + 19235 * G + 9798 * R + (1 << 14)) >> 15) / 255.0
            H, W = gray.shape
            rw, rh = int(np.rint(W * c)), int(np.rint(H * c))
            x0, y0 = synth.crop_origin(ref * v["xp"][f], ref * v["yp"][f])
            crop = np.zeros((DIM, DIM))
            xs, ys = np.arange(x0, min(x0 + DIM, rw)), np.arange(y0, min(y0 + DIM, rh))
            if len(xs) and len(ys):
                def taps(p, n):
                    s = (p + 0.5) / c - 0.5
                    i = np.floor(s)
                    w = s - i
                    return np.clip(i, 0, n - 1).astype(int), np.clip(i + 1, 0, n - 1).astype(int), w
                xa, xb, wx = taps(xs, W)
                ya, yb, wy = taps(ys, H)
                top = gray[np.ix_(ya, xa)] * (1 - wx) + gray[np.ix_(ya, xb)] * wx
                bot = gray[np.ix_(yb, xa)] * (1 - wx) + gray[np.ix_(yb, xb)] * wx
                crop[:len(xs), :len(ys)] = (top * (1 - wy[:, None]) + bot * wy[:, None]).T
            out.append(crop.reshape(-1))
        return out
    if kind not in ("render", "loss_grad"):
        return None                                       # iterates of a line search: no such value
    m, fr = _make_frames(case["V"], F, seed, want_targets=kind == "loss_grad")
    K = m.n_expr
    mean32, mean, E, tex = torch.as_tensor(m.mean).cuda(), _dev(m.mean), _dev(m.E), _dev(m.tex)
    tri = tuple(torch.as_tensor(m.tl.astype(np.int64)).cuda())
    taps = _dev(np.asarray(synth.KERNEL_SIGMA_TAPS[0.75], np.float32))
    states = fr.state_true if kind == "render" else fr.state_init
    lam, L = (fr.lam_true, _light(F)[1]) if kind == "render" else _light(F)
    images, losses, grads = [], [], []
    for f in range(F):
        x0, y0 = int(fr.x0y0[f, 0]), int(fr.x0y0[f, 1])
        frag = _fragments(m, mean32, E, tri, states[f], fr.cam[f], x0, y0)
        z = [_dev(states[f]), _dev(lam[f]), _dev(L[f])]
        if kind == "loss_grad":
            z = [t.requires_grad_(True) for t in z]
        P = mean + (E.reshape(-1, K) @ z[0][:K]).reshape(-1, 3).T
        img = _image(tri, tex, frag, P, _rotmat(z[0][K + 3:]), z[0][K:K + 3], z[1], z[2], _dev(fr.cam[f]), x0, y0)
        if kind == "render":
            images.append(img.cpu().numpy())
            continue
        loss = _loss(img, _dev(fr.target[f]), frag[1], taps)
        loss.backward()
        losses.append(loss.item())
        grads.append([t.grad.cpu().numpy() for t in z])
    if kind == "render":
        return np.stack(images), None
    return [np.array(losses)] + [np.stack([g[i] for g in grads]) for i in range(3)]
