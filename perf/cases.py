"""The calls that this framework is timed on, and their plain 64-bit values.

A user of the framework traces channels (tracer.Scene, tracer.trace_channel),
optimises the metasurface phases and the AP codes on them
(objective.capacity_objective, objective.ObjectivePlan, objective.Model) and
trains and queries the placement surrogate (surrogate.MLP).  listed() has one
case per kind of call at a size that the configurations, the tests or
bench.py use, or an odd neighbour of it; draw() spreads the same kinds over
their whole range.
"""
import math

import numpy as np
import torch

from automs_gb300 import objective, scenes, surrogate, tracer

LAM = scenes.WAVE_LEN_60GHZ
N0 = 1e-9                                 # noise power of the capacity, go.py:183-184
EPS = float(torch.finfo(torch.float32).eps)
TX = (6.0, 0.5, 2.5)                      # AP of the shoebox rooms
MS_C = (6.0, 8.0 - 1e-3, 2.0)             # metasurface on the wall across
NO_DIR = (0.0, 0.0, 0.0)


def listed():
    return [
        # build_channel on a small furnished room, as a first look at a floor
        # plan: the reference's default launch (100 x 100) and reflection
        # count (4), some furniture penetrable; a new scene on every call
        dict(name="trace-oneshot-room", kind="trace", link="ap-rx", oneshot=True, boxes=4, tess=1,
             room_tess=1, ap=4, ms=0, rx0=24, rx1=24, launch=100, refl=4, penetrable=True),
        # the headline coverage map: 2,172 triangles, 16 Tx elements, 128 x 128
        # Rx, a million launched rays, then the map in dB
        dict(name="trace-coverage-128", kind="trace", link="ap-rx", oneshot=False, boxes=20,
             tess=3, room_tess=1, ap=16, ms=0, rx0=128, rx1=128, launch=1000, refl=2,
             penetrable=False),
        # AP -> Rx of a channel set in a large, finely meshed room (60k
        # triangles), 256 x 256 Rx, three reflections
        dict(name="trace-ap-rx-60k", kind="trace", link="ap-rx", oneshot=False, boxes=200,
             tess=5, room_tess=13, ap=16, ms=0, rx0=256, rx1=256, launch=1000, refl=3,
             penetrable=False),
        # AP -> metasurface of the same set: the receivers are the 1,024
        # elements, half a wavelength apart
        dict(name="trace-ap-ms-60k", kind="trace", link="ap-ms", oneshot=False, boxes=200,
             tess=5, room_tess=13, ap=16, ms=32, rx0=0, rx1=0, launch=1000, refl=3,
             penetrable=False),
        # metasurface -> Rx: 1,024 sources, a ragged Rx grid; the trace that a
        # placement study spends its time in
        dict(name="trace-ms-rx", kind="trace", link="ms-rx", oneshot=False, boxes=60, tess=3,
             room_tess=4, ap=0, ms=32, rx0=101, rx1=83, launch=500, refl=2, penetrable=False),
        # one step of a phase optimisation on fixed channels (one code)
        dict(name="objective-c1", kind="objective", plan=True, C=1, S=16, M=1024, R=4096),
        # the same step on freshly traced channels, without a plan: a 48 x 48
        # metasurface and a 256 x 256 map, the middle of the batched placements
        dict(name="objective-c1-64k", kind="objective", plan=False, C=1, S=16, M=2304, R=65536),
        # one step of a 60-code codebook optimisation on a 256 x 256 map
        dict(name="codebook-60-64k", kind="objective", plan=True, C=60, S=16, M=1024, R=65536),
        # a codebook of the 36-element AP without a metasurface, odd Rx count
        dict(name="codebook-no-ms", kind="objective", plan=False, C=30, S=36, M=0, R=5929),
        # Model of two metasurfaces, paths of up to two hops: loss and
        # gradients as optimize_model takes them
        dict(name="model-two-ms", kind="model", C=30, S=36, m0=24, m1=16, R=2116),
        # one training step of the placement surrogate, the study's batch
        dict(name="surrogate-train", kind="train", B=64, d_in=72, hidden=512, d_out=4096),
        # scoring one batch of annealing moves
        dict(name="surrogate-score", kind="score", B=256, d_in=72, hidden=512, d_out=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("trace", "trace", "trace", "objective", "objective", "model", "train",
                       "score"))
    if kind == "trace":
        link = rng.choice(("ap-rx", "ap-rx", "ap-ms", "ms-rx"))
        big = rng.random() < 0.4
        boxes, tess = (_log(rng, 40, 200), rng.randint(3, 5)) if big else (_log(rng, 2, 40),
                                                                         rng.randint(1, 3))
        c = dict(kind="trace", link=link, oneshot=rng.random() < 0.3, boxes=boxes, tess=tess,
                 room_tess=rng.randint(1, 13), ap=0 if link == "ms-rx" else rng.randint(1, 36),
                 ms=0 if link == "ap-rx" else rng.randint(6, 32), rx0=0, rx1=0,
                 launch=_log(rng, 64, 800), refl=rng.randint(0, 4) if not big else
                 rng.randint(1, 3), penetrable=rng.random() < 0.25)
        if link != "ap-ms":
            hi = 72 if link == "ms-rx" else 200
            c["rx0"], c["rx1"] = _log(rng, 7, hi), _log(rng, 7, hi)
        if link == "ms-rx" or c["penetrable"]:
            c["refl"] = min(c["refl"], 2)
        return c
    if kind == "objective":
        C = rng.choice((1, 1, 2, rng.randint(3, 64)))
        M = rng.choice((0, 1, 1)) * _log(rng, 16, 4096 if C <= 2 else 2048)
        plan = M > 0 and rng.random() < 0.6
        hi = 65536 if plan or C <= 2 else 16384
        return dict(kind="objective", plan=plan, C=C, S=rng.randint(1, 36), M=M,
                    R=_log(rng, 128, hi))
    if kind == "model":
        return dict(kind="model", C=rng.randint(1, 60), S=rng.randint(4, 36),
                    m0=rng.randint(5, 32), m1=rng.randint(5, 32), R=_log(rng, 200, 8000))
    return dict(kind=kind, B=_log(rng, 1, 1024 if kind == "train" else 4096),
                d_in=rng.randint(16, 96), hidden=128 * rng.randint(1, 6),
                d_out=128 * rng.randint(2, 32))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _channel(g, *shape):
    """CN(0, 1) fading scaled by the free-space loss over 2 to 15 m."""
    d = torch.rand(shape, generator=g, device="cuda").mul_(13.0).add_(2.0)
    d = (LAM / (4 * math.pi * math.sqrt(2.0))) / d
    re = torch.randn(shape, generator=g, device="cuda").mul_(d)
    im = torch.randn(shape, generator=g, device="cuda").mul_(d)
    return torch.complex(re, im)


def _quads(p0, u, v, nu, nv):
    """2 nu nv triangles of the quad p0 + s u + t v."""
    s = np.arange(nu)[:, None, None]
    t = np.arange(nv)[None, :, None]
    at = lambda a, b: p0 + u * ((s + a) / nu) + v * ((t + b) / nv)  # noqa: E731
    a, b, c, d = at(0, 0), at(1, 0), at(1, 1), at(0, 1)
    return np.stack([np.stack([a, b, c], 2), np.stack([a, c, d], 2)], 2).reshape(-1, 3, 3)


def _box(lo, hi, n):
    e = np.diag(hi - lo)
    x, y, z = e
    return np.concatenate([_quads(p, u, v, n, n) for p, u, v in (
        (lo, x, y), (lo + z, x, y), (lo, x, z), (lo + y, x, z), (lo, y, z), (lo + x, y, z))])


def _room(case, seed):
    """Shoebox room with floor-standing boxes, as scenes.shoebox_scene makes."""
    rng = np.random.default_rng([int(seed), case["boxes"], case["tess"]])
    X, Y, Z = 12.0, 8.0, 3.0
    shell = _box(np.zeros(3), np.array([X, Y, Z]), case["room_tess"])
    n6 = len(shell) // 6
    tris, mats = [shell], [np.repeat([0, 1, 2], [n6, n6, 4 * n6])]
    for b in range(case["boxes"]):
        while True:
            (sx, sy), h = rng.uniform(0.2, 1.5, 2), rng.uniform(0.3, 2.0)
            cx, cy = rng.uniform(0, X), rng.uniform(0, Y)
            lo = np.array([max(cx - sx / 2, 0.0), max(cy - sy / 2, 0.0), 0.0])
            hi = np.array([min(cx + sx / 2, X), min(cy + sy / 2, Y), h])
            if all(np.any(p < lo - 0.05) or np.any(p > hi + 0.05) for p in (TX, MS_C)):
                break
        t = _box(lo, hi, case["tess"])
        tris.append(t)
        mats.append(np.full(len(t), 3 + b))
    prop = np.repeat(rng.uniform(0.3, 0.7, 3 + case["boxes"])[:, None], 19, 1)
    if case["penetrable"]:
        prop[3::3] *= -1.0  # every third box lets rays through
    return (np.concatenate(tris).astype(np.float32), np.concatenate(mats).astype(np.int32),
            prop.astype(np.float32))


def _prepare_trace(case, seed):
    tris, mat, prop = _room(case, seed)
    cuda = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda")  # noqa: E731
    rng = np.random.default_rng([int(seed), 7])
    at = np.array([rng.uniform(-0.2, 0.2), 0.0, rng.uniform(-0.1, 0.1)])  # arrays' place
    link = case["link"]
    if link != "ms-rx":
        src, sdir, sbp = scenes.ula(np.add(TX, at), (1, 0, 0), case["ap"], LAM / 2), (0., 1., 0.), 2
    if link != "ap-rx":
        pos, quad, nrm = scenes.metasurface(np.add(MS_C, at), (0, -1, 0), (0, 0, -1), case["ms"],
                                            LAM / 2)
        nrm = tuple(float(x) for x in nrm)
    if link == "ms-rx":
        src, sdir, sbp = pos, nrm, 1
    if link == "ap-ms":
        dst, ddir, dbp = pos, nrm, 1
    else:
        dst, ddir, dbp = scenes.rx_grid(0.25, 11.75, case["rx0"], 0.25, 7.75, case["rx1"],
                                        1.5), NO_DIR, 0
    p = tracer.make_params(launch_x=case["launch"], launch_y=case["launch"], wave_len=LAM,
                           max_reflection=case["refl"], src_bptype=sbp, dst_bptype=dbp,
                           src_dir=sdir, dst_dir=ddir)
    s = dict(kind="trace", src=cuda(src), dst=cuda(dst), params=p,
             arrays=(cuda(tris), cuda(mat), cuda(prop)), coverage=link == "ap-rx")
    if not case["oneshot"]:
        s["scene"] = tracer.Scene(*s["arrays"])
    return s


def _prepare_objective(case, seed):
    g = _gen(seed)
    C, S, M, R = case["C"], case["S"], case["M"], case["R"]
    s = dict(kind="objective", R=R, Hd=_channel(g, S, R), Ha=None, Hr=None, phi=None, plan=None)
    theta = torch.rand((C, S), generator=g, device="cuda").mul_(2 * math.pi)
    s["W"] = (torch.polar(torch.ones_like(theta), -theta) / math.sqrt(S)).requires_grad_()
    if M:
        s["Ha"], s["Hr"] = _channel(g, S, M), _channel(g, M, R)
        s["phi"] = torch.rand(M, generator=g, device="cuda").mul_(2 * math.pi).requires_grad_()
    # one code: the mean over the Rx; codebooks: the reference's sum and its
    # 10% code dropout
    s["w"] = 1.0 / R if C == 1 else 1.0
    s["drop"] = torch.rand(C, generator=g, device="cuda") < 0.1 if C > 2 else None
    if case["plan"]:
        s["plan"] = objective.ObjectivePlan(s["Hd"], s["Ha"], s["Hr"], c_max=C)
    return s


class _Surface:
    max_phase = 2 * math.pi


def _model_inputs(case, seed):
    g = _gen(seed)
    S, M, R = case["S"], (case["m0"] ** 2, case["m1"] ** 2), case["R"]
    ch = {"src_to_dst": _channel(g, S, R), "ms{0}_to_ms{1}": _channel(g, M[0], M[1])}
    for i in range(2):
        ch["src_to_ms{%d}" % i] = _channel(g, S, M[i])
        ch["ms{%d}_to_dst" % i] = _channel(g, M[i], R)
    theta = torch.rand((case["C"], S), generator=g, device="cuda").mul_(2 * math.pi)
    phi = [torch.rand(m, generator=g, device="cuda").mul_(2 * math.pi) for m in M]
    return ch, theta, phi


def _prepare_model(case, seed):
    ch, theta, phi = _model_inputs(case, seed)
    model = objective.Model("two-ms", ch, [_Surface(), _Surface()], max_ms_reflex=2,
                            code_num=case["C"], drop_rate=0.0)
    with torch.no_grad():
        model.antenna_theta.copy_(theta)
        for t, p in zip(model.ms_theta, phi):
            t.copy_(p)
    return dict(kind="model", model=model)


def _dims(case):
    return [case["d_in"]] + [case["hidden"]] * 4 + [case["d_out"]]


def _mlp_inputs(case, seed):
    """Weights (He-uniform) and Adam moments of a run some way into its
    training, a batch and its targets."""
    g = _gen(seed)
    dims, parts = _dims(case), []
    for a, b in zip(dims[:-1], dims[1:]):
        parts.append((torch.rand(a * b, generator=g, device="cuda") * 2 - 1) * math.sqrt(6.0 / a))
        parts.append((torch.rand(b, generator=g, device="cuda") * 2 - 1) * 0.05)
    params = torch.cat(parts)
    m1 = torch.randn(params.numel(), generator=g, device="cuda") * 1e-4
    m2 = torch.rand(params.numel(), generator=g, device="cuda") * 1e-6 + 1e-8
    X = torch.randn((case["B"], case["d_in"]), generator=g, device="cuda")
    T = torch.randn((case["B"], case["d_out"]), generator=g, device="cuda")
    return params, m1, m2, X, T


def _prepare_mlp(case, seed):
    params, m1, m2, X, T = _mlp_inputs(case, seed)
    net = surrogate.MLP(_dims(case), max_batch=4096)
    net.load_state_dict(dict(dims=_dims(case), params=params, adam_m=m1, adam_v=m2,
                             adam_step=200))
    return dict(kind=case["kind"], net=net, X=X, T=T)


def prepare(case, seed):
    return {"trace": _prepare_trace, "objective": _prepare_objective, "model": _prepare_model,
            "train": _prepare_mlp, "score": _prepare_mlp}[case["kind"]](case, seed)


# --------------------------------------------------------------- one pass
COUNTS = ("rx_paths", "rx_fail", "fwd_records", "unique_records", "unique_paths", "rounds",
          "tasks", "overflow")


def run(s):
    kind = s["kind"]
    if kind == "trace":
        if "scene" in s:
            res, st = s["scene"].trace(s["src"], s["dst"], s["params"])
            H = torch.complex(res[..., 0], res[..., 1])
        else:
            H, st = tracer.trace_channel(*s["arrays"], s["src"], s["dst"], s["params"])
        out = dict(H=H, counts=[st[k] for k in COUNTS])
        if s["coverage"]:
            out["db"] = tracer.coverage_db(H)
        return out
    if kind == "objective":
        loss, amp = objective.capacity_objective(s["W"], s["Hd"], s["Ha"], s["Hr"], s["phi"],
                                                 2 * math.pi, s["w"], s["drop"],
                                                 return_recv=True, plan=s["plan"])
        leaves = [s["W"]] + ([s["phi"]] if s["phi"] is not None else [])
        return dict(loss=loss.detach(), amp=amp, grads=torch.autograd.grad(loss, leaves))
    if kind == "model":
        m = s["model"]
        loss = m()
        loss.backward()
        out = dict(loss=loss.detach(), amp=m.result, theta=m.antenna_theta.grad,
                   phi=[t.grad for t in m.ms_theta])
        m.zero_grad(set_to_none=True)
        return out
    if kind == "train":
        loss = s["net"].train_step(s["X"], s["T"], lr=1e-3)
        return dict(loss=loss, params=s["net"].get_params())
    return dict(Y=s["net"](s["X"]))


# ------------------------------------------------------------ least work
def _queries(tris):
    """Operations of one closest-hit query in an ideal tree of four-triangle
    leaves: two 18-operation box tests a level and four 40-operation
    triangle tests."""
    return 36 * math.ceil(math.log2(max(2, tris / 4))) + 160


def work(case):
    kind = case["kind"]
    if kind == "trace":
        tris = 12 * case["room_tess"] ** 2 + 12 * case["boxes"] * case["tess"] ** 2
        S = case["ap"] or case["ms"] ** 2
        R = case["ms"] ** 2 if case["link"] == "ap-ms" else case["rx0"] * case["rx1"]
        rays = case["launch"] ** 2
        # every launched ray up to its last reflection; the direct path of
        # every pair (the reflected ones depend on the scene)
        q = rays * (case["refl"] + 1) + S * R
        return dict(bytes=40.0 * tris + 12.0 * (S + R) + 8.0 * S * R, flops=float(q * _queries(tris)))
    if kind == "objective":
        C, S, M, R = case["C"], case["S"], case["M"], case["R"]
        rows = M + S
        return dict(bytes=8.0 * (R * rows + S * M + 2 * C * S) + 4.0 * C * R + 8.0 * M,
                    flops=16.0 * C * (R * rows + S * M))
    if kind == "model":
        C, S, R = case["C"], case["S"], case["R"]
        M = case["m0"] ** 2 + case["m1"] ** 2
        MM = case["m0"] ** 2 * case["m1"] ** 2
        return dict(bytes=8.0 * (R * (M + S) + S * M + MM + 2 * C * S) + 4.0 * C * R + 8.0 * M,
                    flops=16.0 * C * (R * (M + S) + 2 * S * M + 2 * MM))
    dims = _dims(case)
    n = sum((a + 1) * b for a, b in zip(dims[:-1], dims[1:]))
    B = case["B"]
    if kind == "train":
        # weights and both moments read and written, the weights handed back
        return dict(bytes=28.0 * n + 4.0 * B * (dims[0] + dims[-1]), flops=6.0 * B * n)
    return dict(bytes=2.0 * n + 4.0 * B * (dims[0] + dims[-1]), flops=2.0 * B * n)


# ------------------------------------------------------------ 64-bit values
def _capacity(Y, w, drop):
    """Loss of go.py:159-226 from Y [C, R] complex128."""
    cap = torch.log2(1 + (Y.abs() + EPS) ** 2 / N0)
    if drop is not None:
        cap = torch.where(drop[:, None], torch.zeros_like(cap), cap)
    top = cap.max(0).values
    loss = -w * top.sum()
    if Y.shape[0] > 1:
        loss = loss + torch.linalg.vector_norm(cap * (cap != top).double())
    return loss


def _exact_objective(case, seed):
    case = dict(case, plan=False)
    s = _prepare_objective(case, seed)
    wide = lambda t: t.detach().to(torch.complex128)  # noqa: E731
    W = wide(s["W"]).requires_grad_()
    U, leaves = None, [W]
    if s["phi"] is not None:
        phi = s["phi"].detach().double().requires_grad_()
        leaves.append(phi)
        U = (W @ wide(s["Ha"])) * torch.polar(torch.ones_like(phi), phi)
    # over blocks of Rx: the gradients of Y first, then the sums over Rx
    blocks = [slice(a, min(a + 8192, case["R"])) for a in range(0, case["R"], 8192)]
    with torch.no_grad():
        Y = torch.cat([W @ wide(s["Hd"][:, b]) + (U @ wide(s["Hr"][:, b]) if U is not None else 0)
                       for b in blocks], 1)
    Y.requires_grad_()
    loss = _capacity(Y, s["w"], s["drop"])
    gY, = torch.autograd.grad(loss, Y)
    gW = torch.zeros_like(W)
    gU = torch.zeros_like(U) if U is not None else None
    with torch.no_grad():
        for b in blocks:
            gW += gY[:, b] @ wide(s["Hd"][:, b]).mH
            if U is not None:
                gU += gY[:, b] @ wide(s["Hr"][:, b]).mH
    grads = [gW]
    if U is not None:
        more = torch.autograd.grad(U, leaves, grad_outputs=gU)
        grads = [gW + more[0], more[1]]
    return dict(loss=loss.detach(), amp=Y.detach().abs(), grads=grads)


def _exact_model(case, seed):
    ch, theta, phi = _model_inputs(case, seed)
    ch = {k: v.to(torch.complex128) for k, v in ch.items()}
    theta = theta.double().requires_grad_()
    phi = [p.double().requires_grad_() for p in phi]
    S = case["S"]
    A = torch.ones(theta.shape, dtype=torch.float64, device="cuda") / math.sqrt(S / 36)
    if S == 36:
        A[:, [0, 5, 30, 35]] = 0
    W = torch.polar(A, -theta)
    e = [torch.polar(torch.ones_like(p), p) for p in phi]
    V0 = (W @ ch["src_to_ms{0}"]) * e[0]
    V1 = (W @ ch["src_to_ms{1}"]) * e[1]
    U0 = V0 + (V1 @ ch["ms{0}_to_ms{1}"].mT) * e[0]
    U1 = V1 + (V0 @ ch["ms{0}_to_ms{1}"]) * e[1]
    Y = W @ ch["src_to_dst"] + U0 @ ch["ms{0}_to_dst"] + U1 @ ch["ms{1}_to_dst"]
    loss = _capacity(Y, 1.0, None)
    g = torch.autograd.grad(loss, [theta] + phi)
    return dict(loss=loss.detach(), amp=Y.detach().abs(), theta=g[0], phi=list(g[1:]))


def _forward(dims, p, X):
    H, k = X, 0
    for i, (a, b) in enumerate(zip(dims[:-1], dims[1:])):
        H = H @ p[k:k + a * b].view(b, a).T + p[k + a * b:k + a * b + b]
        k += (a + 1) * b
        if i < len(dims) - 2:
            H = H.relu()
    return H


def _exact_mlp(case, seed):
    params, m1, m2, X, T = (t.double() for t in _mlp_inputs(case, seed))
    params.requires_grad_()
    Y = _forward(_dims(case), params, X)
    if case["kind"] == "score":
        return dict(Y=Y.detach())
    loss = ((Y - T) ** 2).mean()
    g, = torch.autograd.grad(loss, params)
    m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
    step = 1e-3 * (m1 / (1 - 0.9 ** 201)) / ((m2 / (1 - 0.999 ** 201)).sqrt() + 1e-8)
    return dict(loss=loss.detach(), params=params.detach() - step)


def exact(case, seed):
    """The traces have none: which rays reach a receiver is defined by the
    float32 arithmetic of the geometry, and verifying them one by one in
    plain numpy takes minutes."""
    if case["kind"] == "trace":
        return None
    return {"objective": _exact_objective, "model": _exact_model, "train": _exact_mlp,
            "score": _exact_mlp}[case["kind"]](case, seed)
