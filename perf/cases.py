"""The calls whose speed is measured: the work a reconstruction does through the package's public entry points.

Three kinds of case, each through `dragonfly_b200._lib`:

* "iterate": one EMC iteration from host buffers (Context.run_iteration_host), as a reconstruction script runs it:
  the start model and the scale factors go up, the iteration runs, the new model, the most likely orientations, the
  per-frame likelihoods and the scale factors come back. 3-D volumes, several modes and 2-D image stacks; from a random
  start model at low beta (broad probabilities) and near the solution at beta 1 (peaked ones); dim to bright frames;
  full and refined (coarse-to-fine) orientation searches.
* "slice": one slice of the model (Context.slice_gen), the smallest call.
* "propose" / "train": the proposal network's inference (ProposalNet.topk and logits) and the gradients of one training
  batch.

Sizes are those of the benchmark's workloads (the 260 x 257 production detector with a 201^3 model, the batched
reconstructions of 51^3 to 151^3 on square detectors of the model's size), of the tests (41^3 with 48 x 48 pixels,
61^3 with 64 x 64) and of the profiles (3240 orientations), with odd ones between. Frames, models and orientations are
synthetic, made from the seed: |F|^2 of Gaussian atoms in a ball, Poisson counts of its slices at uniformly random
orientations with lognormal fluence.
"""
import math

import numpy as np
import torch

from dragonfly_b200._lib import Context, ProposalNet
from dragonfly_b200.quatgen import quat_gen
from dragonfly_b200.synth import flat_detector

DEV = "cuda"
SIGMA = 0.4                  # lognormal width of the fluence
BETA_START = 0.01            # beta of a first iteration from a random model
TINY = np.finfo(np.float64).tiny


def _it(name, size, nx, ny, div, frames, photons, **kw):
    case = dict(name=name, kind="iterate", size=size, nx=nx, ny=ny, div=div, frames=frames, photons=photons, modes=1,
                two_d=False, scaling=True, late=False, coarse=0, budget_mb=0)
    case.update(kw)
    return case


def listed():
    return [
        # a single slice at the production detector: viewers, simulators and tests call it one orientation at a time
        dict(name="slice_one", kind="slice", size=201, nx=260, ny=257),
        # a first try on a small detector without scale factors: launches and latency count
        _it("first_try", 41, 48, 48, 2, 450, 80., scaling=False),
        # the small configuration of the profiles: 3240 orientations, 64 x 64 pixels
        _it("small", 61, 64, 64, 4, 3000, 300.),
        # batched reconstructions of the benchmark: the 95^3 and the 125^3 one (fewer frames)
        _it("medium", 95, 95, 95, 7, 40000, 200.),
        # near the solution: true model and scales, beta 1, so each frame keeps few orientations
        _it("converged", 125, 125, 125, 6, 30000, 400., late=True),
        # bright particles, an even model size and a rectangular detector: multi-photon pixels everywhere
        _it("bright", 110, 117, 101, 5, 15000, 1500.),
        # four modes sharing one orientation set
        _it("modes", 81, 83, 83, 4, 20001, 200., modes=4),
        # 2-D class averages: image stacks with in-plane angles
        _it("planar", 101, 101, 101, 180, 20000, 250., modes=10, two_d=True, scaling=False),
        # coarse-to-fine refinement: each frame near the cells that a coarse run found for it
        _it("refined", 85, 91, 91, 6, 12000, 300., late=True, coarse=2),
        # the network's proposals for newly measured frames, at the production's number of cells
        dict(name="propose", kind="propose", classes=3240, images=3000, keep=16),
        # one training batch of the network: loss and gradients
        dict(name="train", kind="train", classes=3240, images=256),
        # the production workload (50100 orientations, gap rows, central hole) with a share of its frames in several chunks
        _it("production", 201, 260, 257, 10, 60000, 300., budget_mb=12000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["iterate"] * 6 + ["refined", "modes", "planar", "slice", "propose", "train"])
    if kind == "slice":
        return dict(kind="slice", size=_log(rng, 31, 201), nx=_log(rng, 32, 260), ny=_log(rng, 32, 260))
    if kind == "propose":
        return dict(kind="propose", classes=rng.choice([420, 1380, 3240]), images=_log(rng, 500, 5000),
                    keep=rng.randint(4, 32))
    if kind == "train":
        return dict(kind="train", classes=rng.choice([60, 420, 1380, 3240]), images=rng.choice([64, 128, 256]))
    size = _log(rng, 31, 201)
    nx = min(260, max(32, int(size * rng.uniform(0.9, 1.3))))
    ny = min(260, max(32, int(size * rng.uniform(0.9, 1.3))))
    photons = float(_log(rng, 50, 1500))
    frames = _log(rng, 300, 60000)
    case = _it("", size, nx, ny, rng.randint(2, 10), frames, photons, scaling=rng.random() < 0.7,
               late=rng.random() < 0.4)
    del case["name"]
    if kind == "refined":
        case.update(div=rng.randint(4, 7), coarse=2, late=True)
    elif kind == "modes":
        case.update(modes=rng.randint(2, 6), div=rng.randint(2, 5))
    elif kind == "planar":
        case.update(modes=rng.randint(1, 12), div=rng.randint(60, 360), two_d=True, scaling=rng.random() < 0.5)
    # orientation blocks and frames stay below the production case's
    while _pixels(case) * _orientations(case) * case["modes"] > 3.3e9 and case["div"] > 2:
        case["div"] -= 1
    per_frame = _orientations(case) * case["modes"] * photons
    case["frames"] = max(300, min(frames, int(8e11 / per_frame)))
    if _orientations(case) * case["modes"] * case["frames"] > 1e9:
        case["budget_mb"] = 12000
    return case


def _pixels(case):
    return case["nx"] * case["ny"]


def _orientations(case):
    n = case["div"]
    return n if case["two_d"] else 10 * (5 * n ** 3 + n)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _detector(case):
    """Flat detector; the production one has six gap rows and a 10-pixel hole."""
    size = case["size"]
    big = case["nx"] >= 250
    hole = 10. if big else max(2., case["nx"] / 25.)
    qmax = 100. * (size / 201.) if big else (size - 3) / 2.
    gap = list(range(case["nx"] // 2 - 3, case["nx"] // 2 + 3)) if big else None
    q, corr, mask, _, _ = flat_detector(case["nx"], case["ny"], qmax, size, hole_radius=hole, gap_rows=gap)
    if case.get("two_d"):
        q = q.copy()
        q[:, 2] = 0.
    return q, corr, mask


def _atoms(size, two_d, shift, gen):
    """|F|^2 of 1000 Gaussian atoms in a ball (or disc) around the centre, the last 50 shifted."""
    dim = 2 if two_d else 3
    pos = torch.randn(1000, dim, generator=gen, dtype=torch.float64)
    pos *= 0.15 * size * torch.rand(1000, 1, generator=gen, dtype=torch.float64) ** (1. / dim) / \
        pos.norm(dim=1, keepdim=True)
    pos[950:, 0] += shift
    idx = pos.round().long() % size
    flat = idx[:, 0]
    for k in range(1, dim):
        flat = flat * size + idx[:, k]
    rho = torch.zeros(size ** dim, dtype=torch.float64).index_add_(0, flat, torch.ones(1000, dtype=torch.float64))
    f = torch.fft.fftn(rho.reshape((size,) * dim).to(DEV))
    k = torch.fft.fftfreq(size, dtype=torch.float64, device=DEV) ** 2
    k2 = k
    for _ in range(1, dim):
        k2 = k2[..., None] + k
    f = f * torch.exp(-2. * math.pi ** 2 * k2)
    return torch.fft.fftshift(f.abs() ** 2).contiguous()


def _rotations(q):
    """Rotation matrices [n, 3, 3] of quaternions [n, >= 4]."""
    q0, q1, q2, q3 = (q[:, k] for k in range(4))
    rows = [1. - 2. * (q2 * q2 + q3 * q3), 2. * (q1 * q2 + q0 * q3), 2. * (q1 * q3 - q0 * q2),
            2. * (q1 * q2 - q0 * q3), 1. - 2. * (q1 * q1 + q3 * q3), 2. * (q0 * q1 + q2 * q3),
            2. * (q0 * q2 + q1 * q3), 2. * (q2 * q3 - q0 * q1), 1. - 2. * (q1 * q1 + q2 * q2)]
    return torch.stack(rows, 1).reshape(-1, 3, 3)


def _positions(orient, qvals, size, two_d):
    """Pixel positions in the model [n, P, dim] under orientations [n, .] (quaternions, or angles in column 0)."""
    if two_d:
        c, s = torch.cos(orient[:, 0]), torch.sin(orient[:, 0])
        rot = torch.stack([c, -s, s, c], 1).reshape(-1, 2, 2)
        return torch.einsum("nij,pj->npi", rot, qvals[:, :2]) + size // 2
    return torch.einsum("nij,pj->npi", _rotations(orient), qvals) + size // 2


def _corners(pos, size):
    """Cell corners of positions [..., dim]: [(flat index, weight)], and which positions are inside the model."""
    base = pos.trunc()
    ok = ((base >= 0) & (base <= size - 2)).all(-1)
    f = pos - base
    i0 = torch.where(ok[..., None], base, torch.zeros_like(base)).long()
    out = []
    dim = pos.shape[-1]
    for corner in range(2 ** dim):
        w, idx = None, None
        for k in range(dim):
            up = corner >> (dim - 1 - k) & 1
            wk = f[..., k] if up else 1. - f[..., k]
            w = wk if w is None else w * wk
            ik = i0[..., k] + up
            idx = ik if idx is None else idx * size + ik
        out.append((idx, w))
    return out, ok


def _slices(model, orient, qvals, corr, two_d, outside):
    size = model.shape[0]
    cor, ok = _corners(_positions(orient, qvals, size, two_d), size)
    flat = model.reshape(-1)
    v = sum(w * flat[i] for i, w in cor) * corr
    return torch.where(ok, v, torch.full_like(v, outside))


def _inputs(case, seed):
    """Everything of an "iterate" case, on the host (numpy), from the seed."""
    gen = torch.Generator().manual_seed(seed)
    dgen = torch.Generator(device=DEV).manual_seed(seed + 1)
    size, two_d, M, N = case["size"], case["two_d"], case["modes"], case["frames"]
    qvals, corr, mask = _detector(case)
    if two_d:
        quats = np.zeros((case["div"], 5))
        quats[:, 0] = np.arange(case["div"]) * 2. * np.pi / case["div"]
        quats[:, 4] = 1. / case["div"]
    else:
        quats = np.ascontiguousarray(quat_gen(case["div"]))
    dq, dc = torch.from_numpy(qvals).to(DEV), torch.from_numpy(corr).to(DEV)
    dm = torch.from_numpy(mask).to(DEV)
    truth = torch.stack([_atoms(size, two_d, 0.04 * size * m, gen) for m in range(M)])

    def orientations(n):
        if two_d:
            return torch.rand(n, 1, generator=gen, dtype=torch.float64) * 2. * math.pi
        q = torch.randn(n, 4, generator=gen, dtype=torch.float64)
        return q / q.norm(dim=1, keepdim=True)

    # scale every mode to the wanted mean count on the detector
    probe = orientations(24).to(DEV)
    for m in range(M):
        mean = _slices(truth[m], probe, dq, dc, two_d, 0.)[:, dm <= 1].sum(1).mean()
        truth[m] *= case["photons"] / mean
    true_q = orientations(N)
    phi = torch.exp(SIGMA * torch.randn(N, generator=gen, dtype=torch.float64))
    mode = torch.randint(0, M, (N,), generator=gen)
    t32, q32, c32 = truth.float(), dq.float(), dc.float()
    c32 = c32 * (dm <= 1)
    block = max(16, min(2048, int(2e7 / _pixels(case))))
    ones, multi, po, pm, cm = [], [], [], [], []
    for s in range(0, N, block):
        e = min(N, s + block)
        lam = torch.zeros(e - s, qvals.shape[0], device=DEV)
        for m in range(M):
            mine = (mode[s:e] == m).nonzero()[:, 0].to(DEV)
            if mine.numel():
                lam[mine] = _slices(t32[m], true_q[s:e].to(DEV).float()[mine], q32, c32, two_d, 0.)
        counts = torch.poisson(lam.clamp_(min=0.) * phi[s:e, None].to(DEV).float(), generator=dgen).to(torch.int32)
        one, more = counts == 1, counts > 1
        ones.append(one.sum(1).to(torch.int32))
        multi.append(more.sum(1).to(torch.int32))
        po.append(one.nonzero()[:, 1].to(torch.int32))
        where = more.nonzero(as_tuple=True)
        pm.append(where[1].to(torch.int32))
        cm.append(counts[where])
    ones, multi, po, pm, cm = (torch.cat(x).cpu().numpy() for x in (ones, multi, po, pm, cm))
    if case["late"]:
        model = truth.cpu().numpy()
        scale = phi.numpy().copy()
    else:
        level = case["photons"] / max(1, int((mask == 0).sum())) * 2.
        model = (torch.rand(truth.shape, generator=gen, dtype=torch.float64) * level).numpy()
        scale = np.ones(N)
    inp = dict(qvals=qvals, corr=corr, mask=mask, quats=quats, model=model, scale=scale, ones=ones, multi=multi, po=po,
               pm=pm, cm=cm)
    if case["coarse"]:
        # cells of the coarse set: the nearest one of every fine orientation, and each frame's 12 nearest
        coarse = quat_gen(case["coarse"])
        near = lambda a: (a.to(DEV) @ torch.from_numpy(coarse[:, :4].T.copy()).to(DEV)).abs()
        inp["cells"] = near(torch.from_numpy(quats[:, :4].copy())).argmax(1).to(torch.int32).cpu().numpy()
        inp["relevant"] = near(true_q).topk(12, dim=1).indices.sort(1).values.to(torch.int32).cpu().numpy()
        inp["num_coarse"] = coarse.shape[0]
    return inp


def _schedule(case):
    """Arguments of Context.params: the first iteration of a run, or one near its end with the scales known."""
    if case["late"]:
        return dict(iteration=1, need_scaling=int(case["scaling"]), update_scale=1, known_scale=int(case["scaling"]))
    return dict(iteration=1, need_scaling=int(case["scaling"]), update_scale=1, known_scale=0)


def _beta(case):
    return 1. if case["late"] else BETA_START


def _images(case, seed):
    """Network inputs: log(1 + photons) on the 32 x 32 grid, a blurred random pattern per image."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    n = case["images"]
    coarse = torch.rand(n, 1, 8, 8, generator=gen, device=DEV) ** 3
    lam = torch.nn.functional.interpolate(coarse, size=(32, 32), mode="bilinear", align_corners=True)[:, 0]
    lam = lam / lam.sum((1, 2), keepdim=True) * 300.
    return torch.log1p(torch.poisson(lam, generator=gen)).reshape(n, 1024)


def prepare(case, seed):
    if case["kind"] in ("propose", "train"):
        net = ProposalNet(case["classes"], batch=256, seed=1 + seed % 1000)
        images = _images(case, seed).cpu().numpy()
        state = dict(case=case, net=net, images=images)
        if case["kind"] == "train":
            state["labels"] = np.random.default_rng(seed).integers(0, case["classes"], case["images"], dtype=np.int32)
            net.set_images(images)
        return state
    if case["kind"] == "slice":
        rng = np.random.default_rng(seed)
        qvals, corr, mask = _detector(case)
        c = Context(0)
        c.set_detector(qvals, corr, mask)
        model = _atoms(case["size"], False, 0., torch.Generator().manual_seed(seed)).cpu().numpy()[None]
        c.set_model(model)
        quat = rng.normal(size=4)
        return dict(case=case, ctx=c, quat=quat / np.linalg.norm(quat))
    inp = _inputs(case, seed)
    c = Context(0)
    if case["budget_mb"]:
        c.set_option("pair_budget_mb", case["budget_mb"])
    c.set_detector(inp["qvals"], inp["corr"], inp["mask"])
    c.set_frames(inp["ones"], inp["multi"], inp["po"], inp["pm"], inp["cm"])
    c.set_quaternions(inp["quats"])
    if case["two_d"]:
        c.set_model_type("2d")
    c.set_model(inp["model"])
    c.calc_beta(_beta(case), int(case["scaling"]))
    if case["coarse"]:
        c.set_refinement(inp["num_coarse"], inp["cells"], inp["relevant"])
    host = lambda a: torch.from_numpy(a.copy()).pin_memory().numpy()
    return dict(case=case, ctx=c, params=c.params(**_schedule(case)), start=inp["model"], scale=inp["scale"],
                model=host(inp["model"]), rmax=host(np.zeros(case["frames"], np.int32)),
                likelihood=host(np.zeros(case["frames"])))


def run(state):
    case = state["case"]
    if case["kind"] == "slice":
        return state["ctx"].slice_gen(state["quat"])
    if case["kind"] == "propose":
        state["net"].set_images(state["images"])
        return dict(cells=state["net"].topk(case["keep"]), logits=state["net"].logits())
    if case["kind"] == "train":
        grads, loss = state["net"].gradients(state["labels"])
        return dict(grads=grads, loss=loss)
    c = state["ctx"]
    np.copyto(state["model"], state["start"])
    if case["scaling"]:
        c.set_scale(state["scale"])
    ll, rms = c.run_iteration_host(state["params"], state["model"], 0., state["rmax"], state["likelihood"])
    out = dict(model=state["model"], rmax=state["rmax"], likelihood=state["likelihood"], mean=ll, change=rms)
    if case["scaling"]:
        out["scale"] = c.frame_params()["scale"]
    return out


def work(case):
    if case["kind"] == "slice":
        return dict(bytes=8. * (5. * _pixels(case) + 8. * _pixels(case)), flops=60. * _pixels(case))
    if case["kind"] in ("propose", "train"):
        macs = 1024 * 9 * 32 + 256 * 288 * 32 + 256 * 288 * 64 + 64 * 576 * 64 + 4096 * 256 + 256. * case["classes"]
        params = 4. * (9 * 32 + 288 * 32 + 288 * 64 + 576 * 64 + 4096 * 256 + 256. * case["classes"])
        n = case["images"]
        if case["kind"] == "propose":
            return dict(bytes=params + n * (4096. + 4. * case["keep"] + 4. * case["classes"]), flops=2. * macs * n)
        return dict(bytes=2. * params + 4096. * n, flops=6. * macs * n)
    M, N, P = case["modes"], case["frames"], _pixels(case)
    R = _orientations(case) * M
    voxels = M * float(case["size"]) ** (2 if case["two_d"] else 3)
    entries = N * min(float(P), case["photons"] * math.exp(SIGMA ** 2 / 2.))   # photons, about the sparse words
    pairs = R * entries
    if case["coarse"]:
        pairs *= 12. / _orientations(dict(case, div=case["coarse"]))
    corners = 4 if case["two_d"] else 8
    flops = 4. * pairs + R * float(P) * (15. + 2. * corners) + R * float(P) * (15. + 4. * corners)
    return dict(bytes=4. * entries + 16. * voxels + 8. * 5. * R + 8. * 5. * P + 28. * N, flops=flops)


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] in ("propose", "train"):
        return _exact_network(case, seed)
    if case["kind"] == "slice":
        rng = np.random.default_rng(seed)
        qvals, corr, _ = (torch.from_numpy(a).to(DEV) for a in _detector(case))
        model = _atoms(case["size"], False, 0., torch.Generator().manual_seed(seed))
        quat = rng.normal(size=4)
        quat = torch.from_numpy(quat / np.linalg.norm(quat)).to(DEV)[None]
        return _slices(model, quat, qvals, corr, False, TINY)[0].cpu().numpy()
    return _exact_iteration(case, _inputs(case, seed))


def _exact_network(case, seed):
    """Logits, or loss and gradients, in 64 bits without any rounding of weights or activations."""
    train = case["kind"] == "train"
    net = ProposalNet(case["classes"], batch=256, seed=1 + seed % 1000)
    flat = torch.from_numpy(net.params()).to(DEV).double().requires_grad_(train)
    net.close()
    logits = torch.cat([_forward(flat, x, case["classes"]) for x in _images(case, seed).split(256)])
    if not train:
        return dict(cells=None, logits=logits.cpu().numpy())
    labels = torch.from_numpy(np.random.default_rng(seed).integers(0, case["classes"], case["images"])).to(DEV)
    loss = torch.nn.functional.cross_entropy(logits, labels)
    loss.backward()
    return dict(grads=flat.grad.cpu().numpy(), loss=float(loss))


def _forward(flat, images, classes):
    x = images.double().reshape(-1, 1, 32, 32)
    at = 0
    for kind, cin, cout, stride in ((0, 1, 32, 1), (0, 32, 32, 2), (0, 32, 64, 1), (0, 64, 64, 2), (1, 4096, 256, 0),
                                    (1, 256, classes, 0)):
        fan = 9 * cin if kind == 0 else cin
        w, b = flat[at:at + cout * fan].reshape(cout, fan), flat[at + cout * fan:at + cout * fan + cout]
        at += cout * fan + cout
        if kind == 0:
            ho = x.shape[2] // stride
            pad = torch.nn.functional.pad(x, (1, 1, 1, 1))
            cols = torch.cat([pad[:, :, ky:ky + stride * ho:stride, kx:kx + stride * ho:stride]
                              for ky in range(3) for kx in range(3)], 1)
            x = (torch.einsum("ok,nkhw->nohw", w, cols) + b[:, None, None]).relu()
        else:
            x = x.permute(0, 2, 3, 1).reshape(x.shape[0], -1) if x.dim() == 4 else x
            x = x @ w.T + b
            x = x.relu() if cin == 4096 else x
    return x


def _csr(rows, cols, vals, shape):
    return torch.sparse_coo_tensor(torch.stack([rows, cols]), vals, shape).coalesce().to_sparse_csr()


def _exact_iteration(case, inp):
    size, two_d, M, N = case["size"], case["two_d"], case["modes"], case["frames"]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    qvals, corr, mask, quats = dev(inp["qvals"]), dev(inp["corr"]), dev(inp["mask"]), dev(inp["quats"])
    model, scale0 = dev(inp["model"]), dev(inp["scale"])
    P, n_rot = qvals.shape[0], quats.shape[0]
    R = n_rot * M
    frame = torch.arange(N, device=DEV)
    rows = torch.cat([torch.repeat_interleave(frame, dev(inp["ones"]).long()),
                      torch.repeat_interleave(frame, dev(inp["multi"]).long())])
    cols = torch.cat([dev(inp["po"]), dev(inp["pm"])]).long()
    cnt = torch.cat([torch.ones(inp["po"].size, dtype=torch.float64, device=DEV), dev(inp["cm"]).double()])
    good = mask[cols] == 0
    fcounts = torch.zeros(N, dtype=torch.float64, device=DEV).index_add_(0, rows[good], cnt[good])
    sum_fact = torch.zeros_like(fcounts).index_add_(0, rows[good], torch.lgamma(cnt[good] + 1.))
    by_frame = _csr(rows[good], cols[good], cnt[good], (N, P))
    keep = mask[cols] < 2
    by_pixel = _csr(cols[keep], rows[keep], cnt[keep], (P, N))
    del rows, cols, cnt, good, keep
    used = mask == 0
    block = max(1, min(512, int(3.5e7 / P)))
    ranges = [(m, b, min(n_rot, b + block)) for b in range(0, n_rot, block) for m in range(M)]

    # photon sums of every (orientation, frame) pair; orientation r = rotation * M + mode
    x = torch.empty(n_rot, M, N, dtype=torch.float64, device=DEV)
    u = torch.empty(n_rot, M, dtype=torch.float64, device=DEV)
    for m, b, e in ranges:
        w = _slices(model[m], quats[b:e], qvals, corr, two_d, TINY)
        if two_d:
            w = w.clamp(min=TINY)
        u[b:e, m] = w[:, used].sum(1)
        logs = torch.where(used, w.log(), torch.zeros_like(w))
        x[b:e, m] = (by_frame @ logs.T.contiguous()).T
    x, u = x.reshape(R, N), u.reshape(R)
    lw = quats[:, 4].log().repeat_interleave(M)
    rescale = fcounts.sum() / N / (quats[:, 4].repeat_interleave(M) * u).sum() * M
    par = _schedule(case)
    sd = scale0 if par["need_scaling"] and par["known_scale"] else rescale.expand(N)
    cells = dev(inp["cells"]).long() if case["coarse"] else None
    allowed = None
    if case["coarse"]:
        allowed = torch.zeros(N, inp["num_coarse"], dtype=torch.bool, device=DEV)
        allowed.scatter_(1, dev(inp["relevant"]).long(), True)

    # log-likelihoods, pruning and probabilities, a block of frames at a time
    beta = _beta(case)
    thr = 14. / beta
    like = torch.empty(N, dtype=torch.float64, device=DEV)
    psum_d = torch.empty_like(like)
    psum_r = torch.zeros(R, dtype=torch.float64, device=DEV)
    step = max(1, int(1e8 / R))
    index = torch.arange(R, device=DEV)[:, None]
    for b in range(0, N, step):
        e = min(N, b + step)
        y = x[:, b:e] + (lw[:, None] - u[:, None] * sd[None, b:e])
        if allowed is not None:
            y = torch.where(allowed[b:e].T[cells], y, torch.full_like(y, -math.inf))
        top = y.max(0).values
        first = (y == top).to(torch.uint8).argmax(0)
        kept = torch.where(index <= first, y > top - thr, y + thr > top)
        p = torch.where(kept, torch.exp(beta * (y - top)), torch.zeros_like(y))
        p /= p.sum(0)
        like[b:e] = torch.where(kept, p * y, torch.zeros_like(y)).sum(0) - sum_fact[b:e]
        psum_d[b:e] = rescale * (p * u[:, None]).sum(0)
        psum_r += (p * scale0[b:e] if par["need_scaling"] else p).sum(1)
        x[:, b:e] = torch.where(p > 1e-6, p, torch.zeros_like(p))
    x, psum_r = x.reshape(n_rot, M, N), psum_r.reshape(n_rot, M)

    # tomograms and merge
    V = size ** (2 if two_d else 3)
    total = torch.zeros(M, V, dtype=torch.float64, device=DEV)
    weight = torch.zeros_like(total)
    pix = (mask <= 1).nonzero()[:, 0]
    for m, b, e in ranges:
        live = (psum_r[b:e, m] > 0).nonzero()[:, 0]
        if not live.numel():
            continue
        view = (by_pixel @ x[b:e, m][live].T.contiguous()).T[:, pix] / psum_r[b:e, m][live][:, None] / corr[pix]
        cor, ok = _corners(_positions(quats[b:e][live], qvals[pix], size, two_d), size)
        for i, w in cor:
            w = torch.where(ok, w, torch.zeros_like(w)).reshape(-1)
            i = i.reshape(-1)
            total[m].index_add_(0, i, w * view.reshape(-1))
            weight[m].index_add_(0, i, w)

    # model update
    if not two_d:
        lo = 1 - size % 2
        s, w = (t.reshape(M, size, size, size)[:, lo:, lo:, lo:] for t in (total, weight))
        both = w + w.flip(1, 2, 3)
        avg = torch.where(both > 0, (s * w + (s * w).flip(1, 2, 3)) / both, torch.zeros_like(s))
        s.copy_(avg)
    new = torch.where(weight > 0, total / weight, total).reshape(model.shape)
    change = float(((new - model) ** 2).sum().div(M * V).sqrt())
    out = dict(rmax=None, likelihood=like.cpu().numpy(), mean=float(like.sum() / N))
    if case["scaling"]:
        scale = fcounts / psum_d
        if not two_d:
            mean = scale.sum() / N
            new[0] *= mean
            scale = scale / mean
            change *= float(mean)
        out["scale"] = scale.cpu().numpy()
    out.update(model=new.cpu().numpy(), change=change)
    return out
