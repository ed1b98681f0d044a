"""The work a user has the framework do, as cases that can be timed and compared: the spiking brain
(`Brain.step`), the optic lobe's substeps (`OpticCore.substeps`), its gradients (`OpticRollout`), the
eye's ray tracer (`BatchWorld.column_radiance`) and the whole fly (`WholeFly.step`), at the sizes of
the benchmark's configurations and below. Graphs come from `flyb200.synthetic` with a fixed seed (a
user has one connectome); states, held inputs and poses come from the case's seed."""
import functools
import math
import pathlib
import sys

import numpy as np
import torch

sys.path.insert(0, str(pathlib.Path(__file__).resolve().parent.parent / "flyverse-core_b200"))

from flyb200 import autotune, synthetic  # noqa: E402
from flyb200.adjoint import OpticAdjoint, OpticRollout  # noqa: E402
from flyb200.batch_world import BatchWorld  # noqa: E402
from flyb200.brain import Brain, LIFParams  # noqa: E402
from flyb200.optic import OpticCore  # noqa: E402
from flyb200.whole import WholeFly  # noqa: E402
from flyb200.world import MATERIALS, make_room  # noqa: E402

LANES = 4_294_967_296                       # 2^32
LARGEST_STEPS = 71_618 * 64 * 40            # neuron-steps of the largest brain case


def listed():
    return [
        # a circuit model, one fly, a 10 ms frame of 0.1 ms steps: nothing but latency
        dict(name="brain 2k x1", kind="brain", n=2_000, edges=20_000, cells=50, hz=150.0, batch=1, steps=100, dt=0.1,
             plastic=False, delivery=""),
        # the full spiking tier of one fly, half a frame: an interactive run
        dict(name="brain 72k x1", kind="brain", n=71_618, edges=15_000_000, cells=2_000, hz=100.0, batch=1, steps=50,
             dt=0.1, plastic=False, delivery=""),
        # a parameter sweep over 64 flies at dense firing, with the launch a user's tuning settled on
        dict(name="brain 72k x64", kind="brain", n=71_618, edges=15_000_000, cells=2_000, hz=100.0, batch=64, steps=40,
             dt=0.1, plastic=False, delivery="staged-pull"),
        # adapting cells with depressing synapses at the frame loop's 0.5 ms step, an odd number of flies
        dict(name="brain plastic 20k x11", kind="brain", n=20_011, edges=4_000_000, cells=500, hz=100.0, batch=11, steps=20,
             dt=0.5, plastic=True, delivery=""),
        # one frame (ten 1 ms substeps) of the full optic lobe for one fly, a ragged group and a full batch
        dict(name="lobe 89k x1", kind="lobe", m=89_390, nnz=6_000_000, batch=1, steps=10),
        dict(name="lobe 89k x12", kind="lobe", m=89_390, nnz=6_000_000, batch=12, steps=10),
        dict(name="lobe 89k x64", kind="lobe", m=89_390, nnz=6_000_000, batch=64, steps=10),
        # fitting pair gains and time constants: one full lobe, and a small lobe over a batch of stimuli
        dict(name="gradient 89k x1", kind="gradient", m=89_390, nnz=6_000_000, batch=1, steps=60),
        dict(name="gradient 20k x16", kind="gradient", m=20_000, nnz=1_340_000, batch=16, steps=40),
        # what every fly sees this frame, for one fly and for the batch
        dict(name="eye x1", kind="eye", radius=16, batch=1),
        dict(name="eye x64", kind="eye", radius=16, batch=64),
        # the coupled fly of the benchmark, two steps a call from a captured graph
        dict(name="whole fly x64", kind="fly", batch=64, steps=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("brain", "brain", "lobe", "lobe", "gradient", "eye"))
    if kind == "brain":
        n = _log(rng, 500, 71_618)
        dt = rng.choice((0.1, 0.1, 0.5))
        plastic = rng.random() < 0.3
        pull = not plastic and dt == 0.1 and rng.random() < 0.3      # pull delivery: 32 or 64 flies
        batch = rng.choice((32, 64)) if pull else _log(rng, 1, 64)
        steps = max(10, min(rng.randint(15, 50), LARGEST_STEPS // (n * batch)))
        return dict(kind=kind, n=n, edges=int(n * _log(rng, 10, 209)), cells=max(10, n // 36), hz=float(rng.randint(20, 200)),
                    batch=batch, steps=steps, dt=dt, plastic=plastic, delivery="staged-pull" if pull else "")
    if kind == "lobe":
        m = _log(rng, 2_000, 89_390)
        return dict(kind=kind, m=m, nnz=int(m * rng.uniform(20, 67)), batch=_log(rng, 1, 64), steps=rng.randint(5, 10))
    if kind == "gradient":
        m = _log(rng, 2_000, 89_390)
        batch = _log(rng, 1, max(1, min(32, 400_000 // m)))
        return dict(kind=kind, m=m, nnz=int(m * rng.uniform(20, 67)), batch=batch, steps=rng.randint(15, 50))
    return dict(kind=kind, radius=rng.randint(3, 16), batch=_log(rng, 1, 64))


# ------------------------------------------------------------------ graphs (built once per size)
@functools.lru_cache(maxsize=4)
def _spiking(n, edges, cells, hz):
    return synthetic.lif_config2(seed=0, n=n, edges=edges, n_poisson=cells, poisson_hz=hz)


@functools.lru_cache(maxsize=4)
def _lobe(m, nnz):
    return synthetic.optic_config3(seed=0, m=m, nnz=nnz, n_types=min(700, m // 4), n_spk=max(100, m // 2))


@functools.lru_cache(maxsize=1)
def _whole():
    return synthetic.whole_fly_config5(seed=0)


def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


# ------------------------------------------------------------------ the spiking brain
def _lif_params(case, base):
    more = dict(base, dt=case["dt"])
    if case["plastic"]:
        more.update(adapt_jump=1.5, std_u=0.2)
    return LIFParams(**more)


def _active_state(n, batch, seed):
    """Membranes spread below threshold, synaptic drive decaying from recent input, per-fly current: (B, n) each."""
    g = _rng(seed)
    v = -52.0 + 6.9 * torch.rand(batch, n, generator=g, device="cuda")
    syn = 18.0 * torch.rand(batch, n, generator=g, device="cuda")
    cur = 2.0 + 4.0 * torch.rand(batch, 1, generator=g, device="cuda").expand(batch, n)
    return v, syn, cur


def _set_active(brain, seed):
    v, syn, cur = _active_state(brain.n, brain.B, seed)
    brain.v, brain.g, brain.drive = v, syn, cur


def _prepare_brain(case, seed):
    cfg = _spiking(case["n"], case["edges"], case["cells"], case["hz"])
    brain = Brain(cfg.c, _lif_params(case, cfg.params), device="cuda", seed=seed, batch=case["batch"])
    brain.record_activity = True
    brain.set_poisson(cfg.poisson_idx, case["hz"])
    if case["delivery"]:        # install the launch that tuning chose for this density of spikes
        autotune.tune_lif(brain, steps=2, candidates=(("step", 128, 2, case["delivery"]),))
    _set_active(brain, seed)
    return brain, case["steps"]


def _run_brain(state):
    brain, steps = state
    brain.step(steps)
    return dict(v=brain.v, g=brain.g, rate=brain.rate, adapt=brain.adapt, res=brain.res, refrac=brain.refrac,
                spikes=brain.spikes, counts=brain.spike_counts, pending=brain.ring)


def _work_brain(case):
    """State and pending input once each way per call, a step's ring slot read and its spike bits
    written per step, the spikes' synapses (at about 1 % of the cells per step) read and delivered."""
    items, s = case["n"] * case["batch"], case["steps"]
    events = 0.01 * s * case["batch"] * case["edges"]
    ring = 8 if case["plastic"] else 4
    return dict(bytes=items * (4.0 * 17 + s * (ring + 0.125)) + case["edges"] * 8.0 + events * ring,
                flops=items * s * 20.0 + events)


def _philox(seed, step, neuron, fly):
    """24-bit uniforms of Philox4x32-10 (Salmon et al., SC'11) for counter (step, neuron, fly) and key `seed`."""
    low = np.uint64(LANES - 1)
    c = [np.uint64(step & (LANES - 1)), np.uint64(step >> 32), neuron.astype(np.uint64), fly.astype(np.uint64)]
    c = [np.broadcast_to(x, np.broadcast_shapes(neuron.shape, fly.shape)) for x in c]
    k0, k1 = np.uint64(seed & (LANES - 1)), np.uint64(seed >> 32)
    for r in range(10):
        if r:
            k0, k1 = (k0 + np.uint64(0x9E3779B9)) & low, (k1 + np.uint64(0xBB67AE85)) & low
        p, q = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(q >> np.uint64(32)) ^ c[1] ^ k0, q & low, (p >> np.uint64(32)) ^ c[3] ^ k1, p & low]
    return (c[0] >> np.uint64(8)).astype(np.float64) / 2**24


def _csr64(M):
    M = M.tocsr()
    return torch.sparse_csr_tensor(torch.from_numpy(M.indptr.astype(np.int64)), torch.from_numpy(M.indices.astype(np.int64)),
                                   torch.from_numpy(M.data.astype(np.float64)), M.shape, device="cuda",
                                   check_invariants=False)


def _exact_brain(case, seed):
    """The leaky integrate-and-fire equations step by step in 64 bits; the refractory timer counts
    down in its own 32-bit steps of dt. No value for the pending-input ring (whole numbers)."""
    cfg = _spiking(case["n"], case["edges"], case["cells"], case["hz"])
    p = _lif_params(case, cfg.params)
    v, g, cur = (x.double().t().contiguous() for x in _active_state(case["n"], case["batch"], seed))
    W = _csr64(cfg.c.W)
    delay = round(p.delay / p.dt)
    a_m, a_s, a_r = (math.exp(-p.dt / t) for t in (p.tau_m, p.tau_syn, p.rate_tau))
    a_ad, a_res = math.exp(-p.dt / p.adapt_tau) if p.adapt_jump else 0.0, math.exp(-p.dt / p.std_tau)
    rate, adapt, counts, res = torch.zeros_like(v), torch.zeros_like(v), torch.zeros_like(v), torch.ones_like(v)
    refrac = torch.zeros_like(v, dtype=torch.float32)
    cells = torch.from_numpy(cfg.poisson_idx).cuda()
    prob = float(np.float32(case["hz"]) * np.float32(p.dt / 1000.0))
    sent = []
    for s in range(case["steps"]):
        g = g * a_s + (p.w_syn * (W @ sent[s - delay]) if s >= delay else 0.0)
        target = p.v_rest + g + cur - adapt
        v = target + (v - target) * a_m
        v[refrac > 0] = p.v_reset
        refrac = (refrac - p.dt).clamp(min=0.0)
        spike = (v >= p.v_th).double()
        draws = _philox(seed, s, cfg.poisson_idx[:, None], np.arange(case["batch"])[None, :])
        spike[cells] = torch.maximum(spike[cells], (torch.from_numpy(draws) < prob).double().cuda())
        fired = spike > 0
        v[fired], refrac[fired] = p.v_reset, p.t_ref
        adapt = adapt * a_ad + spike * p.adapt_jump
        sent.append(spike * res)
        if s >= delay:
            sent[s - delay] = None
        if p.std_u:
            res = 1.0 - (1.0 - res * (1.0 - p.std_u * spike)) * a_res
        counts += spike
        rate = rate * a_r + spike * (1.0 - a_r) * 1000.0 / p.dt
    return dict(v=v.t(), g=g.t(), rate=rate.t(), adapt=adapt.t(), res=res.t(), refrac=refrac.double().t(), spikes=spike.t(),
                counts=counts.t(), pending=None)


# ------------------------------------------------------------------ the optic lobe
def _lobe_state(m, batch, seed):
    """v, adapt, held photoreceptor and feedback input of a lobe at work, [m][batch] each."""
    g = _rng(seed)
    scale = (0.25, 0.05, 0.2, 0.05)
    return [s * torch.randn(m, batch, generator=g, device="cuda") for s in scale]


def _prepare_lobe(case, seed):
    o = _lobe(case["m"], case["nnz"])
    core = OpticCore(o.W_rr(), o.a, o.b, batch=case["batch"], device="cuda", gain_rr=o.gain_rr, adapt_gain=o.adapt_gain,
                     aad=o.aad)
    for to, x in zip((core.v_s, core.adapt_s, core.pr_in, core.spk_in), _lobe_state(o.m, case["batch"], seed)):
        to.copy_(x)
    return core, case["steps"]


def _run_lobe(state):
    core, steps = state
    core.substeps(steps)
    return dict(v=core.v_s, adapt=core.adapt_s, dr=core.dr_out)


def _exact_lobe(case, seed):
    o = _lobe(case["m"], case["nnz"])
    v, ad, pr, spk = (x.double() for x in _lobe_state(o.m, case["batch"], seed))
    W = _csr64(o.W_rr())
    a, b = (torch.from_numpy(x.astype(np.float64)).cuda()[:, None] for x in (o.a, o.b))
    dr = (v + b).clamp(0, 1) - b
    for _ in range(case["steps"]):
        inp = o.gain_rr * (W @ dr) + pr - o.adapt_gain * ad + spk
        v = inp + (v - inp) * a
        ad = dr + (ad - dr) * o.aad
        dr = (v + b).clamp(0, 1) - b
    return dict(v=v, adapt=ad, dr=dr)


def _work_lobe(case):
    units = case["m"] * case["batch"]
    return dict(bytes=case["steps"] * (case["nnz"] * 8.0 + case["m"] * 12.0 + units * 32.0),
                flops=case["steps"] * (2.0 * case["nnz"] * case["batch"] + 12.0 * units))


# ------------------------------------------------------------------ gradients of the lobe
def _fit_state(o, case, seed):
    v0, ad0, pr, spk = _lobe_state(o.m, case["batch"], seed)
    g = _rng(seed + 1_000_003)
    gains = torch.from_numpy(o.gain0).cuda() * (0.8 + 0.4 * torch.rand(len(o.gain0), generator=g, device="cuda"))
    tau = torch.from_numpy(o.tau_of_type).cuda() * (0.9 + 0.2 * torch.rand(o.n_types, generator=g, device="cuda"))
    cot = torch.randn(o.m, case["batch"], generator=g, device="cuda")
    return v0, 0.4 * ad0, pr, spk, gains, tau, cot


def _prepare_gradient(case, seed):
    o = _lobe(case["m"], case["nnz"])
    v0, ad0, pr, spk, gains, tau, cot = _fit_state(o, case, seed)
    engine = OpticAdjoint(o.W0, o.pair_id, len(o.gain0), o.type_of, o.n_types, o.b, pr, spk, dt_ms=o.dt_ms,
                          batch=case["batch"], adapt_tau_ms=o.adapt_tau_ms, checkpoint=20)
    leaves = [x.requires_grad_() for x in (gains, tau, v0, ad0)]
    return engine, leaves, cot, case["steps"]


def _run_gradient(state):
    engine, leaves, cot, steps = state
    v, ad = OpticRollout.apply(*leaves, engine, steps)
    d_gains, d_tau, d_v0, d_ad0 = torch.autograd.grad(v, leaves, cot)
    return dict(v=v.detach(), adapt=ad.detach(), d_gains=d_gains, d_tau=d_tau, d_v0=d_v0, d_adapt0=d_ad0)


def _exact_gradient(case, seed):
    o = _lobe(case["m"], case["nnz"])
    v0, ad0, pr, spk, gains, tau, cot = (x.double() for x in _fit_state(o, case, seed))
    leaves = [x.requires_grad_() for x in (gains, tau, v0, ad0)]
    row = torch.from_numpy(np.repeat(np.arange(o.m), np.diff(o.W0.indptr))).cuda()
    col = torch.from_numpy(o.W0.indices.astype(np.int64)).cuda()
    w0 = torch.from_numpy(o.W0.data.astype(np.float64)).cuda()
    w = (gains[torch.from_numpy(o.pair_id.astype(np.int64)).cuda()] * w0)[:, None]
    a = torch.exp(-o.dt_ms / tau[torch.from_numpy(o.type_of.astype(np.int64)).cuda()])[:, None]
    b = torch.from_numpy(o.b.astype(np.float64)).cuda()[:, None]

    def substep(v, ad, w, a):
        dr = (v + b).clamp(0, 1) - b
        rec = torch.zeros_like(v).index_add(0, row, w * dr[col])
        inp = o.gain_rr * rec + pr - o.adapt_gain * ad + spk
        return inp + (v - inp) * a, dr + (ad - dr) * o.aad

    v, ad = v0, ad0
    for _ in range(case["steps"]):      # each substep is run again in the backward pass: memory for one at a time
        v, ad = torch.utils.checkpoint.checkpoint(substep, v, ad, w, a, use_reentrant=False)
    d_gains, d_tau, d_v0, d_ad0 = torch.autograd.grad(v, leaves, cot)
    return dict(v=v.detach(), adapt=ad.detach(), d_gains=d_gains, d_tau=d_tau, d_v0=d_v0, d_adapt0=d_ad0)


def _work_gradient(case):
    """The rollout, and per reversed substep the matrix, its gradient accumulator both ways and the state."""
    f, units = _work_lobe(case), case["m"] * case["batch"]
    return dict(bytes=f["bytes"] + case["steps"] * (case["nnz"] * 16.0 + units * 32.0),
                flops=f["flops"] + case["steps"] * (4.0 * case["nnz"] * case["batch"] + 12.0 * units))


# ------------------------------------------------------------------ the eye
@functools.lru_cache(maxsize=4)
def _eye(radius):
    return synthetic.eye_grid(radius)[1:]


def _prepare_eye(case, seed):
    world = BatchWorld([make_room(b)[0] for b in range(case["batch"])], device="cuda")
    world.set_eye(*_eye(case["radius"]))
    return world, synthetic.fly_poses(case["batch"], seed=seed)


def _run_eye(state):
    world, poses = state
    return world.column_radiance(*poses)


def _nearest(w, o, d):
    """t, unit normal and object number of the nearest hit of rays o + t d (M, 3), t = 1e9 for none."""
    M = len(d)
    rows = torch.arange(M, device="cuda")
    ts, ns = [], []

    def per_object(items, *fields):
        return [torch.tensor([getattr(x, f) for x in items], dtype=torch.float64, device="cuda") for f in fields]

    c, r = per_object(w.spheres, "center", "radii")
    oc, dd = (o[:, None] - c) / r, d[:, None] / r
    a, b, e = (dd * dd).sum(-1), 2 * (oc * dd).sum(-1), (oc * oc).sum(-1) - 1
    disc = b * b - 4 * a * e
    sq = disc.clamp(min=0).sqrt()
    t0, t1 = (-b - sq) / (2 * a), (-b + sq) / (2 * a)
    t = torch.where(t0 > 1e-4, t0, t1)
    ts.append(torch.where((disc > 0) & (t > 1e-4), t, 1e9))
    k = ts[-1].argmin(1)
    n = (o + d * ts[-1][rows, k][:, None] - c[k]) / r[k] ** 2
    ns.append(n / n.norm(dim=1, keepdim=True).clamp(min=1e-9))
    lo, hi = per_object(w.boxes, "lo", "hi")
    inv = 1 / torch.where(d.abs() < 1e-9, 1e-9, d)
    x, y = (lo - o[:, None]) * inv[:, None], (hi - o[:, None]) * inv[:, None]
    enter, axis = torch.minimum(x, y).max(-1)
    leave = torch.maximum(x, y).min(-1).values
    ts.append(torch.where((leave > enter) & (enter > 1e-4), enter, 1e9))
    k = axis[rows, ts[-1].argmin(1)]
    ns.append(-torch.nn.functional.one_hot(k, 3) * torch.sign(d))
    pt, pn = per_object(w.planes, "point", "normal")
    den = d @ pn.t()
    t = ((pt - o[:, None]) * pn).sum(-1) / torch.where(den.abs() < 1e-9, 1e-9, den)
    ts.append(torch.where((t > 1e-4) & (den.abs() > 1e-9), t, 1e9))
    k = ts[-1].argmin(1)
    ns.append(torch.where((den[rows, k] > 0)[:, None], -pn[k], pn[k]))
    t, k = torch.cat(ts, 1).min(1)
    kind = (k >= len(c)).long() + (k >= len(c) + len(lo)).long()
    return t, torch.stack(ns)[kind, rows], k


def _noise(p, period):
    """Trilinear value noise of a lattice hash."""
    q = p / period
    i, f = q.floor().long(), q - q.floor()
    f = f * f * (3 - 2 * f)
    out = 0.0
    for x, y, z in ((x, y, z) for x in (0, 1) for y in (0, 1) for z in (0, 1)):
        h = ((i[:, 0] + x) * 374761393 + (i[:, 1] + y) * 668265263 + (i[:, 2] + z) * 2147483647) % 2147483647
        h = ((h ^ (h >> 13)) * 1274126177) % 2147483647
        value = (h & 65535).double() / 32768 - 1
        wx, wy, wz = (f[:, c] if s else 1 - f[:, c] for c, s in enumerate((x, y, z)))
        out = out + wx * wy * wz * value
    return out


def _shade(w, o, d):
    t, n, k = _nearest(w, o, d)
    p = o + d * t[:, None]
    to = torch.tensor(w.light_pos, dtype=torch.float64, device="cuda") - p
    dist = to.norm(dim=1)
    ray = to / dist[:, None].clamp(min=1e-9)
    lit = (_nearest(w, p + n * 1e-3, ray)[0] >= dist).double()
    shine = (n * ray).sum(1).clamp(min=0) * lit * 4 / (1 + dist * dist)
    mats = [MATERIALS[x.material] for x in (*w.spheres, *w.boxes, *w.planes)]
    table = {f: torch.tensor([getattr(m, f) for m in mats], dtype=torch.float64, device="cuda")[k.clamp(max=len(mats) - 1)]
             for f in ("refl", "refl2", "emit", "scale", "pattern")}
    fx, fy = (p[:, c].div(table["scale"]).floor() for c in (0, 1))
    kinds = [torch.zeros_like(lit, dtype=torch.bool), (fx + fy) % 2 == 1,
             torch.where(n[:, 0].abs() > 0.5, fy, fx) % 2 == 1, (fy % 2 == 1) | ((fx + 3 * fy) % 7 == 0)]
    second = torch.stack(kinds)[table["pattern"].long(), torch.arange(len(d), device="cuda")]
    refl = torch.where(second[:, None], table["refl2"], table["refl"])
    grain = 0.5 * _noise(p, 0.02) + 0.3 * _noise(p, 0.008) + 0.2 * _noise(p, 0.003)
    refl = refl * (1 + w.detail * grain).clamp(min=0.1)[:, None]
    colour, ambient = (torch.tensor(x, dtype=torch.float64, device="cuda") for x in (w.light_color, w.ambient))
    return torch.where((t < 1e9)[:, None], refl * (ambient + colour * shine[:, None]) + table["emit"], 0.0)


def _exact_eye(case, seed):
    dirs, weights = (torch.as_tensor(np.asarray(x, np.float64), device="cuda") for x in _eye(case["radius"]))
    out = []
    for b, pose in enumerate(zip(*synthetic.fly_poses(case["batch"], seed=seed))):
        eye, *axes = (torch.as_tensor(x, dtype=torch.float64, device="cuda") for x in pose)
        rays = dirs.reshape(-1, 3) @ torch.stack(axes)
        rad = _shade(make_room(b)[0], eye.expand_as(rays), rays)
        out.append((rad.reshape(len(dirs), -1, 4) * weights.reshape(1, -1, 1)).sum(1))
    return torch.stack(out)


def _work_eye(case):
    """Rays against a room of 34 objects, once to the eye and once to the light, and three octaves of noise."""
    columns = 2 * (3 * case["radius"] * (case["radius"] + 1) + 1)
    rays = columns * 7 * case["batch"]
    return dict(bytes=columns * case["batch"] * 16.0 + columns * 7 * 24.0, flops=rays * (2 * 34 * 20.0 + 3 * 100.0))


# ------------------------------------------------------------------ the whole fly
def _prepare_fly(case, seed):
    cfg = _whole()
    fly = WholeFly(cfg, case["batch"], device="cuda", seed=seed)
    autotune.tune_lif(fly.lif, steps=2, candidates=(("step", 128, 2, "staged-pull"),))
    fly.set_radiance(torch.from_numpy(cfg.optic.grating(0.0, case["batch"], seed=seed)).cuda(), 0.1)
    _set_active(fly.lif, seed)
    for to, x in zip((fly.optic.v_s, fly.optic.adapt_s), _lobe_state(cfg.optic.m, case["batch"], seed)):
        to.copy_(x)
    fly.step(1)                  # the carried optic state of a running fly
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream), torch.cuda.graph(graph, stream=stream):
        fly.step(case["steps"])
    torch.cuda.current_stream().wait_stream(stream)
    return fly, graph


def _run_fly(state):
    fly, graph = state
    graph.replay()
    lif, optic = fly.lif, fly.optic
    return dict(v=lif.v, g=lif.g, rate=lif.rate, drive=lif.drive, spikes=lif.spikes, optic_v=optic.v_s, optic_adapt=optic.adapt_s)


def _work_fly(case):
    """One step of 77,716 spiking and 89,390 graded cells over 25.6 M synapses, with the spikes and
    rates of every step visible to the other half of the fly."""
    spiking, units = 77_716 * case["batch"], 89_390 * case["batch"]
    per_step = spiking * 60.0 + units * 32.0 + 6_000_000 * 8.0 + 19_316_403 * 4.0
    return dict(bytes=case["steps"] * per_step, flops=case["steps"] * (spiking * 20.0 + units * 12.0 + 2.0 * 6_000_000 * case["batch"]))


# ------------------------------------------------------------------ by kind
KINDS = {
    "brain": (_prepare_brain, _run_brain, _work_brain, _exact_brain),
    "lobe": (_prepare_lobe, _run_lobe, _work_lobe, _exact_lobe),
    "gradient": (_prepare_gradient, _run_gradient, _work_gradient, _exact_gradient),
    "eye": (_prepare_eye, _run_eye, _work_eye, _exact_eye),
    # the coupled fly couples a chaotic spike train to sums in 32 bits: no value in 64 bits
    "fly": (_prepare_fly, _run_fly, _work_fly, None),
}


def prepare(case, seed):
    return case["kind"], KINDS[case["kind"]][0](case, int(seed))


def run(state):
    kind, held = state
    return KINDS[kind][1](held)


def work(case):
    return KINDS[case["kind"]][2](case)


def exact(case, seed):
    fn = KINDS[case["kind"]][3]
    return None if fn is None else fn(case, int(seed))
