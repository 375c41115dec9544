"""The calls whose time this repository is measured by.

Each case is one call (or the few calls a program makes in a row) through the
public entry points of ``wgdna``: the C ABI of ``include/wgdna.h`` as the
ctypes binding declares it, or the Python functions above it.  ``prepare``
makes what the program holds before the call (a context, an earlier stage's
result on the device, a network's parameters), ``run`` is the call.

Operations:

* ``transport``  Phase A + B on the device; results, dose grid and rad_buf
* ``irt``        IRT chemistry on the rad_buf the transport left on the device
* ``track``      IRT chemistry of a host rad_buf: synthetic spur tracks
* ``batch``      transport, IRT and direct SSB + DSB scoring in a row
* ``validate``   run_at_energy with device chemistry and damage scoring, host
                 readbacks included (one row of run_validation)
* ``data``       surrogate.track_data: transport, descriptors, IRT with curves
* ``chemistry``  the surrogate's G(t) of the tracks of a transport
* ``predict``    surrogate.predict on host descriptors
* ``train``      surrogate training from fresh weights on loaded data
* ``score``      direct SSB + DSB scoring of the rad_buf on the device
* ``grid``       the grid-hash chemistry, positions and alive flags read back
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "webgpu-dna_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import wgdna  # noqa: E402
from wgdna import _lib, app, chemistry, dispatch, surrogate, synthetic  # noqa: E402

LCG0 = 0x12345678          # the scoring generator's start (makeSsbRng)
VC = 128                   # dose grid edge
# rad_buf entries and electron steps per eV of primary energy (10 keV: 1294
# entries and 7.7 k steps per primary), for the estimates of work()
ENTRIES_PER_EV, STEPS_PER_EV = 0.1294, 0.77
HITS_BYTES = 2 * 441 * 8823


def listed():
    return [
        # the smallest call of the ESTAR sweep: a handful of short tracks, a quick check
        {"name": "transport-100eV", "op": "transport", "np": 64, "lo": 100.0, "hi": 100.0, "dna": 0, "ce": 7.4,
         "box": 15000.0},
        # the transport of the headline workload
        {"name": "transport-10keV", "op": "transport", "np": 4096, "lo": 10000.0, "hi": 10000.0, "dna": 1, "ce": 7.5,
         "box": 15000.0},
        # the chemistry of the headline workload
        {"name": "irt-10keV", "op": "irt", "np": 4096, "lo": 10000.0, "hi": 10000.0, "ce": 7.5, "box": 15000.0},
        # the single-track workload: one 2.7 um track of 510 spurs from host memory
        {"name": "track-510", "op": "track", "tracks": 1, "spurs": 510},
        # a source spectrum in one launch (the mixed-energy workload), the largest call
        {"name": "batch-mixed", "op": "batch", "np": 65536, "lo": 100.0, "hi": 30000.0, "dna": 0, "ce": 7.5,
         "box": 15000.0},
        # the validation run's 10 keV row, as the application calls it
        {"name": "validate-10keV", "op": "validate", "np": 4096, "ce": 7.4, "box": 15000.0},
        # one batch of training data of the surrogate
        {"name": "data-1keV", "op": "data", "np": 4096, "lo": 1000.0, "hi": 1000.0, "ce": 7.5, "box": 15000.0},
        # the surrogate in place of the IRT (the damage sweep's chemistry step)
        {"name": "chemistry-10keV", "op": "chemistry", "np": 4096, "lo": 10000.0, "hi": 10000.0, "ce": 7.5,
         "box": 15000.0},
        # the surrogate on stored descriptors: the three held-out batches of one energy
        {"name": "predict-12288", "op": "predict", "rows": 12288},
        # two epochs of surrogate training at the recipe's batch size
        {"name": "train-16384", "op": "train", "rows": 16384, "batch": 1024, "epochs": 2},
        # the damage scoring of the headline workload
        {"name": "score-10keV", "op": "score", "np": 4096, "lo": 10000.0, "hi": 10000.0, "ce": 7.5, "box": 15000.0},
        # the other chemistry backend on one batch of short tracks
        {"name": "grid-1keV", "op": "grid", "np": 4096, "lo": 1000.0, "hi": 1000.0, "ce": 7.5, "box": 15000.0},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    op = rng.choice(["transport", "transport", "irt", "irt", "track", "batch", "batch", "validate", "data", "chemistry",
                     "predict", "train", "score", "grid"])
    if op == "track":
        return {"op": op, "tracks": rng.randint(1, 24), "spurs": int(_log(rng, 8, 511))}
    if op == "predict":
        return {"op": op, "rows": int(_log(rng, 1, 65536))}
    if op == "train":
        rows = int(_log(rng, 1000, 40000))
        return {"op": op, "rows": rows, "batch": min(rows, rng.choice([256, 512, 1000, 1024, 2048])), "epochs": 1}
    ce, box = rng.choice([7.4, 7.5]), rng.choice([15000.0, 15000.0, 400.0])
    if op == "validate":
        return {"op": op, "np": int(_log(rng, 64, 4096)), "ce": ce, "box": 15000.0}
    # one energy or a spectrum; at most the 10 keV workload's energy in all
    e = round(_log(rng, 100.0, 30000.0), 1)
    if op == "grid":
        # all tracks start at the origin, whose cells hold most of the pairs: at
        # most the listed 4096 tracks, and enough radicals that the yields do not
        # depend on single reactions
        e = round(_log(rng, 1000.0, 20000.0), 1)
        n = int(_log(rng, 2e6 / e, 4.1e6 / e))
        return {"op": op, "np": n, "lo": e, "hi": e, "ce": ce, "box": 15000.0}
    lo, hi = (e, e) if rng.random() < 0.6 else (100.0, max(e, 200.0))
    n = int(_log(rng, 16, max(32.0, min(16384.0, 4.1e7 / hi))))
    case = {"op": op, "np": n, "lo": lo, "hi": hi, "ce": ce, "box": box}
    if op in ("transport", "batch"):
        case["dna"] = rng.randint(0, 1)
    return case


# ------------------------------------------------------------------ inputs
def _context(case):
    """A context sized as the benchmark sizes it: rad_buf and secondaries from the batch's energy."""
    ev = case["np"] * case["hi"] if case["lo"] == case["hi"] else case["np"] * 1.4 * _mean(case)
    return wgdna.Context(max_primaries=case["np"], max_rad=max(int(ev * 0.16), 1_000_000),
                         max_sec=max(int(ev * 0.03), 100_000))


def _mean(case):
    lo, hi = case["lo"], case["hi"]
    return lo if lo == hi else (hi - lo) / math.log(hi / lo)


class _Buffer:
    """A device buffer of a context as torch sees it; it keeps the context, which owns the memory."""

    def __init__(self, ctx, ptr, n, typestr):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": (int(n),), "typestr": typestr, "data": (int(ptr), False), "version": 3}


def device_tensor(ctx, ptr, n, typestr):
    return torch.as_tensor(_Buffer(ctx, ptr, n, typestr), device="cuda")


def _views(ctx, n):
    """The context's device buffers: results, dose grid, rad_buf (rows past the stored entries stay zero), hit bytes."""
    v = _lib.DeviceView()
    _lib.check("wgdna_device_views", _lib.lib().wgdna_device_views(ctx.h, C.byref(v)))
    rad = device_tensor(ctx, v.rad, 4 * ctx.max_rad, "<f4").view(-1, 4).zero_()
    return {"results": device_tensor(ctx, v.results, 8 * n, "<f4").view(n, 8),
            "dose": device_tensor(ctx, v.dose, v.dose_words, "<i4"), "rad": rad,
            "hits": device_tensor(ctx, v.hits, v.hits_bytes, "|u1")}


def _transport_state(case, seed):
    ctx = _context(case)
    n, lo, hi = case["np"], case["lo"], case["hi"]
    p = wgdna.transport_params(n, hi, case["box"], case["ce"], dna=wgdna.build_dna_target(), seed=seed,
                               dna_enable=case.get("dna", 0))
    st = {"ctx": ctx, "p": p, "stats": _lib.TransportStats(), "op": case["op"], "E": _mean(case)}
    if lo != hi:
        st["energies"] = torch.from_numpy(synthetic.mixed_energies(n, lo, hi, key=seed)).pin_memory()
        p.E_per_primary = st["energies"].data_ptr()
    st |= _views(ctx, n)
    torch.cuda.synchronize()
    return st


def _transport(st):
    _lib.check("wgdna_transport", _lib.lib().wgdna_transport(st["ctx"].h, C.byref(st["p"]), C.byref(st["stats"])))


def _network(seed):
    """Parameters (W1, b1, ..., W4, b4) of the surrogate and its standardisation, of a trained network's scale."""
    g = np.random.Generator(np.random.Philox(key=int(seed) + 1))
    parts = []
    for n_in, n_out in ((64, 128), (128, 128), (128, 128), (128, 80)):
        parts.append(g.normal(0.0, math.sqrt(1.5 / n_in), size=n_out * n_in))
        parts.append(g.normal(0.0, 0.1, size=n_out))
    params = np.concatenate(parts).astype(np.float32)
    norm = np.concatenate([g.normal(0, 1, 64), g.uniform(0.3, 2, 64), g.uniform(0.3, 4, 80), g.uniform(0.05, 0.6, 80)])
    return params, norm.astype(np.float32)


def _rows(seed, rows, norm):
    """Descriptors and G(t) curves of `rows` tracks: correlated, with a track-to-track spread."""
    g = np.random.Generator(np.random.Philox(key=int(seed) + 2))
    z = g.normal(size=(rows, 64)).astype(np.float32)
    z[:, 1:] = 0.6 * z[:, :1] + 0.8 * z[:, 1:]
    mix = (g.normal(size=(64, 80)) / 8).astype(np.float32)
    t = np.tanh(z @ mix) + 0.1 * g.normal(size=(rows, 80)).astype(np.float32)
    return (norm[:64] + norm[64:128] * z).astype(np.float32), (norm[128:208] + norm[208:] * t).astype(np.float32)


def prepare(case, seed):
    op = case["op"]
    L = _lib.lib()
    if op == "track":
        rads = [synthetic.synthetic_track(key=1000 * seed + k, n_spurs=case["spurs"],
                                          length_nm=2700.0 * case["spurs"] / 510.0, pid=k) for k in range(case["tracks"])]
        rad = np.concatenate(rads)
        return {"op": op, "ctx": wgdna.Context(max_primaries=16, max_rad=1_000_000, max_sec=100_000), "rad": rad,
                "tracks": case["tracks"], "seed": seed}
    if op in ("predict", "train"):
        ctx = wgdna.Context(max_primaries=16, max_rad=1_000_000, max_sec=100_000)
        params, norm = _network(seed)
        X, G = _rows(seed, case["rows"], norm)
        _lib.check("wgdna_surrogate_params", L.wgdna_surrogate_params(ctx.h, None, _lib.ptr(params)))
        _lib.check("wgdna_surrogate_norm", L.wgdna_surrogate_norm(ctx.h, None, _lib.ptr(norm)))
        if op == "train":
            _lib.check("wgdna_surrogate_load", L.wgdna_surrogate_load(ctx.h, _lib.ptr(X), _lib.ptr(G), case["rows"]))
        return {"op": op, "ctx": ctx, "X": X, "batch": case.get("batch"), "epochs": case.get("epochs"), "seed": seed}
    if op == "validate":
        n = case["np"]
        ctx = wgdna.Context(max_primaries=n, max_rad=max(n * 1600, 1_000_000), max_sec=max(n * 300, 100_000))
        rad = _views(ctx, n)["rad"]
        torch.cuda.synchronize()
        return {"op": op, "ctx": ctx, "np": n, "ce": case["ce"], "box": case["box"], "dna": wgdna.build_dna_target(),
                "rad": rad, "seed": seed}
    if op == "data":
        ctx = _context(case)
        n, lo, hi = case["np"], case["lo"], case["hi"]
        E = np.full(n, lo, np.float32) if lo == hi else synthetic.mixed_energies(n, lo, hi, key=seed)
        return {"op": op, "ctx": ctx, "E": E, "seed": seed, "ce": case["ce"], "box": case["box"]}
    st = _transport_state(case, seed)
    st["seed"] = seed
    if op in ("irt", "chemistry", "score", "grid"):
        _transport(st)
    if op == "chemistry":
        ctx = st["ctx"]
        params, norm = _network(seed)
        X = np.zeros((case["np"], 64), np.float32)
        k = C.c_uint64()
        _lib.check("wgdna_track_descriptors",
                   L.wgdna_track_descriptors(ctx.h, _lib.ptr(X), case["np"], C.byref(k)))
        norm[:64], s = X.mean(axis=0), X.std(axis=0)
        norm[64:128] = np.where(s > 1e-6, s, 1.0)
        _lib.check("wgdna_surrogate_params", L.wgdna_surrogate_params(ctx.h, None, _lib.ptr(params)))
        _lib.check("wgdna_surrogate_norm", L.wgdna_surrogate_norm(ctx.h, None, _lib.ptr(norm)))
    return st


# ------------------------------------------------------------------ the calls
def _transport_out(st):
    s = st["stats"]
    return {"results": st["results"], "dose": st["dose"], "rad": st["rad"],
            "rad_n": int(s.rad_n_stored), "counters": np.array(s.counters), "sec_stats": np.array(s.sec_stats), "n_therm": int(s.n_therm),
            "dep_units": int(s.dep_units), "dep_eV": float(s.dep_eV_f64)}


def _irt_out(r):
    return {"counts": np.array(r.counts), "G": np.array(r.G), "rxn": np.array(r.rxn_counts, np.int64),
            "reacted": int(r.n_reacted), "events": int(r.n_events), "pairs": int(r.n_pairs)}


def _irt(st):
    r = _lib.IrtResult()
    _lib.check("wgdna_irt", _lib.lib().wgdna_irt(st["ctx"].h, st["stats"].n_therm, st["E"], st["seed"] + 1, C.byref(r)))
    return _irt_out(r)


def _score(st):
    a, b = _lib.SsbResult(), _lib.DsbResult()
    _lib.check("wgdna_score", _lib.lib().wgdna_score(st["ctx"].h, LCG0, C.byref(a), C.byref(b)))
    return {"ssb": int(a.ssb), "in_reach": int(a.in_reach), "candidates": int(a.candidates), "lcg": int(a.lcg_state),
            "dsb": int(b.dsb), "dsb_expected": float(b.dsb_expected), "hits": st["hits"]}


def run(st):
    op = st["op"]
    L = _lib.lib()
    if op == "transport":
        _transport(st)
        return _transport_out(st)
    if op == "irt":
        return _irt(st)
    if op == "batch":
        _transport(st)
        return {"irt": _irt(st), "score": _score(st), "transport": _transport_out(st)}
    if op == "score":
        return _score(st)
    if op == "track":
        r = chemistry.run_chemistry_worker(st["ctx"], st["rad"], st["rad"].shape[0], st["tracks"], 10000.0,
                                           seed=st["seed"])
        return {"counts": r["counts"], "reacted": r["n_reacted"], "pairs": r["n_pairs"], "events": r["n_events"],
                "rxn": np.array([x["count"] for x in r["rxn_info"]], np.int64)}
    if op == "validate":
        ctx, dna = st["ctx"], st["dna"]
        r = dispatch.run_at_energy(ctx, 10000, st["np"], st["box"], st["ce"], dna, "device", seed=st["seed"])
        d = app.score_damage_at_10kev(ctx, dna, r["chem_result"], r["rad_buf_final"], r["rad_n_stored"],
                                      r["total_deposited_eV"], st["box"], wgdna.make_ssb_rng(),
                                      lambda *_: None, r["kernel_dna_hits"])
        # (the host rad_buf's length differs from seed to seed: its device
        # original is returned, and the damage numbers come from the host copy)
        return {"results": r["results"], "dose": r["dose_arr"].view(np.int32), "rad": st["rad"],
                "csda": r["mean_total"], "ions": r["mean_ions"], "cons": r["cons_ratio"],
                "hits": r["kernel_dna_hits"], "counts": r["chem_result"]["counts"],
                "events": r["chem_result"]["n_events"], "ssb": d["ssb_dir"], "dsb": d["dsb"],
                "dsb_expected": d["dsb_expected"]}
    if op == "data":
        X, G, E, r = surrogate.track_data(st["ctx"], st["E"], st["seed"], box_nm=st["box"], ce_eV=st["ce"])
        return {"X": X, "G": G, "E": E, "irt": _irt_out(r)}
    if op == "chemistry":
        G = np.zeros((16, 5))
        _lib.check("wgdna_surrogate_chemistry", L.wgdna_surrogate_chemistry(st["ctx"].h, _lib.ptr(G), None))
        return G
    if op == "predict":
        return surrogate.predict(st["ctx"], st["X"])
    if op == "train":
        ctx = st["ctx"]
        losses = np.zeros(st["epochs"], np.float32)
        params = np.zeros(_lib.SG_NPARAM, np.float32)
        _lib.check("wgdna_surrogate_init", L.wgdna_surrogate_init(ctx.h, st["seed"]))
        _lib.check("wgdna_surrogate_train", L.wgdna_surrogate_train(ctx.h, st["epochs"], st["batch"], 5e-4, st["seed"],
                                                                    _lib.ptr(losses)))
        _lib.check("wgdna_surrogate_params", L.wgdna_surrogate_params(ctx.h, _lib.ptr(params), None))
        return {"params": params, "losses": losses}
    # grid
    # Which of several pairs in contact reacts depends on thread timing, so the
    # positions and flags differ from run to run; the yields are what is compared.
    n = int(st["stats"].rad_n_stored)
    r = chemistry.run_chemistry_grid(st["ctx"], st["stats"].n_therm, st["E"], rad_n=n, seed=st["seed"])
    keys = ("G_OH", "G_eaq", "G_H", "G_H2O2", "G_H2")
    return np.array([[t[k] for k in keys] for t in r["timeline"]])


# ------------------------------------------------------------------ what a call cannot do without
def _pairs(case):
    """Species pairs of all tracks: n (n - 1) / 2 with n proportional to the energy."""
    lo, hi = case["lo"], case["hi"]
    e2 = lo * lo if lo == hi else (hi * hi - lo * lo) / (2.0 * math.log(hi / lo))
    return 0.5 * case["np"] * e2 * ENTRIES_PER_EV ** 2


def work(case):
    op = case["op"]
    if op == "track":
        n = 6.0 * case["spurs"]
        return {"bytes": 16 * n * case["tracks"] + 400, "flops": case["tracks"] * (25 * n * n / 36 / 2 * 8 + 200 * n)}
    if op == "predict":
        return {"bytes": case["rows"] * 4 * (64 + 80) + 2 * 51664, "flops": case["rows"] * 2.0 * 51200}
    if op == "train":
        n = case["rows"] // case["batch"] * case["batch"] * case["epochs"]
        return {"bytes": n * 4 * (64 + 80) + 4 * 51664, "flops": n * 6.0 * 51200}
    if op == "validate":
        case = dict(case, lo=10000.0, hi=10000.0)
    ev = case["np"] * _mean(case)
    rad = 16 * ENTRIES_PER_EV * ev
    tr = {"bytes": 32 * case["np"] + 4 * VC ** 3 + rad, "flops": 150 * STEPS_PER_EV * ev}
    irt = {"bytes": rad + 700, "flops": 8 * _pairs(case)}
    score = {"bytes": rad + HITS_BYTES, "flops": 30 * ENTRIES_PER_EV * ev}
    parts = {"transport": [tr], "irt": [irt], "score": [score], "batch": [tr, irt, score], "validate": [tr, irt, score],
             "data": [tr, irt, {"bytes": case["np"] * 4 * (64 + 80), "flops": 60 * ENTRIES_PER_EV * ev}],
             "chemistry": [{"bytes": rad + 2 * 51664, "flops": 60 * ENTRIES_PER_EV * ev + case["np"] * 2.0 * 51200}],
             "grid": [{"bytes": rad * 2.25, "flops": 133 * 100 * ENTRIES_PER_EV * ev}]}[op]
    return {k: float(sum(p[k] for p in parts)) for k in ("bytes", "flops")}


# ------------------------------------------------------------------ in 64 bits
_OFF = (0, 8192, 8320, 24704, 24832, 41216, 41344, 51584, 51664)
_SHAPES = ((128, 64), (128, 128), (128, 128), (80, 128))


def _layers(params):
    p = torch.as_tensor(params, dtype=torch.float64)
    return [(p[_OFF[2 * k]:_OFF[2 * k + 1]].view(_SHAPES[k]), p[_OFF[2 * k + 1]:_OFF[2 * k + 2]]) for k in range(4)]


def _mlp(params, x):
    for k, (w, b) in enumerate(_layers(params)):
        x = x @ w.T + b
        if k < 3:
            x = 0.5 * x * (1.0 + torch.erf(x / math.sqrt(2.0)))
    return x


_M64 = (1 << 64) - 1


def _splitmix(state):
    state = (state + 0x9E3779B97F4A7C15) & _M64
    z = ((state ^ (state >> 30)) * 0xBF58476D1CE4E5B9) & _M64
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & _M64
    return state, z ^ (z >> 31)


def _fresh(seed):
    """wgdna_surrogate_init's Glorot-uniform weights (splitmix64 draws) with zero biases."""
    state, p = seed ^ 0x5EED5EED, np.zeros(_OFF[-1], np.float32)
    for k, (n_out, n_in) in enumerate(_SHAPES):
        a = math.sqrt(6.0 / (n_in + n_out))
        for i in range(n_in * n_out):
            state, z = _splitmix(state)
            p[_OFF[2 * k] + i] = (2.0 * ((z >> 11) / 9007199254740992.0) - 1.0) * a
    return p


def exact(case, seed):
    """The surrogate in 64 bits.  The other operations have no value that a few
    lines of numpy could give: their histories and event orders are checked
    against the repository's CPU oracle in its tests."""
    op = case["op"]
    if op not in ("predict", "train"):
        return None
    params, norm = _network(seed)
    X, G = _rows(seed, case["rows"], norm)
    nrm = torch.as_tensor(norm, dtype=torch.float64)
    x = (torch.as_tensor(X, dtype=torch.float64) - nrm[:64]) / nrm[64:128]
    if op == "predict":
        return (_mlp(params, x) * nrm[208:] + nrm[128:208]).numpy()
    t = (torch.as_tensor(G, dtype=torch.float64) - nrm[128:208]) / nrm[208:]
    p = torch.as_tensor(_fresh(seed), dtype=torch.float64)
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    n, B, step, losses = case["rows"], case["batch"], 0, []
    state = seed ^ 0xA5A5A5A5
    for _ in range(case["epochs"]):
        perm = list(range(n))
        for i in range(n - 1, 0, -1):
            state, z = _splitmix(state)
            j = z % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        total = 0.0
        for b in range(n // B):
            at = torch.as_tensor(perm[b * B:(b + 1) * B])
            q = p.clone().requires_grad_(True)
            loss = (_mlp(q, x[at]) - t[at]).square().mean()
            g, = torch.autograd.grad(loss, q)
            total += float(loss.detach())
            step += 1
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            p = p - 5e-4 * (m / (1 - 0.9 ** step)) / ((v / (1 - 0.999 ** step)).sqrt() + 1e-8)
        losses.append(total / (n // B))
    return {"params": p.numpy(), "losses": np.array(losses)}
