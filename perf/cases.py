"""The workloads the framework's speed is measured on, through its public entry points.

Simulation (``modlefork_gb300.engine``): whole cells of the loop-extrusion epoch loop, as the
per-chromosome call, as one batched launch over a genome's chromosomes, and as a parameter
sweep's chunk with its training targets.
Surrogate (``modlefork_gb300.surrogate``, ``surrogate_ops``): inference, the gradients of a
training step, its optimiser step, single convolutions, and the scores of predicted maps.

A case is a dict of plain values; ``kind`` names the path.  ``listed`` gives the fixed cases,
``draw`` random ones of the same ranges.  ``prepare`` makes the inputs from the seed alone and what
a program keeps (engine context, uploaded chromosomes, network), ``run`` is one pass, ``exact`` the
same outputs in 64-bit arithmetic from plain torch and numpy where they are computed numbers.
"""

import math
import os

import numpy as np
import torch

from modlefork_gb300 import autotune, engine, genome, sweep
from modlefork_gb300 import surrogate as S
from modlefork_gb300 import surrogate_ops as ops
from modlefork_gb300 import train_surrogate

WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(engine.__file__)), "data", "surrogate_unet.npz")
DEV = "cuda:0"
LENGTH = 4000  # bins of a surrogate window
NROWS = 600    # diagonals of its band
MBP = 1_000_000


def listed():
    return [
        # the smallest simulation call: a 10 Mbp chromosome's 64 cells (the parity workload)
        {"name": "cells_10mbp", "kind": "cells", "bp": 10 * MBP, "lefs": 20.0, "bars": 10.0, "lifetime": 200_000,
         "speed": 2500, "num_cells": 64, "cells": 64, "density": 1.0, "burnin": True},
        # an ordinary per-chromosome call: one chromosome at the genome workload's densities
        {"name": "cells_73mbp", "kind": "cells", "bp": 73_000_451, "lefs": 20.0, "bars": 20.0, "lifetime": 200_000,
         "speed": 4000, "num_cells": 512, "cells": 152, "density": 1.0, "burnin": True},
        # the largest per-chromosome call: the genome workload's longest chromosome, a rank's share of its
        # 512 cells, started from the steady state's contacts (the burn-in switched off)
        {"name": "cells_250mbp", "kind": "cells", "bp": 249_999_451, "lefs": 20.0, "bars": 20.0, "lifetime": 200_000,
         "speed": 4000, "num_cells": 512, "cells": 304, "density": 1.0, "burnin": False},
        # a rank's share of a genome in one batched launch: the genome workload's densities, 24 chromosomes
        {"name": "genome_batch", "kind": "genome", "chroms": 24, "bp_min": 40 * MBP, "bp_max": 110 * MBP,
         "num_cells": 512, "cells": 24, "density": 1.0},
        # a chunk of the parameter sweep: 20 Mbp windows, each with its own configuration, and their targets
        {"name": "sweep_chunk", "kind": "sweep", "sets": 2, "cells": 1024, "density": 5.0},
        # one map: the latency of a single prediction
        {"name": "predict_1", "kind": "predict", "batch": 1},
        # the inference batch of the command line and the benchmark
        {"name": "predict_256", "kind": "predict", "batch": 256},
        # forward and backward pass of a training step at the default batch
        {"name": "gradients_16", "kind": "gradients", "batch": 16},
        # the optimiser step of that training
        {"name": "adam_step", "kind": "adam", "widths": 5},
        # a decoder level's convolution as the training forward runs it (both outputs kept)
        {"name": "conv_dec1a", "kind": "conv", "op": "forward", "batch": 32, "length": 2000, "cin": 384, "cout": 128,
         "taps": 3},
        # weight and bias gradients of an encoder convolution at a ragged length
        {"name": "conv_wgrad", "kind": "conv", "op": "wgrad", "batch": 16, "length": 999, "cin": 256, "cout": 256,
         "taps": 3},
        # per-map Pearson r and relative L2 of a held-out evaluation
        {"name": "scores_32", "kind": "scores", "maps": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cells", "cells", "genome", "sweep", "predict", "predict", "gradients", "conv", "conv", "conv",
                       "scores"])
    if kind == "cells":
        bp = _log_int(rng, 3 * MBP, 250 * MBP)
        return {"kind": kind, "bp": bp, "lefs": round(rng.uniform(5.0, 20.0), 2), "bars": round(rng.uniform(5.0, 40.0), 2),
                "lifetime": _log_int(rng, 100_000, 400_000), "speed": rng.randrange(2500, 5001),
                "num_cells": 512, "cells": _log_int(rng, 8, 152), "density": round(rng.uniform(0.2, 1.0), 2),
                "burnin": bp < 60 * MBP}
    if kind == "genome":
        lo = _log_int(rng, 2 * MBP, 40 * MBP)
        return {"kind": kind, "chroms": rng.randrange(2, 25), "bp_min": lo, "bp_max": lo + _log_int(rng, MBP, 70 * MBP),
                "num_cells": 512, "cells": _log_int(rng, 4, 24), "density": round(rng.uniform(0.3, 1.0), 2)}
    if kind == "sweep":
        sets = rng.randrange(1, 9)
        return {"kind": kind, "sets": sets, "cells": _log_int(rng, 32, 1024 // sets), "density": 1.0}
    if kind == "predict":
        return {"kind": kind, "batch": _log_int(rng, 2, 255)}
    if kind == "gradients":
        return {"kind": kind, "batch": rng.choice([n for n in range(1, 33) if n != 16])}
    if kind == "conv":
        op = rng.choice(["forward", "dgrad", "wgrad"])
        cin, cout = 64 * rng.randrange(1, 17), 64 * rng.randrange(1, 9)
        return {"kind": kind, "op": op, "batch": _log_int(rng, 1, 64), "length": _log_int(rng, 61, 4000) // 2 * 2 + 1,
                "cin": cin, "cout": cout, "taps": rng.choice([1, 3, 3])}
    return {"kind": kind, "maps": rng.choice([n for n in range(1, 65) if n != 32])}


# ---------------------------------------------------------------------------------------------
# simulation
# ---------------------------------------------------------------------------------------------
def _chromosome(rng, name, bp, bars_per_mbp, cfg):
    chrom = engine.Chromosome(name, bp)
    nb = max(1, int(round(bp / 1e6 * bars_per_mbp)))
    recs = genome.bed_records(rng, bp, nb, rng.beta(8.0, 2.0, size=nb))
    return chrom, engine.barriers_from_bed(chrom, recs, cfg.barrier_occupied_stp, cfg.barrier_not_occupied_stp)


def _cells_config(case, seed):
    return genome.genome_config(number_of_lefs_per_mbp=case["lefs"], avg_lef_processivity=case["lifetime"],
                                rev_extrusion_speed=case["speed"], fwd_extrusion_speed=case["speed"], rev_speed_set=1,
                                fwd_speed_set=1, rev_extrusion_speed_std=0.05, fwd_extrusion_speed_std=0.05,
                                num_cells=case["num_cells"], target_contact_density=case["density"], seed=seed,
                                skip_burnin=0 if case["burnin"] else 1)


def _cell_tasks(cfg, chrom, num_cells, cells):
    nl = engine.num_lefs(cfg, chrom.simulated_size)
    targets, epochs = engine.task_targets(cfg, chrom.simulated_size, nl, num_cells)
    seeds = np.array([engine.cell_seed(chrom.name, chrom.size, cfg.seed, i) for i in range(cells)], dtype=np.uint64)
    return nl, seeds, targets[:cells], epochs


def _counters(stats):
    """Per-cell results: epochs, burn-in epochs, contacts, missed updates, LEF-epochs, draws."""
    return np.array([[s.epochs, s.burnin_epochs, s.contacts, s.missed_updates, s.lef_epochs, s.rng_draws]
                     for s in stats], dtype=np.int64)


def _prepare_cells(case, seed):
    rng = np.random.default_rng([seed, 1])
    cfg = _cells_config(case, seed)
    chrom, bars = _chromosome(rng, "chr1", case["bp"], case["bars"], cfg)
    eng = engine.Engine(cfg, 0)
    autotune.apply_all(eng)
    cid = eng.upload_chrom(chrom, bars)
    nl, seeds, targets, epochs = _cell_tasks(cfg, chrom, case["num_cells"], case["cells"])
    nrows, ncols = engine.band_shape(cfg, chrom.simulated_size)
    return {"eng": eng, "cid": cid, "nl": nl, "seeds": seeds, "targets": targets, "epochs": epochs,
            "band": np.zeros(nrows * ncols, dtype=np.uint32)}


def _run_cells(s):
    # the drop-in call of a worker: contacts are added into its host matrix
    missed, stats = s["eng"].simulate_cells(s["cid"], s["seeds"], s["targets"], s["epochs"], s["nl"], s["band"])
    return {"band": s["band"].view(np.int32), "missed": int(missed), "cells": _counters(stats)}


def _prepare_genome(case, seed):
    rng = np.random.default_rng([seed, 2])
    cfg = genome.genome_config(num_cells=case["num_cells"], target_contact_density=case["density"], seed=seed)
    eng = engine.Engine(cfg, 0)
    autotune.apply_all(eng)
    # lengths evenly spread over the range (so that one seed's genome is as large as another's)
    n = case["chroms"]
    lengths = [int(case["bp_min"] + (case["bp_max"] - case["bp_min"]) * (k + 0.5) / n) for k in range(n)]
    tasks, bands = [], {}
    for k, bp in enumerate(lengths):
        chrom, bars = _chromosome(rng, f"chr{k + 1}", bp, 20.0, cfg)
        cid = eng.upload_chrom(chrom, bars)
        nl, seeds, targets, epochs = _cell_tasks(cfg, chrom, case["num_cells"], case["cells"])
        nrows, ncols = engine.band_shape(cfg, chrom.simulated_size)
        bands[cid] = torch.zeros(nrows * ncols, dtype=torch.int32, device=DEV)
        tasks += [(cid, int(x), int(t), epochs, nl) for x, t in zip(seeds, targets)]
    torch.cuda.synchronize()
    return {"eng": eng, "tasks": tasks, "bands": bands, "ptrs": {c: b.data_ptr() for c, b in bands.items()}}


def _run_batch(s):
    missed, stats = s["eng"].simulate_batch(s["tasks"], s["ptrs"])
    return missed, _counters(stats)


def _run_genome(s):
    missed, cells = _run_batch(s)
    return {"bands": [s["bands"][c] for c in sorted(s["bands"])], "missed": [missed[c] for c in sorted(missed)],
            "cells": cells}


def _prepare_sweep(case, seed):
    eng = engine.Engine(genome.genome_config(), 0)
    autotune.apply_all(eng)
    tasks, bands = [], {}
    for k in range(case["sets"]):
        cfg, chrom, bars, _, _ = sweep.window(k, seed=seed % 100_000, cells=case["cells"], density=case["density"])
        cid = eng.upload_chrom(chrom, bars)
        eng.set_chrom_config(cid, cfg)
        nl, seeds, targets, epochs = _cell_tasks(cfg, chrom, case["cells"], case["cells"])
        bands[cid] = torch.zeros(LENGTH * NROWS, dtype=torch.int32, device=DEV)
        tasks += [(cid, int(x), int(t), epochs, nl) for x, t in zip(seeds, targets)]
    torch.cuda.synchronize()
    return {"eng": eng, "tasks": tasks, "bands": bands, "ptrs": {c: b.data_ptr() for c, b in bands.items()},
            "targets": torch.empty(case["sets"], LENGTH, NROWS, dtype=torch.float32, device=DEV)}


def _run_sweep(s):
    missed, cells = _run_batch(s)
    for j, c in enumerate(sorted(s["bands"])):
        ops.band_target(s["bands"][c], LENGTH, NROWS, s["targets"][j])
    return {"bands": [s["bands"][c] for c in sorted(s["bands"])], "missed": [missed[c] for c in sorted(missed)],
            "cells": cells, "targets": s["targets"]}


# ---------------------------------------------------------------------------------------------
# surrogate
# ---------------------------------------------------------------------------------------------
def _windows(seed, n):
    """Tracks [n, 4, LENGTH] and parameters [n, 4] distributed as the sweep's windows (host arrays)."""
    rng = np.random.default_rng([seed, 3])
    lefs, life = rng.uniform(5.0, 40.0, n), rng.uniform(50e3, 500e3, n)
    speed, bars = rng.uniform(1e3, 5e3, n), rng.uniform(10.0, 60.0, n)
    counts = np.round(20.0 * bars).astype(np.int64)
    total = int(counts.sum())
    at = np.repeat(np.arange(n), counts) * LENGTH + rng.integers(0, LENGTH, total)
    plus = rng.random(total) < 0.5
    track = np.zeros((n, 4, LENGTH), dtype=np.float32)
    track[:, 0] = np.bincount(at, weights=rng.beta(8.0, 2.0, total), minlength=n * LENGTH).reshape(n, LENGTH)
    track[:, 1] = np.bincount(at[plus], minlength=n * LENGTH).reshape(n, LENGTH)
    track[:, 2] = np.bincount(at[~plus], minlength=n * LENGTH).reshape(n, LENGTH)
    track[:, 3] = (lefs / sweep.PARAM_SCALE[0])[:, None]
    params = (np.stack([lefs, life, speed, bars], axis=1) / sweep.PARAM_SCALE).astype(np.float32)
    return track, params


def _inputs(seed, n):
    track, params = _windows(seed, n)
    return torch.from_numpy(track).to(DEV), torch.from_numpy(params).to(DEV)


def _targets(seed, n):
    """Maps like a simulated window's: the distance decay of a band, log-normal around it."""
    gen = torch.Generator(device=DEV).manual_seed(seed + 17)
    d = torch.arange(NROWS, device=DEV, dtype=torch.float32)
    row = torch.log1p(40.0 * (1.0 + d).pow(-0.75))
    return (row * torch.exp(0.2 * torch.randn(n, LENGTH, NROWS, device=DEV, generator=gen))).contiguous()


def _network():
    autotune.apply_all()
    return train_surrogate.load_weights(WEIGHTS)


def _prepare_predict(case, seed):
    track, params = _inputs(seed, case["batch"])
    x = torch.empty(case["batch"], LENGTH, S.IN_CH, dtype=torch.bfloat16, device=DEV)
    return {"net": _network(), "track": track, "params": params, "x": x}


def _run_predict(s):
    ops.assemble_input(s["track"], s["params"], s["x"])
    return s["net"].forward(s["x"])


def _prepare_gradients(case, seed):
    track, params = _inputs(seed, case["batch"])
    x = torch.empty(case["batch"], LENGTH, S.IN_CH, dtype=torch.bfloat16, device=DEV)
    ops.assemble_input(track, params, x)
    return {"net": _network(), "x": x, "target": _targets(seed, case["batch"])}


def _run_gradients(s):
    net = s["net"]
    loss = net.loss_and_grad(s["x"], s["target"])
    return {"loss": loss, "w": dict(net.gw), "b": dict(net.gb)}


def _adam_inputs(seed, n):
    """Gradient (with the training's loss scale) and moments of a training under way."""
    gen = torch.Generator(device=DEV).manual_seed(seed + 5)
    g = torch.randn(n, device=DEV, generator=gen) * (1e-3 * S.LOSS_SCALE)
    m = torch.randn(n, device=DEV, generator=gen) * 3e-4
    v = (torch.randn(n, device=DEV, generator=gen) * 1e-3).square() + 1e-9
    return g, m, v


ADAM_STEP, ADAM_LR = 1000, 1e-4


def _prepare_adam(case, seed):
    if case["widths"] != 5:
        raise ValueError("the shipped network has five levels")
    net = _network()
    g, m, v = _adam_inputs(seed, net.p.numel())
    net.g.copy_(g)
    net.m.copy_(m)
    net.v.copy_(v)
    net.step_count = ADAM_STEP - 1
    return {"net": net}


def _run_adam(s):
    net = s["net"]
    net.adam_step(ADAM_LR)
    return {"p": net.p, "m": net.m, "v": net.v, "bf16": net.pb, "transposed": dict(net.wt)}


def _conv_inputs(case, seed):
    """Activations, weights, bias, pre-activations and output gradient of one convolution."""
    B, L, ci, co, taps = (case[k] for k in ("batch", "length", "cin", "cout", "taps"))
    gen = torch.Generator(device=DEV).manual_seed(seed + 29)

    def normal(*shape, scale=1.0):
        return torch.randn(*shape, device=DEV, generator=gen) * scale

    x = torch.nn.functional.silu(normal(B, L, ci)).to(torch.bfloat16)
    w = normal(co, taps, ci, scale=1.6 / math.sqrt(taps * ci)).to(torch.bfloat16)
    b = normal(co, scale=0.1)
    z = normal(B, L, ci).to(torch.bfloat16)
    dz = normal(B, L, co, scale=1e-2).to(torch.bfloat16)
    return x, w, b, z, dz


def _prepare_conv(case, seed):
    autotune.apply_all()
    x, w, b, z, dz = _conv_inputs(case, seed)
    B, L, ci, co = (case[k] for k in ("batch", "length", "cin", "cout"))
    s = {"op": case["op"], "x": x, "w": w, "b": b, "z": z, "dz": dz}
    if case["op"] == "forward":
        s["pre"] = torch.empty(B, L, co, dtype=torch.bfloat16, device=DEV)
        s["post"] = torch.empty_like(s["pre"])
    elif case["op"] == "dgrad":
        s["wt"] = torch.empty(ci, case["taps"], co, dtype=torch.bfloat16, device=DEV)
        ops.weight_transpose(w, s["wt"])
        s["dx"] = torch.empty(B, L, ci, dtype=torch.bfloat16, device=DEV)
    else:
        s["dw"] = torch.zeros(co, case["taps"], ci, device=DEV)
        s["db"] = torch.zeros(co, device=DEV)
    return s


def _run_conv(s):
    if s["op"] == "forward":
        ops.conv_forward(s["x"], s["w"], bias=s["b"], act=ops.ACT_SILU, out_pre=s["pre"], out_post=s["post"])
        return {"pre": s["pre"], "post": s["post"]}
    if s["op"] == "dgrad":
        ops.conv_forward(s["dz"], s["wt"], out_post=s["dx"], gate=s["z"])
        return {"dx": s["dx"]}
    s["dw"].zero_()
    s["db"].zero_()
    ops.conv_wgrad(s["x"], s["dz"], s["dw"])
    ops.bias_grad(s["dz"], s["db"])
    return {"dw": s["dw"], "db": s["db"]}


def _prepare_scores(case, seed):
    ref = _targets(seed, case["maps"])
    gen = torch.Generator(device=DEV).manual_seed(seed + 31)
    pred = ref + 0.1 * torch.randn(ref.shape, device=DEV, generator=gen)
    return {"pred": pred, "ref": ref}


def _run_scores(s):
    r, l2 = S.evaluate(s["pred"], s["ref"])
    return {"r": r, "l2": l2}


# ---------------------------------------------------------------------------------------------
# the same in 64 bits, from plain torch
# ---------------------------------------------------------------------------------------------
def _conv64(x, w, b=None):
    """x [B, L, Cin], w [Cout, taps, Cin] in float64: the zero-padded convolution over positions."""
    B, L, _ = x.shape
    taps = w.shape[1]
    pad = (taps - 1) // 2
    y = None
    for t in range(taps):
        lo, hi = max(0, pad - t), min(L, L + pad - t)
        part = torch.zeros(B, L, w.shape[0], dtype=x.dtype, device=x.device)
        part[:, lo:hi] = x[:, lo + t - pad:hi + t - pad] @ w[:, t].T
        y = part if y is None else y + part
    return y if b is None else y + b


def _silu64(z):
    return z * torch.sigmoid(z)


def _weights64():
    z = np.load(WEIGHTS)
    P = {}
    for k in z.files:
        if k.startswith("w_"):
            w = torch.from_numpy(z[k].copy()).view(torch.bfloat16).to(DEV).double()
            P[k[2:]] = [w, torch.from_numpy(z["b_" + k[2:]]).to(DEV).double()]
    return P


def _input64(seed, n):
    """[n, LENGTH, 8]: the channels of the network's input that are used, rounded to BF16 as stored."""
    track, params = _inputs(seed, n)
    x = torch.cat([track.transpose(1, 2), params[:, None, :].expand(n, LENGTH, 4)], dim=2)
    return x.to(torch.bfloat16).double()


def _forward64(P, x):
    D = sum(k.startswith("enc") and k.endswith("a") for k in P)
    first = [P["enc0a"][0][:, :, :x.shape[2]], P["enc0a"][1]]
    skips, h = [], x
    for i in range(D):
        h = _silu64(_conv64(h, *(first if i == 0 else P[f"enc{i}a"])))
        h = _silu64(_conv64(h, *P[f"enc{i}b"]))
        skips.append(h)
        h = 0.5 * (h[:, 0::2] + h[:, 1::2])
    h = _silu64(_conv64(_silu64(_conv64(h, *P["mid_a"])), *P["mid_b"]))
    for i in reversed(range(D)):
        h = torch.cat([h.repeat_interleave(2, dim=1), skips[i]], dim=2)
        h = _silu64(_conv64(_silu64(_conv64(h, *P[f"dec{i}a"])), *P[f"dec{i}b"]))
    return _conv64(h, P["head"][0][:NROWS], P["head"][1][:NROWS])


def _exact_predict(case, seed):
    P = _weights64()
    x = _input64(seed, case["batch"])
    with torch.no_grad():
        return torch.cat([_forward64(P, x[i:i + 8]) for i in range(0, x.shape[0], 8)])


def _exact_gradients(case, seed):
    P = _weights64()
    for name in P:
        P[name] = [p.requires_grad_(True) for p in P[name]]
    x, target = _input64(seed, case["batch"]), _targets(seed, case["batch"])
    count, loss = target.numel(), 0.0
    for i in range(0, x.shape[0], 4):  # gradients add up over the maps
        part = (_forward64(P, x[i:i + 4]) - target[i:i + 4].double()).square().sum()
        (part * (S.LOSS_SCALE / count)).backward()
        loss += float(part.detach())
    return {"loss": torch.tensor([loss / count], dtype=torch.float64), "w": {k: P[k][0].grad for k in P},
            "b": {k: P[k][1].grad for k in P}}


def _exact_adam(case, seed):
    z = np.load(WEIGHTS)
    parts = []
    for k in z.files:  # weights and biases in network order, each padded to 64 elements
        if k.startswith("w_"):
            for t in (torch.from_numpy(z[k].copy()).view(torch.bfloat16).double().reshape(-1),
                      torch.from_numpy(z["b_" + k[2:]]).double()):
                parts += [t, torch.zeros(-t.numel() % 64, dtype=torch.float64)]
    p = torch.cat(parts).to(DEV)
    g, m, v = (t.double() for t in _adam_inputs(seed, p.numel()))
    g = g / S.LOSS_SCALE
    m = 0.9 * m + 0.1 * g
    v = 0.999 * v + 0.001 * g * g
    p = p - ADAM_LR * (m / (1 - 0.9 ** ADAM_STEP)) / ((v / (1 - 0.999 ** ADAM_STEP)).sqrt() + 1e-8)
    return {"p": p, "m": m, "v": v, "bf16": None, "transposed": None}


def _exact_conv(case, seed):
    x, w, b, z, dz = (t.double() for t in _conv_inputs(case, seed))
    if case["op"] == "forward":
        pre = _conv64(x, w, b)
        return {"pre": pre, "post": _silu64(pre)}
    if case["op"] == "dgrad":
        s = torch.sigmoid(z)
        return {"dx": _conv64(dz, w.flip(1).permute(2, 1, 0)) * (s * (1 + z * (1 - s)))}
    L, taps = x.shape[1], w.shape[1]
    pad, dw = (taps - 1) // 2, []
    for t in range(taps):
        lo, hi = max(0, pad - t), min(L, L + pad - t)
        dw.append(dz[:, lo:hi].reshape(-1, dz.shape[2]).T @ x[:, lo + t - pad:hi + t - pad].reshape(-1, x.shape[2]))
    return {"dw": torch.stack(dw, dim=1), "db": dz.sum(dim=(0, 1))}


def _exact_scores(case, seed):
    s = _prepare_scores(case, seed)
    r, l2 = [], []
    for p, t in zip(s["pred"], s["ref"]):
        p, t = p.double().reshape(-1), t.double().reshape(-1)
        dp, dt = p - p.mean(), t - t.mean()
        r.append(float((dp * dt).sum() / ((dp * dp).sum() * (dt * dt).sum()).sqrt()))
        l2.append(float((p - t).norm() / t.norm()))
    return {"r": np.array(r), "l2": np.array(l2)}


# ---------------------------------------------------------------------------------------------
def _cell_bytes(cfg, bp, nbars, num_cells, cells, burnin=300.0):
    """Positions and binding epochs of the LEFs read and written once per epoch, barrier positions and
    states, one band pixel per contact; epochs of the contact target and of a typical burn-in."""
    nl = engine.num_lefs(cfg, bp)
    targets, _ = engine.task_targets(cfg, bp, nl, num_cells)
    per_epoch = max(1.0, round(nl * 2.0 * cfg.rev_extrusion_speed / cfg.contact_sampling_interval))
    contacts = float(targets[:cells].sum())
    epochs = contacts / per_epoch + burnin * cells
    return 24.0 * nl * epochs + 6.0 * nbars * epochs + 8.0 * contacts


def _layers():
    """(length divisor, cin, cout, taps) of the shipped network's convolutions."""
    out, w, cin = [], (64, 128, 256, 384, 512), 64
    for i, c in enumerate(w):
        out += [(1 << i, cin, c, 3), (1 << i, c, c, 3)]
        cin = c
    out += [(32, 512, 512, 3), (32, 512, 512, 3)]
    ch = 512
    for i in reversed(range(5)):
        out += [(1 << i, ch + w[i], w[i], 3), (1 << i, w[i], w[i], 3)]
        ch = w[i]
    return out + [(1, 64, 640, 1)]


def work(case):
    kind = case["kind"]
    if kind == "cells":
        return {"bytes": _cell_bytes(_cells_config(case, 1), case["bp"], case["bars"] * case["bp"] / 1e6,
                                     case["num_cells"], case["cells"], 300.0 if case["burnin"] else 0.0), "flops": 0}
    if kind == "genome":
        cfg = genome.genome_config(num_cells=case["num_cells"], target_contact_density=case["density"])
        n, total = case["chroms"], 0.0
        for k in range(n):
            bp = int(case["bp_min"] + (case["bp_max"] - case["bp_min"]) * (k + 0.5) / n)
            total += _cell_bytes(cfg, bp, bp / 50_000, case["num_cells"], case["cells"])
        return {"bytes": total, "flops": 0}
    if kind == "sweep":
        cfg = genome.genome_config(number_of_lefs_per_mbp=22.5, num_cells=case["cells"],
                                   target_contact_density=case["density"], rev_extrusion_speed=3000,
                                   fwd_extrusion_speed=3000, rev_speed_set=1, fwd_speed_set=1)
        one = _cell_bytes(cfg, sweep.WINDOW_BP, 700, case["cells"], case["cells"])
        return {"bytes": case["sets"] * (one + 8.0 * LENGTH * NROWS), "flops": 0}
    if kind == "adam":
        n = sum(ci * co * t + co for _, ci, co, t in _layers())
        return {"bytes": 32.0 * n, "flops": 12.0 * n}
    if kind == "scores":
        return {"bytes": 8.0 * case["maps"] * LENGTH * NROWS, "flops": 12.0 * case["maps"] * LENGTH * NROWS}
    if kind == "conv":
        B, L, ci, co, taps = (case[k] for k in ("batch", "length", "cin", "cout", "taps"))
        rows = B * L
        flops = 2.0 * rows * ci * co * taps
        if case["op"] == "forward":
            return {"bytes": 2.0 * (rows * (ci + 2 * co) + ci * co * taps), "flops": flops}
        if case["op"] == "dgrad":
            return {"bytes": 2.0 * (rows * (2 * ci + co) + ci * co * taps), "flops": flops}
        return {"bytes": 2.0 * rows * (ci + co) + 4.0 * ci * co * taps, "flops": flops}
    flops = sum(2.0 * (LENGTH // d) * ci * co * t for d, ci, co, t in _layers()) * case["batch"]
    n = sum(ci * co * t + co for _, ci, co, t in _layers())
    maps = 4.0 * case["batch"] * LENGTH * NROWS
    if kind == "predict":
        return {"bytes": maps + 16.0 * case["batch"] * LENGTH + 2.0 * n, "flops": flops}
    return {"bytes": maps + 128.0 * case["batch"] * LENGTH + 6.0 * n, "flops": 3.0 * flops}


_KINDS = {
    "cells": (_prepare_cells, _run_cells, None),
    "genome": (_prepare_genome, _run_genome, None),
    "sweep": (_prepare_sweep, _run_sweep, None),
    "predict": (_prepare_predict, _run_predict, _exact_predict),
    "gradients": (_prepare_gradients, _run_gradients, _exact_gradients),
    "adam": (_prepare_adam, _run_adam, _exact_adam),
    "conv": (_prepare_conv, _run_conv, _exact_conv),
    "scores": (_prepare_scores, _run_scores, _exact_scores),
}


def prepare(case, seed):
    return {"kind": case["kind"], "state": _KINDS[case["kind"]][0](case, seed)}


def run(s):
    return _KINDS[s["kind"]][1](s["state"])


def exact(case, seed):
    """What run returns for these inputs, in 64 bits; None for whole numbers."""
    f = _KINDS[case["kind"]][2]
    return None if f is None else f(case, seed)
