"""The work users have this framework do, as cases that can be timed and checked.

Every case names one public entry point (``kind``) and the sizes of one call:

* ``evaluate`` - ``B200DecoderEvaluator.evaluate_batch``, the drop-in call of the GA loop on a host population;
* ``decode``   - ``DeviceDecoder.decode`` of a population that is already on the GPU;
* ``multi``    - ``MultiDecoder.decode``, uneven instances in one launch;
* ``fit``      - ``DeviceBRKGA.fit``, a whole run of a few generations;
* ``greedy``   - ``initial_solution``, the first individual of a run;
* ``predict``  - ``Surrogate.predict`` on the candidates of a screened generation;
* ``train``    - ``Surrogate.train``, the online learning of one generation.

Instances come from the seeded generators of ``brkga_fft2_b200.instances`` in the shapes of its named workloads.  A case
fixes the instance; the populations, weights and targets come from the seed.  Populations are uniform random keys, which
is what a GA's first generation, its mutants and most of its offspring look like to the decoder.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

from brkga_fft2_b200 import THRESH_F32, THRESH_F64, abi, instances, pack_problem
from brkga_fft2_b200.evaluator import B200DecoderEvaluator, DeviceDecoder, MultiDecoder, _NativeProblem
from brkga_fft2_b200.ga import DeviceBRKGA
from brkga_fft2_b200.initial import initial_solution
from brkga_fft2_b200.surrogate import Surrogate

# Instance shapes: parts, machines, plate of the first half of the machines (rows x cols) and of the second half,
# mask sides, per-machine time constants.
P50M2 = dict(parts=50, machines=2, rows=250, cols=250, rows2=250, cols2=250, side_min=10, side_max=80, scaled=False)
P100M4 = dict(parts=100, machines=4, rows=300, cols=300, rows2=250, cols2=250, side_min=10, side_max=120, scaled=True)
P200M6 = dict(parts=200, machines=6, rows=400, cols=400, rows2=400, cols2=400, side_min=10, side_max=80, scaled=False)
P400M8 = dict(parts=400, machines=8, rows=600, cols=600, rows2=600, cols2=600, side_min=20, side_max=240, scaled=False)


def listed():
    return [
        # One chromosome with its placements: inspecting or re-checking a solution.  The latency of a single decode.
        dict(name="evaluate_p50m2_1_log", kind="evaluate", pop=1, log=True, f64=False, instance=0, **P50M2),
        # The GA's default population (100) on the smallest benchmark size, host buffers in and out.
        dict(name="evaluate_p50m2_100", kind="evaluate", pop=100, log=False, f64=False, instance=0, **P50M2),
        # The headline workload through the drop-in evaluator, as the reference's GA loop calls it.
        dict(name="evaluate_p100m4_500", kind="evaluate", pop=500, log=False, f64=False, instance=0, **P100M4),
        # The headline workload with the population on the GPU: one generation's decode.
        dict(name="decode_p100m4_500", kind="decode", pop=500, f64=False, instance=0, **P100M4),
        # The same instance at throughput: a large population or several runs' rows at once.
        dict(name="decode_p100m4_4000", kind="decode", pop=4000, f64=False, instance=0, **P100M4),
        # Many small parts on large plates, six machines, the C++ decoder's float64 thresholds.
        dict(name="decode_p200m6_1000", kind="decode", pop=1000, f64=True, instance=0, **P200M6),
        # The large stress population: 400 parts with masks up to 240 x 240, 600 x 600 plates.
        dict(name="decode_p400m8_4096", kind="decode", pop=4096, f64=False, instance=0, **P400M8),
        # The uneven batch: 64 instances of 25 to 200 parts on plates of 150 to 500 cells in one launch.
        dict(name="multi_64x256", kind="multi", instances=64, pop=256, instance=0),
        # A run of the GA on the headline workload, a few generations of it.
        dict(name="fit_p100m4_500", kind="fit", pop=500, generations=10, instance=0, **P100M4),
        # The greedy first individual of a run.
        dict(name="greedy_p100m4", kind="greedy", instance=0, **P100M4),
        # Screening the headline workload: eight children for each of 450 parent pairs.
        dict(name="predict_p100m4_3600", kind="predict", pop=3600, instance=0, **P100M4),
        # The surrogate's learning in one generation: six steps of 512 rows of a 4,000-row history.
        dict(name="train_p100m4_6x512", kind="train", steps=6, batch=512, history=4000, instance=0, **P100M4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_instance(rng, parts_max=400):
    rows, cols = _log_int(rng, 150, 600), _log_int(rng, 150, 600)
    same = rng.random() < 0.5
    rows2, cols2 = (rows, cols) if same else (_log_int(rng, 150, 600), _log_int(rng, 150, 600))
    small = min(rows, cols, rows2, cols2)
    side_max = max(24, min(240, int(small * rng.uniform(0.15, 0.4))))
    return dict(parts=_log_int(rng, 20, parts_max), machines=rng.randint(1, 8), rows=rows, cols=cols, rows2=rows2,
                cols2=cols2, side_min=rng.randint(6, 20), side_max=side_max, scaled=rng.random() < 0.5,
                instance=rng.randrange(1, 10_000))


def draw(rng):
    kind = rng.choices(["evaluate", "decode", "multi", "fit", "greedy", "predict", "train"], [4, 8, 2, 2, 1, 2, 2])[0]
    if kind == "multi":
        k = rng.randint(2, 64)
        return dict(kind=kind, instances=k, pop=_log_int(rng, 4, 256), instance=rng.randrange(1, 10_000))
    if kind in ("evaluate", "decode"):
        c = _draw_instance(rng)
        # at most a quarter of the parts of the largest listed case
        pop = min(_log_int(rng, 1, 500 if kind == "evaluate" else 4096), 400_000 // c["parts"])
        c.update(kind=kind, pop=pop, f64=rng.random() < 0.3)
        if kind == "evaluate":
            c["log"] = rng.random() < 0.3
        return c
    if kind == "fit":
        c = _draw_instance(rng, 150)
        return dict(c, kind=kind, pop=_log_int(rng, 40, 600), generations=rng.randint(2, 12))
    if kind == "greedy":
        return dict(_draw_instance(rng, 120), kind=kind)
    c = _draw_instance(rng)
    if kind == "predict":
        return dict(c, kind=kind, pop=_log_int(rng, 100, 8000))
    return dict(c, kind=kind, steps=rng.randint(1, 12), batch=128 * rng.randint(1, 8), history=_log_int(rng, 500, 8000))


# ------------------------------------------------------------------ inputs


def _plates(c):
    first = (c["machines"] + 1) // 2
    return [(c["rows"], c["cols"])] * first + [(c["rows2"], c["cols2"])] * (c["machines"] - first)


@functools.lru_cache(maxsize=96)
def _make(parts, plates, seed, side_min, side_max, scaled):
    return instances.make_instance("case", parts, list(plates), seed, bbox_min=side_min, bbox_max=side_max,
                                   scale_machines=scaled)


def _instance(c, offset=0):
    return _make(c["parts"], tuple(_plates(c)), c["instance"] + offset, c["side_min"], c["side_max"], c["scaled"])


@functools.lru_cache(maxsize=96)
def _uneven(seed):
    inst = instances.uneven(seed)
    return inst, _pack(inst, False)


def _pack(inst, f64):
    return pack_problem(inst.problem_data, inst.nb_parts, inst.nb_machines, inst.thresholds, inst.instance_parts,
                        THRESH_F64 if f64 else THRESH_F32)


def _keys(rows, parts, seed):
    return np.random.default_rng(seed).random((rows, 2 * parts)).astype(np.float32)


def _makespans(rows, seed):
    """Targets the size of P100M4 makespans, a few of them infeasible."""
    rng = np.random.default_rng([seed, 7])
    ms = rng.normal(7.5e5, 6e4, rows)
    ms[rng.random(rows) < 0.01] = 1e16
    return ms


def _weights(n_in, in_pad, seed):
    """A flat parameter vector of the size a trained surrogate's has (W1, b1, W2, b2, w3, b3)."""
    g = np.random.default_rng([seed, 3])
    w1 = np.zeros((512, in_pad))
    w1[:, :n_in] = g.uniform(-1, 1, (512, n_in)) * math.sqrt(6 / n_in)
    w2 = g.uniform(-1, 1, (256, 512)) * math.sqrt(6 / 512)
    w3 = g.uniform(-1, 1, 256) * math.sqrt(6 / 256)
    flat = [w1.ravel(), g.normal(0, 0.05, 512), w2.ravel(), g.normal(0, 0.05, 256), w3, g.normal(0, 0.05, 1)]
    return np.concatenate(flat).astype(np.float32)


class _DeviceArray:
    """A float32 device buffer of the library as torch.as_tensor takes it; the tensor keeps the buffer's owner alive."""

    def __init__(self, ptr, n, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f4", data=(ptr, False), version=3)


def _parameters(sur):
    """The surrogate's own parameter block, as a tensor over it."""
    import ctypes
    p = ctypes.c_void_p()
    abi.check(sur.lib.brkga_surrogate_buffers(sur.handle, ctypes.byref(p), None, None, None, None, None, None))
    return torch.as_tensor(_DeviceArray(p.value, sur.n_params, sur), device="cuda")


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"kind": kind}
    if kind == "multi":
        made = [_uneven(c["instance"] * 64 + k) for k in range(c["instances"])]
        s["decoder"] = MultiDecoder([p for _, p in made], [c["pop"]] * len(made))
        s["chroms"] = [torch.from_numpy(_keys(c["pop"], i.nb_parts, [seed, k])).cuda() for k, (i, _) in enumerate(made)]
        return s
    inst = _instance(c, seed % 1000 if kind == "greedy" else 0)
    if kind == "evaluate":
        s["evaluator"] = B200DecoderEvaluator(inst.problem_data, inst.nb_parts, inst.nb_machines, inst.thresholds,
                                              inst.instance_parts, None, "cuda", THRESH_F64 if c["f64"] else THRESH_F32)
        s["population"] = list(_keys(c["pop"], c["parts"], seed))
        s["log"] = c["log"]
    elif kind == "decode":
        s["decoder"] = DeviceDecoder(_pack(inst, c["f64"]), c["pop"])
        s["chrom"] = torch.from_numpy(_keys(c["pop"], c["parts"], seed)).cuda()
    elif kind == "fit":
        ne, nm = -(-c["pop"] // 10), -(-15 * c["pop"] // 100)
        s["ga"] = DeviceBRKGA(None, c["parts"], c["machines"], None, None, num_generations=c["generations"],
                              num_individuals=c["pop"], num_elites=ne, num_mutants=nm, seed=seed, packed=_pack(inst, False))
        s["ga"].prepare()
    elif kind == "greedy":
        s["native"] = _NativeProblem(_pack(inst, False))
        s["inst"], s["seed"] = inst, seed
        s["areas"] = [float(m.sum()) for m in inst.masks]
    else:
        s["native"] = _NativeProblem(_pack(inst, False))
        rows = c["history"] if kind == "train" else 512
        most = max(c.get("pop", 0), c.get("batch", 0), rows)
        s["surrogate"] = sur = Surrogate(s["native"], max_batch=-(-most // 128) * 128, buffer_capacity=20_000, seed=17)
        sur.set_params(_weights(sur.in_features, sur.in_pad, seed))
        seen = torch.from_numpy(_keys(rows, c["parts"], [seed, 1])).cuda()
        sur.observe(seen, torch.from_numpy(_makespans(rows, seed)).cuda())
        if kind == "predict":
            s["chrom"] = torch.from_numpy(_keys(c["pop"], c["parts"], seed)).cuda()
        else:
            s["steps"], s["batch"], s["params"] = c["steps"], c["batch"], _parameters(sur)
    return s


def run(state):
    s, kind = state, state["kind"]
    if kind == "evaluate":
        if s["log"]:
            ms, log = s["evaluator"].evaluate_batch(np.array(s["population"]), return_log=True)
            return np.asarray(ms), log.view(np.int32)
        return np.asarray(s["evaluator"].evaluate_batch(np.array(s["population"])))
    if kind == "decode":
        return s["decoder"].decode(s["chrom"])
    if kind == "multi":
        return s["decoder"].decode(s["chroms"])
    if kind == "fit":
        ga = s["ga"]
        ga.fit()
        return dict(population=ga.population, fitness=ga.fitness, best=ga.best_fitness, solution=ga.solution,
                    min=np.asarray(ga.history["min"]), mean=np.asarray(ga.history["mean"]))
    if kind == "greedy":
        i = s["inst"]
        chrom, ms, (machine, place) = initial_solution(s["native"], i.instance_parts, i.heights, s["areas"], i.thresholds,
                                                       random.Random(s["seed"]))
        return dict(chrom=chrom, makespan=ms, machine=machine, place=place.view(np.int32))
    if kind == "predict":
        return s["surrogate"].predict(s["chrom"])
    s["surrogate"].train(s["steps"], s["batch"])
    return s["params"]


def work(case):
    """Bytes: keys and tables read once, results written once.  Operations of a decode: the words of every part's mask
    compared with the plate at the position it is given, and written there; the search for that position is extra."""
    c, kind = case, case["kind"]
    if kind == "multi":
        made = [_uneven(c["instance"] * 64 + k)[0] for k in range(c["instances"])]
        sizes = [(c["pop"], i) for i in made]
    elif kind in ("predict", "train"):
        n_in = 3 * c["parts"] + 2 * c["machines"]
        params = 512 * n_in + 512 + 256 * 512 + 256 + 256 + 1
        if kind == "predict":
            return dict(bytes=c["pop"] * (8 * c["parts"] + 8) + 2 * params,
                        flops=2 * c["pop"] * (512 * n_in + 256 * 512 + 256))
        return dict(bytes=c["steps"] * (24 * params + 2 * c["batch"] * n_in),
                    flops=2 * c["steps"] * c["batch"] * (2 * 512 * n_in + 3 * 256 * 512 + 2 * 256))
    else:
        rows = c.get("pop", 1)
        if kind == "fit":
            rows += c["generations"] * (c["pop"] - -(-c["pop"] // 10))
        sizes = [(rows, _instance(c))]
    bytes_ = flops = 0
    for rows, inst in sizes:
        words = sum(m.shape[0] * (-(-m.shape[1] // 32)) for m in inst.masks)
        bytes_ += rows * (8 * inst.nb_parts + 8) + 4 * words
        flops += rows * 2 * words
        if c.get("log"):
            bytes_ += rows * inst.nb_parts * inst.nb_machines * 20
    return dict(bytes=bytes_, flops=flops)


# ------------------------------------------------------------------ the same results in 64 bits


class _Placer:
    """Plates of one instance in plain torch: the collision test is a float64 FFT correlation, as the method's papers
    and the reference's CPU path have it."""

    def __init__(self, inst):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.inst, self.parts, self.spectra = inst, [], {}
        for p, m in enumerate(inst.masks):
            n = 2 if np.array_equal(m, np.rot90(m, 2)) else 4
            rot = [np.ascontiguousarray(np.rot90(m, r)) for r in range(n)]
            self.parts.append((rot, int(np.argmin([r.shape[0] for r in rot])), float(m.sum())))

    def spectrum(self, p, L, W):
        """Conjugate spectra of the rotations that fit an L x W plate, and each candidate's rank (-1: outside)."""
        key = (p, L, W)
        if key not in self.spectra:
            rows = torch.arange(L, device=self.dev)[:, None]
            cols = torch.arange(W, device=self.dev)[None, :]
            masks, rank, shapes = [], [], []
            for r, m in enumerate(self.parts[p][0]):
                h, w = m.shape
                if h <= L and w <= W:
                    full = torch.zeros(L, W, dtype=torch.float64, device=self.dev)
                    full[:h, :w] = torch.from_numpy(m.astype(np.float64)).to(self.dev)
                    masks.append(full)
                    rank.append(torch.where((rows <= L - h) & (cols <= W - w), rows * W + (W - 1 - cols), -1))
                    shapes.append((r, h))
            self.spectra[key] = (torch.fft.rfft2(torch.stack(masks)).conj(), torch.stack(rank), shapes) if masks else None
        return self.spectra[key]

    def best(self, plate, p):
        """(newLen, -y, x, rotation, top row) of the best position on a plate, None if there is none."""
        L, W = plate["grid"].shape
        found = self.spectrum(p, L, W)
        if found is None:
            return None
        if plate["fft"] is None:
            plate["fft"] = torch.fft.rfft2(plate["grid"])
        spec, rank, shapes = found
        hits = torch.fft.irfft2(plate["fft"] * spec, s=(L, W))
        top = torch.where(hits < 0.5, rank, -1).amax((1, 2)).tolist()
        keys = []
        for v, (r, h) in zip(top, shapes):
            if v >= 0:
                ty, x = v // W, W - 1 - v % W
                keys.append((max(plate["enc"], L - ty), -(ty + h - 1), x, r, ty))
        return min(keys) if keys else None

    def open(self, m):
        d = self.inst.problem_data.machines[m]
        return dict(grid=torch.zeros(d.bin_length, d.bin_width, dtype=torch.float64, device=self.dev), fft=None, enc=0,
                    area=0.0, pt=0.0, pth=0.0, m=m)

    def put(self, plate, p, r, ty, x):
        m = self.parts[p][0][r]
        h, w = m.shape
        plate["grid"][ty:ty + h, x:x + w] += torch.from_numpy(m.astype(np.float64)).to(self.dev)
        plate["fft"] = None
        plate["enc"] = max(plate["enc"], plate["grid"].shape[0] - ty)
        plate["area"] += self.parts[p][2]
        t = self.inst.problem_data.machines[plate["m"]].parts[p]
        plate["pt"] += t.proc_time
        plate["pth"] = max(plate["pth"], t.proc_time_height)

    def put_new(self, plate, p):
        r = self.parts[p][1]
        ty = plate["grid"].shape[0] - self.parts[p][0][r].shape[0]
        self.put(plate, p, r, ty, 0)
        return r, ty, 0


def _machines_of(keys, inst, f64):
    m = np.zeros(len(keys), np.int64)
    for t in inst.thresholds:
        m += keys.astype(np.float64) > t if f64 else keys > np.float32(t)
    return m


def _exact_decode(c, inst, keys, want_log):
    place, N, M = _Placer(inst), inst.nb_parts, inst.nb_machines
    out = np.zeros(len(keys))
    log = np.full((len(keys), M, N, 5), -1, np.int32)
    for k, row in enumerate(keys):
        machine = _machines_of(row[N:], inst, c["f64"])
        order = np.argsort(row[:N], kind="stable")
        worst = 0.0
        for m in range(M):
            d, plates = inst.problem_data.machines[m], []
            for i, p in enumerate(int(g) for g in order if machine[g] == m):
                for b, plate in enumerate(plates):
                    found = None
                    if plate["area"] + place.parts[p][2] <= d.bin_area:
                        found = place.best(plate, p)
                    if found:
                        r, ty, x = found[3], found[4], found[2]
                        place.put(plate, p, r, ty, x)
                        break
                else:
                    b = len(plates)
                    plates.append(place.open(m))
                    r, ty, x = place.put_new(plates[-1], p)
                log[k, m, i] = p, b, x, ty + place.parts[p][0][r].shape[0] - 1, r
            total = 0.0
            for plate in plates:
                total += (plate["pt"] + plate["pth"]) + d.setup_time
            worst = max(worst, total)
        out[k] = worst
    return (out, log.reshape(len(keys), M, -1)) if want_log else out


def _exact_greedy(inst, seed):
    place, N, M = _Placer(inst), inst.nb_parts, inst.nb_machines
    areas = np.array([p[2] for p in place.parts])
    plates, span, worst, machine, log = [], [0.0] * M, 0.0, [], []
    for p in np.lexsort((-areas, -inst.heights)):
        p, best, choice = int(p), math.inf, None
        for m in range(M):
            d = inst.problem_data.machines[m]
            h, w = place.parts[p][0][0].shape
            if (h > d.bin_length or w > d.bin_width) and (w > d.bin_length or h > d.bin_width):
                continue
            t, held = d.parts[p], False
            cand = ((span[m] + d.setup_time) + t.proc_time) + t.proc_time_height
            if max(worst, cand) <= best:
                best, choice = max(worst, cand), (m, None, None, cand)
            for plate in plates:
                found = place.best(plate, p) if plate["m"] == m else None
                if not found:
                    continue
                if plate["pth"] < t.proc_time_height:
                    cand = ((span[m] - plate["pth"]) + t.proc_time_height) + t.proc_time
                else:
                    cand = span[m] + t.proc_time
                if max(worst, cand) < best or (max(worst, cand) == best and not held):
                    held, best, choice = True, max(worst, cand), (m, plate, found, cand)
        m, plate, found, cand = choice
        if plate is None:
            plate = place.open(m)
            plate["index"] = sum(q["m"] == m for q in plates)
            plates.append(plate)
            r, ty, x = place.put_new(plate, p)
        else:
            r, ty, x = found[3], found[4], found[2]
            place.put(plate, p, r, ty, x)
        span[m] = cand
        worst = max(worst, cand)
        machine.append(m)
        log.append((p, plate["index"], x, ty + place.parts[p][0][r].shape[0] - 1, r))
    rng, chrom, thr = random.Random(seed), np.zeros(2 * N), inst.thresholds
    for m in range(M):
        genes = [log[k][0] for k in sorted((k for k in range(N) if machine[k] == m), key=lambda k: (log[k][1], k))]
        if M == 1:
            key = rng.uniform(0, 1)
        elif m == 0:
            key = rng.uniform(0, thr[0])
        elif m == M - 1:
            key = rng.uniform(thr[m - 1] + 0.0001, 1 - 0.0001)
        else:
            key = rng.uniform(thr[m - 1] + 0.0001, thr[m] - 0.0001)
        for i, v in zip(genes, np.linspace(0, 1, len(genes), endpoint=False)):
            chrom[i], chrom[i + N] = v, key
    return dict(chrom=chrom, makespan=max(span), machine=np.array(machine, np.int32),
                place=np.array(log, np.int32).reshape(-1))


def _features(inst, keys):
    """[rows, 3N + 2M] in 64 bits: per part in decode order its machine and times, per machine its area and time load."""
    N, M = inst.nb_parts, inst.nb_machines
    mach = inst.problem_data.machines
    pt = np.array([[d.parts[p].proc_time for p in range(N)] for d in mach])
    pth = np.array([[d.parts[p].proc_time_height for p in range(N)] for d in mach])
    area = np.array([float(m.sum()) for m in inst.masks])
    plate = np.array([d.bin_area for d in mach])
    rows = np.arange(len(keys))[:, None]
    m = np.stack([_machines_of(k[N:], inst, False) for k in keys])
    order = np.lexsort((keys[:, :N], m), axis=-1)
    m = m[rows, order]
    f = np.zeros((len(keys), 3 * N + 2 * M))
    f[:, 0:3 * N:3] = m / max(M - 1, 1)
    f[:, 1:3 * N:3] = pt[m, order] / pt.max()
    f[:, 2:3 * N:3] = pth[m, order] / pth.max()
    for q in range(M):
        f[:, 3 * N + 2 * q] = (area[order] / plate[q] * (m == q)).sum(1)
        f[:, 3 * N + 2 * q + 1] = (pt[q][order] / pt.max() * (m == q)).sum(1)
    return f


def _philox(c0, c1, c2, c3, k0, k1):
    """First word of Philox4x32-10 (Salmon et al., SC'11)."""
    u = np.uint64
    low = u(0xFFFFFFFF)
    c = [np.asarray(v, u) for v in np.broadcast_arrays(c0, c1, c2, c3)]
    k0, k1 = k0 & 0xFFFFFFFF, k1 & 0xFFFFFFFF
    for _ in range(10):
        a, b = c[0] * u(0xD2511F53), c[2] * u(0xCD9E8D57)
        c = [(b >> u(32)) ^ c[1] ^ u(k0), b & low, (a >> u(32)) ^ c[3] ^ u(k1), a & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c[0]


def _exact_surrogate(c, inst, seed):
    n_in = 3 * c["parts"] + 2 * c["machines"]
    in_pad = -(-n_in // 64) * 64
    flat = torch.from_numpy(_weights(n_in, in_pad, seed)).double()
    sizes = [512 * in_pad, 512, 256 * 512, 256, 256, 1]
    rows = c["history"] if c["kind"] == "train" else 512
    ms = _makespans(rows, seed)
    fine = ms < 1e15
    mu, sd = ms[fine].mean(), ms[fine].std()

    def forward(p, x):
        w1, b1, w2, b2, w3, b3 = torch.split(p, sizes)
        h = torch.relu(x @ w1.view(512, in_pad)[:, :n_in].T + b1)
        return torch.relu(h @ w2.view(256, 512).T + b2) @ w3 + b3

    if c["kind"] == "predict":
        x = torch.from_numpy(_features(inst, _keys(c["pop"], c["parts"], seed)))
        return forward(flat, x) * sd + mu
    x = torch.from_numpy(_features(inst, _keys(rows, c["parts"], [seed, 1])[fine]))
    y = torch.from_numpy((ms[fine] - mu) / sd)
    p, mom, vel = flat.clone(), torch.zeros_like(flat), torch.zeros_like(flat)
    for step in range(c["steps"]):
        nv = min(c["batch"], len(y))
        at = (_philox(np.arange(nv), step, 0x6A7, 0, 17, 0) * np.uint64(len(y)) >> np.uint64(32)).astype(np.int64)
        p.requires_grad_(True)
        ((forward(p, x[at]) - y[at]) ** 2).mean().backward()
        g, p = p.grad, p.detach()
        mom = 0.9 * mom + 0.1 * g
        vel = 0.999 * vel + 0.001 * g * g
        p = p - 1e-3 * (mom / (1 - 0.9 ** (step + 1))) / ((vel / (1 - 0.999 ** (step + 1))).sqrt() + 1e-8)
    return p


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("evaluate", "decode"):
        # about 0.4 ms a correlation; a part is tried on one or two plates where it finds room at once
        if c["pop"] * c["parts"] * max(1.0, c["parts"] / c["machines"] / 12) * (c["rows"] * c["cols"] / 62500) > 12_000:
            return None
        inst = _instance(c)
        return _exact_decode(c, inst, _keys(c["pop"], c["parts"], seed), c.get("log", False))
    if kind == "greedy":
        return _exact_greedy(_instance(c, seed % 1000), seed)
    if kind in ("predict", "train"):
        return _exact_surrogate(c, _instance(c), seed)
    return None  # a launch of many instances, a run of many decodes: minutes
