"""The work this library is timed on: what a program that compiles detector error models asks of it.

Each case is one public entry point at one size.  ``listed()`` gives the fixed cases, ``draw(rng)`` more
of the same ranges, ``prepare`` what a program holds before the call (circuit texts, a driver, a
template, a server, device buffers), ``run`` the call, ``work`` the bytes and operations it cannot do
without, and ``exact`` the answer in 64-bit numpy.

The circuits are the repository's own: rotated surface-code and bivariate-bicycle memories with rounds
up to the distance, uniform noise whose every instruction has its own rate (log-uniform in
[1e-4, 1e-2]), one round in ten taking the basis-switch branch.
"""

from __future__ import annotations

import ctypes
import functools
import math
import random
import re

import numpy as np
import torch

import greenpeas_gb300 as gp
from greenpeas_gb300 import _native
from greenpeas_gb300.autograd import NoiseRateDEM
from greenpeas_gb300.codes import BBCode, SurfaceCode
from greenpeas_gb300.serving import Server

P_LO, P_HI = 1e-4, 1e-2
SENTINEL = 0.000123456789
BB_DISTANCES = (6, 12, 18)
EXACT_MECHANISMS = 250_000  # largest circuit whose exact answer is worked out (a few seconds)


# ---- the cases ----------------------------------------------------------------


def listed() -> list:
    return [
        # One circuit, text in and host arrays out (get_driver(...).compile_detector_error_model):
        # the smallest memory there is, where the call's latency counts ...
        _circuit("compile", "surface", 3, 3, name="compile_surface3_r3"),
        # ... the library's headline circuit, the [[144,12,12]] code ...
        _circuit("compile", "bb", 12, 12, name="compile_bb12_r12"),
        # ... and a large surface code.
        _circuit("compile", "surface", 21, 21, name="compile_surface21_r21"),
        # One prepared circuit run again with its result left on the device, as a decoder on the
        # same GPU reads it: a small code at a lower correlation level ...
        _circuit("device", "bb", 6, 6, level=1, name="device_bb6_r6_L1"),
        # ... the headline circuit ...
        _circuit("device", "bb", 12, 12, name="device_bb12_r12"),
        # ... and the largest circuit of the serving mix.
        _circuit("device", "surface", 25, 25, name="device_surface25_r25"),
        # Long idling between rounds: every idle step repeats the same symptoms, more often than a
        # merge bucket holds, so the whole circuit is sorted.
        {"kind": "idle", "d": 5, "rounds": 5, "idle": 300, "level": 2, "name": "device_idle300_surface5"},
        # Many circuits of mixed sizes in one call, text in and host arrays out.
        {"kind": "batch", "n": 21, "dmax": 21, "level": 2, "name": "batch21_surface3to21"},
        # A prepared batch run again, its results left on the device: the library's batch workload.
        {"kind": "device_batch", "n": 256, "dmax": 21, "level": 2, "name": "device_batch256_surface3to21"},
        # Noise calibration: merged probabilities of a rate tensor and their gradient (forward and backward).
        _circuit("grad", "bb", 12, 12, name="grad_bb12_r12"),
        # Raw mechanisms already on the device, merged without allocating.
        {"kind": "merge", "n": 50001, "stride": 16, "copies": 2.5, "name": "merge_static_50001"},
        # A burst of requests to the compile server: surface and bicycle codes mixed.
        {"kind": "serve", "n": 21, "dmax": 25, "name": "serve_burst21"},
    ]


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["compile", "compile", "device", "device", "idle", "batch", "device_batch", "grad", "merge",
                       "serve"])
    level = rng.choice([0, 1, 2, 2])
    if kind in ("compile", "device"):
        code, d, rounds = _draw_code(rng, 21 if kind == "compile" else 25)
        return _circuit(kind, code, d, rounds, level=level, branch=rng.randrange(1000))
    if kind == "grad":
        code, d, rounds = _draw_code(rng, 12)
        return _circuit(kind, code, d, rounds, level=level, branch=rng.randrange(1000))
    if kind == "idle":
        return {"kind": kind, "d": rng.choice([3, 5]), "rounds": rng.randint(1, 5),
                "idle": _log_int(rng, 40, 300), "level": level}
    if kind == "batch":
        dmax = rng.choice(range(5, 23, 2))
        return {"kind": kind, "n": _log_int(rng, 2, 21), "dmax": dmax, "level": level}
    if kind == "device_batch":
        dmax = rng.choice(range(5, 23, 2))
        return {"kind": kind, "n": _log_int(rng, 2, 200), "dmax": dmax, "level": level}
    if kind == "merge":
        return {"kind": kind, "n": _log_int(rng, 100, 50001), "stride": rng.choice([8, 12, 16]),
                "copies": rng.choice([1.2, 2.5, 6.0])}
    return {"kind": kind, "n": _log_int(rng, 3, 21), "dmax": rng.choice(range(5, 27, 2))}


def _circuit(kind, code, d, rounds, level=2, branch=0, **kw) -> dict:
    return {"kind": kind, "code": code, "d": d, "rounds": rounds, "level": level, "branch": branch, **kw}


def _log_int(rng, lo, hi) -> int:
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _draw_code(rng, dmax):
    """(code, distance, rounds): rounds log-spread from 1 to the largest distance (bicycle codes: the code's)."""
    if rng.random() < 0.4:
        d = rng.choice([x for x in BB_DISTANCES if x <= dmax])
        return "bb", d, _log_int(rng, 1, d)
    d = rng.choice(range(3, dmax + 1, 2))
    return "surface", d, _log_int(rng, 1, dmax)


# ---- circuit texts ------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _code(code, d):
    return SurfaceCode(d) if code == "surface" else BBCode(d)


@functools.lru_cache(maxsize=None)
def _pieces(code, d, rounds, switch):
    """The memory's text cut at its noise rates."""
    text = _code(code, d).get_memory(rounds, SENTINEL, noise="uniform", switch_rounds=switch)
    return re.split(r"\(0\.000123456789\)", text)


def _text(rng, code, d, rounds, branch) -> str:
    """A memory that switches a tenth of its rounds (chosen by ``branch``) and whose every noise
    instruction draws its rate."""
    pick = random.Random(f"{code} {d} {rounds} {branch}")
    pieces = _pieces(code, d, rounds, tuple(r for r in range(rounds) if pick.random() < 0.1))
    out = [pieces[0]]
    for piece in pieces[1:]:
        out.append(f"({_rate(rng):.6g})")
        out.append(piece)
    return "".join(out)


def _rate(rng) -> float:
    return math.exp(rng.uniform(math.log(P_LO), math.log(P_HI)))


def _idle_text(case, rng) -> str:
    """A surface memory that idles after the reset of each round's checks: ``idle`` steps of
    depolarizing noise on the data qubits."""
    code = _code("surface", case["d"])
    data = " ".join(str(q) for q in range(code.num_data))
    text = code.get_memory(case["rounds"], _rate(rng), noise="uniform")
    out, resets = [], 0
    for line in text.splitlines():
        out.append(line)
        if line.startswith("R "):
            resets += 1
            if resets > 1:
                out.append(f"REPEAT {case['idle']} {{\n    DEPOLARIZE1({_rate(rng) / 100:.6g}) {data}\n    TICK\n}}")
    return "\n".join(out) + "\n"


def _texts(case, seed) -> list:
    """The case's circuits: their shapes from the case, their noise rates from the seed."""
    kind, rng = case["kind"], random.Random(f"{case['kind']} {seed}")
    if kind == "idle":
        return [_idle_text(case, rng)]
    if kind not in ("batch", "device_batch", "serve"):
        return [_text(rng, case["code"], case["d"], case["rounds"], case["branch"])]
    shapes, out = random.Random(f"{kind} {case['n']} {case['dmax']}"), []
    for _ in range(case["n"]):
        if kind == "serve" and shapes.random() < 0.5:
            code, d = "bb", shapes.choice(BB_DISTANCES)
        else:
            code, d = "surface", shapes.choice(range(5 if kind == "serve" else 3, case["dmax"] + 1, 2))
        out.append(_text(rng, code, d, d, shapes.randrange(3)))  # (three branches of each: texts are quick to make)
    return out


# ---- what a program holds, and its call ---------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind == "merge":
        return _prepare_merge(case, seed)
    texts = _texts(case, seed)
    if kind == "serve":
        return {"case": case, "texts": texts, "server": Server()}
    if kind == "grad":
        model = NoiseRateDEM(texts[0], correlation_level=case["level"])
        noise = torch.from_numpy(_rates(model.shape, seed)).cuda().requires_grad_()
        n = model(noise.detach()).numel()
        return {"case": case, "model": model, "noise": noise, "weights": torch.from_numpy(_weights(n, seed)).cuda()}
    driver = gp.get_driver(texts[0], gp.CorrelationLevel(case["level"]))
    if kind in ("device", "idle"):
        driver.prepare(texts[0])
    elif kind == "device_batch":
        driver.prepare_batch(texts)
    return {"case": case, "driver": driver, "texts": texts}


def _rates(shape, seed):
    rng = np.random.default_rng([seed, 1])
    return np.exp(rng.uniform(math.log(5e-4), math.log(5e-3), size=shape))


def _weights(n, seed):
    return np.random.default_rng([seed, 2]).standard_normal(n)


def _mechanisms(case, seed):
    """Raw mechanisms as a circuit's noise makes them: symptoms of one to seven nearby detectors,
    each made by ``copies`` mechanisms on average."""
    rng = np.random.default_rng([seed, 3])
    n, stride = case["n"], case["stride"]
    distinct = max(1, int(n / case["copies"]))
    size = np.minimum(rng.choice([1, 2, 3, 4, 5, 6, 7], p=[0.08, 0.3, 0.22, 0.25, 0.06, 0.06, 0.03], size=distinct),
                      stride)
    gaps = rng.integers(1, 60, size=(distinct, stride))
    lists = rng.integers(0, 12000, size=(distinct, 1)) + np.cumsum(gaps, axis=1)
    which = rng.integers(0, distinct, size=n)
    size, lists = size[which].astype(np.int32), lists[which].astype(np.int32)
    lists[np.arange(stride)[None, :] >= size[:, None]] = 0
    probs = np.exp(rng.uniform(math.log(1e-6), math.log(1e-3), size=n))
    return size, lists, probs


def _prepare_merge(case, seed):
    size, lists, probs = _mechanisms(case, seed)
    n, cap = case["n"], 7 * case["n"]
    return {
        "case": case,
        "num_targets": torch.from_numpy(size).cuda(),
        "targets": torch.from_numpy(lists.reshape(-1)).cuda(),
        "probs": torch.from_numpy(probs).cuda(),
        "out_probs": torch.zeros(n, dtype=torch.float64, device="cuda"),
        "out_offsets": torch.zeros(n + 1, dtype=torch.int32, device="cuda"),
        "out_targets": torch.zeros(cap, dtype=torch.int32, device="cuda"),
        "result": torch.zeros(4, dtype=torch.int32, device="cuda"),
    }


def run(state):
    kind = state["case"]["kind"]
    if kind == "compile":
        return _host(state["driver"].compile_detector_error_model(state["texts"][0]))
    if kind in ("device", "idle"):
        state["driver"].run_device()
        return _held(state["driver"], state["driver"].device_dem())
    if kind == "batch":
        return [_host(dem) for dem in state["driver"].compile_batch(state["texts"])]
    if kind == "device_batch":
        state["driver"].run_device()
        return _gather(state["driver"], state["case"]["n"])
    if kind == "grad":
        probs = state["model"](state["noise"])
        loss = (state["weights"] * probs.log()).sum()
        (grad,) = torch.autograd.grad(loss, state["noise"])
        return [probs.detach(), grad]
    if kind == "merge":
        return _run_merge(state)
    tickets = [state["server"].submit(text) for text in state["texts"]]
    return [_host(state["server"].result(t)) for t in tickets]


def _held(driver, arrays) -> list:
    for a in arrays:
        a.driver = driver  # the arrays are views of its buffers
    return list(arrays)


def _gather(driver, n) -> list:
    """Every circuit's model in one set of arrays of the program's own, copied on the driver's stream."""
    dems = [driver.device_dem(i) for i in range(n)]
    with torch.cuda.stream(torch.cuda.ExternalStream(driver.stream)):
        return [torch.cat([d[0] for d in dems]), torch.cat([d[1] for d in dems]), dems[-1][2].clone()]


def _host(dem) -> list:
    return [dem.probs, dem.offsets, dem.targets]


def _run_merge(state):
    case = state["case"]

    def p(name):
        return ctypes.c_void_p(state[name].data_ptr())

    _native.check(_native.lib().gpc_merge_mechanisms_static(
        p("num_targets"), p("targets"), case["stride"], p("probs"), case["n"], p("out_probs"), p("out_offsets"),
        p("out_targets"), 7 * case["n"], p("result"), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return [state["out_probs"], state["out_offsets"], state["out_targets"], state["result"]]


# ---- what a pass cannot do without ----------------------------------------------

# Merged errors per raw mechanism and targets per merged error of the two code families, as the 64-bit
# answers count them at level 2 (the lower levels keep fewer mechanisms of nearly the same symptoms).
MERGED = {"surface": 0.33, "bb": 0.41}
TARGETS = {"surface": 3.4, "bb": 8.1}


@functools.lru_cache(maxsize=None)
def _counts(code, d, rounds, level):
    """(text bytes, noise records, raw mechanisms) of a memory."""
    text = "(0.001234)".join(_pieces(code, d, rounds, ()))
    one, two = {0: (2, 6), 1: (3, 10), 2: (3, 15)}[level]
    records = mechanisms = 0
    for line in text.splitlines():
        name, _, rest = line.partition(" ")
        k = len(rest.split())
        if name.startswith("X_ERROR"):
            records, mechanisms = records + k, mechanisms + k
        elif name.startswith("DEPOLARIZE1"):
            records, mechanisms = records + k, mechanisms + one * k
        elif name.startswith("DEPOLARIZE2"):
            records, mechanisms = records + k // 2, mechanisms + two * (k // 2)
    return len(text), records, mechanisms


def _dem_bytes(code, mechanisms) -> float:
    return MERGED[code] * mechanisms * (8 + 4 + 4 * TARGETS[code])


def work(case) -> dict:
    kind, level = case["kind"], case.get("level", 2)
    if kind == "merge":
        merged = min(case["n"], case["n"] / case["copies"])
        return {"bytes": case["n"] * (4 + 8 + 4 * 3.2) + merged * (12 + 4 * 3.2), "flops": 3.0 * case["n"]}
    if kind == "idle":
        idle = (2 if level == 0 else 3) * case["idle"] * case["d"] ** 2 * case["rounds"]
        _, records, mechanisms = _counts("surface", case["d"], case["rounds"], level)
        records += case["idle"] * case["d"] ** 2 * case["rounds"]
        return {"bytes": records * 16 + _dem_bytes("surface", mechanisms), "flops": 3.0 * (idle + mechanisms)}
    if kind in ("batch", "device_batch"):
        ds = range(3, case["dmax"] + 1, 2)
        codes = [("surface", d, d, case["n"] / len(ds)) for d in ds]
    elif kind == "serve":
        ds = range(5, case["dmax"] + 1, 2)
        codes = [("surface", d, d, case["n"] / 2 / len(ds)) for d in ds]
        codes += [("bb", d, d, case["n"] / 2 / len(BB_DISTANCES)) for d in BB_DISTANCES]
    else:
        codes = [(case["code"], case["d"], case["rounds"], 1)]
    total = flops = 0.0
    for code, d, rounds, n in codes:
        text, records, mechanisms = _counts(code, d, rounds, level)
        # text for the calls that take it, the noise records (16 bytes) for the prepared ones
        read = text if kind in ("compile", "batch", "serve") else 16 * records
        total += n * (read + _dem_bytes(code, mechanisms))
        flops += n * 3.0 * mechanisms * (3 if kind == "grad" else 1)
    return {"bytes": total, "flops": flops}


# ---- the answer in 64 bits --------------------------------------------------------


def exact(case, seed):
    if case["kind"] == "merge":
        return _exact_merge(case, seed)
    if case["kind"] in ("batch", "device_batch", "serve"):
        return None  # many circuits: minutes
    if case["kind"] == "idle":
        if case["idle"] * case["d"] ** 2 * case["rounds"] * 3 > EXACT_MECHANISMS:
            return None
    elif _counts(case["code"], case["d"], case["rounds"], case["level"])[2] > EXACT_MECHANISMS:
        return None
    text = _texts(case, seed)[0]
    if case["kind"] != "grad":
        words, p, _, _, _ = _symptoms(text, case["level"], None)
        dem = _merge(words, p, _order)[0]
        # a program on the device gets signed offsets and targets
        kinds = (np.float64, np.uint32, np.uint32) if case["kind"] == "compile" else (np.float64, np.int32, np.int32)
        return [a.astype(t) for a, t in zip(dem, kinds)]
    ticks = _ticks(text)
    rates = _rates((ticks, 4), seed)
    words, p, src, slope, _ = _symptoms(text, case["level"], rates.reshape(-1))
    (probs, _, _), group = _merge(words, p, _order)
    dl = _weights(probs.size, seed) / probs
    keep = group >= 0
    # dL/dq_m = dL/dp_g prod_{j != m} (1 - 2 q_j), and p_g = (1 - prod (1 - 2 q)) / 2
    rest = (1 - 2 * probs[group[keep]]) / (1 - 2 * p[keep])
    grad = np.zeros(ticks * 4)
    np.add.at(grad, src[keep], dl[group[keep]] * rest * slope[keep])
    return [probs, grad.reshape(ticks, 4)]


def _ticks(text) -> int:
    return sum(line.strip() == "TICK" for line in text.splitlines()) + 1


def _flat(text):
    """(name, argument, targets) of every instruction, repetitions unrolled (none nested)."""
    out, body, times = [], None, 0
    for line in text.splitlines():
        line = line.strip()
        if line.startswith("REPEAT"):
            body, times = [], int(line.split()[1])
        elif line == "}":
            out += body * times
            body = None
        elif line:
            m = re.match(r"([A-Z_0-9]+)(?:\(([^)]*)\))?\s*(.*)", line)
            (out if body is None else body).append((m[1], m[2], m[3].split()))
    return out


ONE = {0: [(1, 0), (0, 1)], 1: [(1, 0), (1, 1), (0, 1)], 2: [(1, 0), (1, 1), (0, 1)]}  # (X, Z) of X, Y, Z
PAULI = {"I": (0, 0), "X": (1, 0), "Y": (1, 1), "Z": (0, 1)}
TWO = {0: "IX IZ XI XX ZI ZZ", 1: "IX IY IZ XI XX XZ YI ZI ZX ZZ",
       2: "IX IY IZ XI XX XY XZ YI YX YY YZ ZI ZX ZY ZZ"}


def _symptoms(text, level, rates):
    """Every mechanism's symptom words, probability, noise source, slope of the probability in its
    source's rate, and the bit count: sensitivities of X and Z on each qubit carried backward."""
    ins = _flat(text)
    ndet = sum(name == "DETECTOR" for name, _, _ in ins)
    nq = 1 + max(int(t) for name, _, ts in ins for t in ts if t.isdigit())
    flips, meas, det, tick, reset, src = {}, 0, 0, 0, {}, []
    for name, arg, ts in ins:  # the bits each measurement feeds, and each instruction's noise sources
        src.append((meas, tick, [reset.get(t, False) for t in ts] if name == "X_ERROR" else None))
        if name == "M":
            meas += len(ts)
            reset.update((t, False) for t in ts)
        elif name == "R":
            reset.update((t, True) for t in ts)
        elif name in ("H", "CX"):
            reset.update((t, False) for t in ts)
        elif name == "TICK":
            tick += 1
        elif name in ("DETECTOR", "OBSERVABLE_INCLUDE"):
            bit = det if name == "DETECTOR" else ndet + int(arg)
            det += name == "DETECTOR"
            for t in ts:
                flips.setdefault(meas + int(t[4:-1]), []).append(bit)
    bits = ndet + 1 + max([int(arg) for name, arg, _ in ins if name == "OBSERVABLE_INCLUDE"], default=-1)
    w = (bits + 63) // 64
    X, Z = np.zeros((nq, w), np.uint64), np.zeros((nq, w), np.uint64)
    words, probs, sources, slopes = [], [], [], []

    def add(rows, kind, arg, source):
        p = float(arg) if rates is None else rates[source]
        p = np.broadcast_to(np.asarray(p, np.float64), (rows.shape[0],))
        q, slope = _split(p, kind)
        k = rows.shape[1]
        words.append(rows.reshape(-1, w))
        probs.append(np.repeat(q, k))
        slopes.append(np.repeat(slope, k))
        sources.append(np.repeat(np.broadcast_to(source, (rows.shape[0],)), k))

    for (name, arg, ts), (first, at, after_reset) in zip(reversed(ins), reversed(src)):
        if name in ("TICK", "DETECTOR", "OBSERVABLE_INCLUDE"):
            continue
        q = np.array([int(t) for t in ts])
        if name == "H":
            X[q], Z[q] = Z[q], X[q]
        elif name == "R":
            X[q], Z[q] = 0, 0
        elif name == "CX":
            c, t = q[0::2], q[1::2]
            X[c] ^= X[t]
            Z[t] ^= Z[c]
        elif name == "M":
            for k, x in enumerate(q):
                for b in flips.get(first + k, ()):
                    X[x, b >> 6] ^= np.uint64(1 << (b & 63))
        elif name == "X_ERROR":
            add(X[q][:, None], 0, arg, at * 4 + np.where(after_reset, 3, 2))
        elif name == "DEPOLARIZE1":
            add(np.stack([X[q] * np.uint64(x) ^ Z[q] * np.uint64(z) for x, z in ONE[level]], 1), 1, arg, at * 4 + 1)
        elif name == "DEPOLARIZE2":
            a, b = q[0::2], q[1::2]
            comps = []
            for pair in TWO[level].split():
                (xa, za), (xb, zb) = PAULI[pair[0]], PAULI[pair[1]]
                comps.append(X[a] * np.uint64(xa) ^ Z[a] * np.uint64(za) ^ X[b] * np.uint64(xb) ^ Z[b] * np.uint64(zb))
            add(np.stack(comps, 1), 2, arg, at * 4)
        else:
            raise ValueError(name)
    return np.concatenate(words), np.concatenate(probs), np.concatenate(sources), np.concatenate(slopes), bits


def _split(p, kind):
    """Probability of one component of a channel of rate p, and its slope in p."""
    if kind == 0:
        return p, np.ones_like(p)
    a, n = (4 / 3, 2) if kind == 1 else (16 / 15, 8)  # (1 - (1 - a p)^(1/n)) / 2
    log = np.log1p(-a * p) / n
    return -np.expm1(log) / 2, a / (2 * n) * np.exp(log) / (1 - a * p)


def _mix(k):
    """The 64-bit finaliser of MurmurHash3."""
    k ^= k >> np.uint64(33)
    k *= np.uint64(0xFF51AFD7ED558CCD)
    k ^= k >> np.uint64(33)
    k *= np.uint64(0xC4CEB9FE1A85EC53)
    return k ^ (k >> np.uint64(33))


def _keys(words):
    """The 128-bit symptom keys that order a compiled model."""
    x, y = np.zeros(len(words), np.uint64), np.zeros(len(words), np.uint64)
    with np.errstate(over="ignore"):
        for j in range(words.shape[1]):
            v, jj = words[:, j], np.uint64(j + 1)
            on = v != 0
            v = v[on]
            x[on] ^= _mix(v * np.uint64(0x9E3779B97F4A7C15) + jj * np.uint64(0xC2B2AE3D27D4EB4F))
            y[on] ^= _mix(v * np.uint64(0xD6E8FEB86659FD93) + jj * np.uint64(0xA0761D6478BD642F)
                          + np.uint64(0x8EBC6AF09C88C6E3))
    return x, y


def _order(x, y, mechanisms):
    """Order of a compiled model's errors: by key bucket (a power of two of them, 16 to 96 mechanisms
    each), then the top bits of the second key half, then the key; by the key alone when a symptom
    fills more than a bucket."""
    mean = 16 if mechanisms <= 16 << 10 else 48 if mechanisms <= 256 << 10 else 96
    b = 4
    while b < 18 and mean << b < mechanisms:
        b += 1
    bucket = x >> np.uint64(64 - b)
    if np.bincount(bucket.astype(np.int64)[(x | y) != 0], minlength=1).max() > 256:
        return np.lexsort((y, x))
    return np.lexsort((y, x, y >> np.uint64(58), bucket))


def _merge(words, p, order):
    """(probabilities, offsets, targets) of the distinct non-empty symptoms, and each mechanism's (-1: empty)."""
    x, y = _keys(words)
    at = order(x, y, len(words))
    at = at[(x[at] | y[at]) != 0]
    group = np.full(len(words), -1)
    if at.size == 0:
        return (np.zeros(0), np.zeros(1, np.int64), np.zeros(0, np.int64)), group
    head = np.ones(at.size, bool)
    head[1:] = (x[at[1:]] != x[at[:-1]]) | (y[at[1:]] != y[at[:-1]])
    start = np.flatnonzero(head)
    group[at] = np.cumsum(head) - 1
    # (1 - prod (1 - 2 p)) / 2
    probs = -np.expm1(np.add.reduceat(np.log1p(-2 * p[at]), start)) / 2
    rows = np.ascontiguousarray(words[at[start]].astype("<u8")).view(np.uint8)
    row, target = np.nonzero(np.unpackbits(rows, axis=1, bitorder="little"))
    offsets = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=start.size))])
    return (probs, offsets, target), group


def _exact_merge(case, seed):
    size, lists, p = _mechanisms(case, seed)
    n = case["n"]
    words = np.zeros((n, (int(lists.max()) + 64) // 64), np.uint64)
    for k in range(case["stride"]):
        on = np.flatnonzero(k < size)
        t = lists[on, k]
        words[on, t >> 6] |= np.uint64(1) << (t & 63).astype(np.uint64)
    (probs, offsets, targets), _ = _merge(words, p, lambda x, y, m: np.lexsort((y, x)))
    out = [np.zeros(n), np.zeros(n + 1, np.int32), np.zeros(7 * n, np.int32), np.zeros(4, np.int32)]
    out[0][:probs.size] = probs
    out[1][:offsets.size] = offsets
    out[2][:targets.size] = targets
    out[3][:2] = probs.size, targets.size
    return out
