"""What is timed: the work a user of this decoder has it do, through the Python API.

Six families, each with the sizes of the tests, the benchmark and the
recipes of this repository:

* ``decode``  LLRs in device memory -> packed bits (and posteriors, iteration
  counts), flooding or layered, plain or with the trained weights;
* ``host``    LLRs in pinned host memory -> packed bits in host memory (the
  reference's call), fp32, fp16 or int8 LLRs;
* ``slot``    one slot of a base station: segment a downlink transport block,
  take the job list of an uplink one, de-rate-match, decode with early stop,
  reassemble with the block CRCs;
* ``mixed``   a job list of many codes, de-rate-matched and decoded;
* ``train``   forward and adjoint of the learned decoder;
* ``sim``     one batch of an FER measurement: generate, decode, count.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from nr_gpu_ldpc_gb300 import Decoder, Trainer, codes, segmentation
from nr_gpu_ldpc_gb300.batch import Batch, make_jobs, mixed_workload
from nr_gpu_ldpc_gb300.learned import load_weights

DEV = "cuda"
#: lifted edges x iterations of the largest listed decode: no drawn case does more
MOST_WORK = 4096 * 316 * 384 * 10
ZS = sorted(codes.LIFTING_SIZES)


def listed():
    return [
        # the smallest call: one transport block's only code block, waited for
        _decode("one_codeword", 1, 384, 1, 10),
        # a control or voice slot: a few short blocks of users at the cell's edge, early stop
        _decode("short_blocks_16", 2, 40, 16, 10, ebn0=3.0, early_stop=True, counts=True),
        # the throughput case: a full GPU of the largest code, every iteration run
        _decode("batch_4096", 1, 384, 4096, 10),
        # a ragged batch of a middle code whose posteriors are used further (soft output)
        _decode("posteriors_1001", 2, 208, 1001, 8, early_stop=True, counts=True, app=True),
        # the trained layered decoder at its operating point
        _decode("layered_learned_4096", 1, 384, 4096, 6, ebn0=1.8, early_stop=True, counts=True,
                layered=True, weights="bg1_L6"),
        # the reference testbench's batch: 40 codewords, 5 iterations, host buffers, waited for
        {"name": "host_f32_40", "family": "host", "bg": 1, "z": 384, "n": 40, "iters": 5, "ebn0": 2.0, "dtype": "f32"},
        # a large batch whose 8-bit LLRs come over the host link
        {"name": "host_i8_2000", "family": "host", "bg": 1, "z": 352, "n": 2000, "iters": 10, "ebn0": 2.0,
         "dtype": "i8"},
        # one slot of a wide carrier: a 26-block transport block each way, new job list
        {"name": "slot_26_blocks", "family": "slot", "bg": 1, "blocks": 26, "k_prime": 8424, "rate": 0.6, "qm": 6,
         "ebn0": 3.5, "iters": 10},
        # the uneven batch of many cells and users (the benchmark's mixed workload)
        {"name": "mixed_8192", "family": "mixed", "n": 8192, "jobs": 2024, "iters": 10},
        # the training configuration: BG2 Z=128, 8 iterations, one chunk of a step
        {"name": "train_flooding_4096", "family": "train", "bg": 2, "z": 128, "n": 4096, "iters": 8,
         "layered": False},
        # training of the layered decoder on the largest code, a small chunk
        {"name": "train_layered_512", "family": "train", "bg": 1, "z": 384, "n": 512, "iters": 6, "layered": True},
        # one batch of an FER curve: generate, decode with early stop, count errors
        {"name": "sim_2000", "family": "sim", "bg": 2, "z": 256, "n": 2000, "iters": 10, "ebn0": 2.5},
    ]


def _decode(name, bg, z, n, iters, ebn0=2.0, early_stop=False, app=False, layered=False, weights="", counts=False):
    c = {"family": "decode", "bg": bg, "z": z, "n": n, "iters": iters, "ebn0": ebn0, "early_stop": early_stop,
         "app": app, "want_iters": counts, "layered": layered, "weights": weights}
    if name:
        c["name"] = name
    return c


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    family = rng.choice(["decode", "decode", "decode", "host", "slot", "mixed", "train", "sim"])
    bg = rng.choice([1, 2])
    z = rng.choice([v for v in ZS if v >= 8])
    edges = 316 if bg == 1 else 197
    iters = rng.choice([5, 8, 10])
    most = max(1, min(4096, MOST_WORK // (edges * z * iters)))
    ebn0 = round(rng.uniform(1.5, 3.5), 2)
    if family == "decode":
        layered = rng.random() < 0.3
        weights = ""
        if rng.random() < 0.3:
            weights = "bg2_T8" if bg == 2 else ("bg1_L6" if layered else "bg1_T10")
        return _decode("", bg, z, log_int(1, most), iters, ebn0, rng.random() < 0.5, rng.random() < 0.25, layered,
                       weights, rng.random() < 0.5)
    if family == "host":
        return {"family": "host", "bg": bg, "z": z, "n": log_int(1, min(most, 2048)), "iters": iters, "ebn0": ebn0,
                "dtype": rng.choice(["f32", "f16", "i8"])}
    if family == "slot":
        k_max = 8448 if bg == 1 else 3840
        return {"family": "slot", "bg": bg, "blocks": rng.randint(2, 40), "k_prime": rng.randint(k_max // 2 + 40, k_max),
                "rate": round(rng.uniform(0.3, 0.85), 2), "qm": rng.choice([1, 2, 4, 6, 8, 10]), "ebn0": ebn0 + 1.5,
                "iters": iters}
    if family == "mixed":
        return {"family": "mixed", "n": log_int(16, 8192), "jobs": rng.randrange(1, 10000), "iters": iters}
    if family == "train":
        layered = rng.random() < 0.4
        z = rng.choice([64, 96, 128, 208, 256, 384])
        t = rng.choice([4, 6, 8])
        most = 4096 * 197 * 128 * 8 // (edges * z * t * (2 if layered else 1))
        return {"family": "train", "bg": bg, "z": z, "n": log_int(64, max(65, min(4096, most))), "iters": t,
                "layered": layered}
    return {"family": "sim", "bg": bg, "z": z, "n": log_int(64, min(most, 4096)), "iters": iters, "ebn0": ebn0}


# ---- inputs ---------------------------------------------------------------------------------
def _edges(bg, z):
    """[(row, column, shift)] of the lifted code, row by row."""
    h = codes.lifted_base(bg, z)
    return [(r, c, int(h[r, c])) for r in range(h.shape[0]) for c in range(h.shape[1]) if h[r, c] >= 0]


def _shape(bg):
    rows, cols = codes.BG_SHAPE[bg]
    return rows, cols, codes.KB_MAX[bg]


def _encode(bg, z, info):
    """Codewords [n, cols, z] (uint8) of the information bits [n, kb, z]."""
    rows, cols, kb = _shape(bg)
    edges = _edges(bg, z)
    n = info.shape[0]
    x = torch.zeros((n, cols, z), dtype=torch.uint8, device=info.device)
    x[:, :kb] = info
    by_row = [[(c, v) for r, c, v in edges if r == k] for k in range(rows)]

    def check(k, skip):
        acc = torch.zeros((n, z), dtype=torch.uint8, device=info.device)
        for c, v in by_row[k]:
            if c not in skip:
                acc ^= torch.roll(x[:, c], -v, 1)
        return acc

    total = torch.zeros((n, z), dtype=torch.uint8, device=info.device)
    seen = {}
    for k in range(4):  # the four core rows: the first parity column is their sum, shifted
        total ^= check(k, range(kb, cols))
        for c, v in by_row[k]:
            if c == kb:
                seen[v] = seen.get(v, 0) + 1
    shift = next(v for v, m in seen.items() if m % 2)
    x[:, kb] = torch.roll(total, shift, 1)
    solved = set(range(kb + 1))
    todo = list(range(rows))
    while todo:
        for k in todo:
            open_ = [c for c, _ in by_row[k] if c not in solved]
            if len(open_) <= 1:
                break
        if open_:  # the one unknown column of the row has shift 0
            x[:, open_[0]] = check(k, open_)
            solved.add(open_[0])
        todo.remove(k)
    return x


def _sigma(bg, ebn0, rate=None):
    rows, cols, kb = _shape(bg)
    r = kb / (cols - 2) if rate is None else rate
    return math.sqrt(1.0 / (2.0 * r * 10 ** (ebn0 / 10)))


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _llrs(bg, z, n, sigma, seed):
    """Codeword bits [n, cols*z] and their LLRs over an AWGN channel, the first
    two columns punctured.  sigma: a number, or one per codeword."""
    rows, cols, kb = _shape(bg)
    g = _generator(seed)
    info = torch.randint(0, 2, (n, kb, z), generator=g, device=DEV, dtype=torch.uint8)
    bits = _encode(bg, z, info).reshape(n, cols * z)
    s = torch.as_tensor(sigma, dtype=torch.float32, device=DEV).reshape(-1, 1)
    llr = torch.empty((n, cols * z), dtype=torch.float32, device=DEV)
    llr.normal_(generator=g)
    llr.mul_(s).add_(1.0 - 2.0 * bits.to(torch.float32)).mul_(2.0 / (s * s))
    llr[:, : 2 * z] = 0
    return bits, llr


def _pack(bits):
    """[n, m] bits -> [n, ceil(m / 8)] bytes, first bit lowest."""
    n, m = bits.shape
    b = torch.nn.functional.pad(bits, (0, -m % 8)).reshape(n, -1, 8)
    return (b << torch.arange(8, device=bits.device, dtype=torch.uint8)).sum(2).to(torch.uint8)


def _unpack(packed, m):
    b = (packed.unsqueeze(2) >> torch.arange(8, device=packed.device, dtype=torch.uint8)) & 1
    return b.reshape(packed.shape[0], -1)[:, :m]


def _train_inputs(case, seed):
    """The training recipe's channel: Eb/N0 uniform in [1, 3] dB per codeword."""
    bg, z, n = case["bg"], case["z"], case["n"]
    eb = 1.0 + 2.0 * torch.rand(n, generator=_generator(seed + 7), device=DEV)
    rows, cols, kb = _shape(bg)
    sigma = torch.sqrt(1.0 / (2.0 * (kb / (cols - 2)) * torch.pow(10.0, eb / 10.0)))
    return _llrs(bg, z, n, sigma, seed)


def _train_weights(case, seed, n_edges):
    """Weights some way into training: spread around the initial 0.75."""
    return 0.75 + 0.1 * (2.0 * torch.rand((case["iters"], n_edges), generator=_generator(seed + 3), device=DEV) - 1.0)


def _weights_of(case):
    return load_weights(case["weights"]) if case["weights"] else None


def prepare(case, seed):
    return {"case": case, **globals()["_prepare_" + case["family"]](case, seed)}


def _prepare_decode(case, seed):
    bits, llr = _llrs(case["bg"], case["z"], case["n"], _sigma(case["bg"], case["ebn0"]), seed)
    dec = Decoder(bg=case["bg"], z=case["z"], max_batch=case["n"])
    if case["layered"]:
        dec.set_schedule("layered")
    if case["weights"]:
        dec.set_weights(_weights_of(case))
    return {"dec": dec, "llr": llr}


def _prepare_host(case, seed):
    bits, llr = _llrs(case["bg"], case["z"], case["n"], _sigma(case["bg"], case["ebn0"]), seed)
    scale = 0.25
    if case["dtype"] == "f16":
        llr = llr.to(torch.float16)
    elif case["dtype"] == "i8":
        llr = torch.clamp(torch.round(llr / scale), -127, 127).to(torch.int8)
    dec = Decoder(bg=case["bg"], z=case["z"], max_batch=case["n"])
    host = torch.empty(llr.shape, dtype=llr.dtype, pin_memory=True)
    host.copy_(llr)
    out = torch.empty((case["n"], dec.packed_bytes), dtype=torch.uint8, pin_memory=True)
    return {"dec": dec, "llr": host, "out": out, "scale": scale}


def _prepare_slot(case, seed):
    bg, n, kp, qm = case["bg"], case["blocks"], case["k_prime"], case["qm"]
    n_bits = n * (kp - 24)  # two blocks or more: each carries a CRC24B
    info = segmentation.segment_info(n_bits, bg)
    z, e = info["zc"], int(kp / case["rate"]) // qm * qm
    e = max(e, -(-(2 * z + 8) // qm) * qm)
    g = _generator(seed)
    tbs = torch.randint(0, 256, (2, (n_bits + 7) // 8), generator=g, device=DEV, dtype=torch.uint8)
    if n_bits % 8:
        tbs[:, -1] &= (1 << (n_bits % 8)) - 1
    rows, cols, kb = _shape(bg)
    stride = (cols * z + 7) // 8
    blocks = torch.zeros((n, stride), dtype=torch.uint8, device=DEV)
    segmentation.segment(tbs[0], info, blocks)
    bits = torch.zeros((n, kb * z), dtype=torch.uint8, device=DEV)
    bits[:, :kp] = _unpack(blocks, kp)
    cw = _encode(bg, z, bits.reshape(n, kb, z)).reshape(n, cols * z)
    # bit selection (redundancy version 0, filler bits left out), interleaver
    keep = np.r_[2 * z:kp, kb * z:cols * z]
    pick = keep[np.arange(e) % keep.size].reshape(qm, e // qm).T.reshape(-1)
    sent = cw[:, torch.from_numpy(np.ascontiguousarray(pick)).to(DEV)].to(torch.float32)
    sigma = _sigma(bg, case["ebn0"], kp / e)
    noise = torch.empty(sent.shape, device=DEV).normal_(generator=g)
    llr_e = ((1.0 - 2.0 * sent + sigma * noise) * (2.0 / sigma ** 2)).contiguous()
    jobs, n_llr, n_e, n_out = make_jobs(np.full(n, bg), z, k_prime=kp, e=e, sigma=sigma, qm=qm)
    return {"batch": Batch(max_jobs=64), "jobs": jobs, "llr_e": llr_e.reshape(-1), "info": info, "n": n,
            "llr": torch.empty(n_llr, device=DEV), "down_tb": tbs[1],
            "down": torch.zeros((n, stride), dtype=torch.uint8, device=DEV),
            "packed": torch.zeros(n_out, dtype=torch.uint8, device=DEV),
            "up_tb": torch.zeros_like(tbs[0]), "iters": torch.zeros(n, dtype=torch.int32, device=DEV),
            "crc": torch.zeros(n, dtype=torch.int32, device=DEV)}


def _prepare_mixed(case, seed):
    bg, z, kp, e, sigma = mixed_workload(case["n"], case["jobs"])
    jobs, n_llr, n_e, n_out = make_jobs(bg, z, kp, e, 0, sigma)
    b = Batch(max_jobs=case["n"])
    b.set_jobs(jobs)
    llr_e = torch.empty(n_e, device=DEV)
    b.gen(seed, 0, llr_e, None)
    return {"batch": b, "llr_e": llr_e, "llr": torch.empty(n_llr, device=DEV),
            "packed": torch.zeros(n_out, dtype=torch.uint8, device=DEV),
            "iters": torch.zeros(case["n"], dtype=torch.int32, device=DEV)}


def _prepare_train(case, seed):
    bits, llr = _train_inputs(case, seed)
    tr = Trainer(bg=case["bg"], z=case["z"], n_iter=case["iters"], batch=case["n"], chunk=case["n"],
                 schedule="layered" if case["layered"] else "flooding")
    w = _train_weights(case, seed, tr.dec.n_edges)
    return {"trainer": tr, "llr": llr, "cw": _pack(bits), "w": w}


def _prepare_sim(case, seed):
    dec = Decoder(bg=case["bg"], z=case["z"], max_batch=case["n"])
    sigma = torch.full((case["n"],), _sigma(case["bg"], case["ebn0"]), dtype=torch.float32, device=DEV)
    return {"dec": dec, "sigma": sigma, "seed": seed}


# ---- one pass -------------------------------------------------------------------------------
def run(state):
    return globals()["_run_" + state["case"]["family"]](state["case"], state)


def _run_decode(case, s):
    r = s["dec"].decode(s["llr"], case["iters"], early_stop=case["early_stop"], want_app=case["app"],
                        want_iters=case["want_iters"], weighted=bool(case["weights"]))
    r = r if isinstance(r, tuple) else (r,)
    out = {"packed": r[0]}
    if case["app"]:
        out["app"] = r[1]
    if case["want_iters"]:
        out["iters"] = r[-1]
    return out


def _run_host(case, s):
    if case["dtype"] == "f32":
        s["dec"].decode_host(s["llr"], s["out"], case["iters"])
    else:
        s["dec"].decode_host_q(s["llr"], s["out"], case["iters"], scale=s["scale"] if case["dtype"] == "i8" else 1.0)
    torch.cuda.current_stream().synchronize()  # the bits are read on the host
    return {"packed": s["out"]}


def _run_slot(case, s):
    b = s["batch"]
    segmentation.segment(s["down_tb"], s["info"], s["down"])
    b.set_jobs(s["jobs"])
    b.derate(s["llr_e"], s["llr"])
    b.decode(s["llr"], s["packed"], case["iters"], early_stop=True, iters=s["iters"])
    segmentation.desegment(s["packed"].reshape(s["n"], -1), s["info"], s["up_tb"], s["crc"])
    return {"down": s["down"], "packed": s["packed"], "up_tb": s["up_tb"], "crc": s["crc"], "iters": s["iters"]}


def _run_mixed(case, s):
    b = s["batch"]
    b.derate(s["llr_e"], s["llr"])
    b.decode(s["llr"], s["packed"], case["iters"], early_stop=True, iters=s["iters"])
    return {"packed": s["packed"], "iters": s["iters"]}


def _run_train(case, s):
    tr = s["trainer"]
    tr.loss.zero_()
    tr.grad.zero_()
    tr.forward(s["llr"], s["cw"], 1.0 / (case["iters"] * case["n"] * tr.dec.n_bp), weights=s["w"])
    tr.backward(case["n"], weights=s["w"])
    return {"loss": tr.loss.float(), "grad": tr.grad.float()}


def _run_sim(case, s):
    dec = s["dec"]
    llr, cw = dec.gen_llr(seed=s["seed"], cw_base=0, sigma=s["sigma"])
    packed, iters = dec.decode(llr, case["iters"], early_stop=True, want_iters=True)
    return {"llr": llr, "cw": cw, "packed": packed, "iters": iters, "counts": dec.count_errors(packed, cw)}


# ---- what a pass cannot do without ----------------------------------------------------------
#: flops of one lifted edge in one iteration: old message out, two-min (2), new
#: message, its difference, posterior
EDGE_FLOPS = 6


def work(case):
    f, it = case["family"], case["iters"]
    if f == "mixed":
        bg, z, kp, e, sigma = mixed_workload(case["n"], case["jobs"])
        edges = np.where(bg == 1, 316, 197) * z
        cols = np.where(bg == 1, 68, 52) * z
        # early stop: about half of the iterations at these signal-to-noise ratios
        return {"bytes": float((4 * e + 4 * cols + cols / 8 + 4).sum()), "flops": float(EDGE_FLOPS * it / 2 * edges.sum())}
    bg = case["bg"]
    rows, cols, kb = _shape(bg)
    if f == "slot":
        n, kp = case["blocks"], case["k_prime"]
        z = segmentation.segment_info(n * (kp - 24), bg)["zc"]
        return {"bytes": n * (4 * kp / case["rate"] + 4 * kp / 8 + cols * z / 8),
                "flops": EDGE_FLOPS * it / 2 * n * z * (316 if bg == 1 else 197)}
    n, z = case["n"], case["z"]
    bits, edges = n * cols * z, n * z * (316 if bg == 1 else 197)
    if f == "train":  # forward and adjoint
        return {"bytes": 4 * bits + bits / 8, "flops": 3 * EDGE_FLOPS * it * edges}
    if f == "sim":
        return {"bytes": 4 * bits + bits / 4, "flops": EDGE_FLOPS * it / 2 * edges + 20 * bits}
    llr = {"f32": 4, "f16": 2, "i8": 1}[case.get("dtype", "f32")]
    return {"bytes": llr * bits + bits / 8 + (4 * bits if case.get("app") else 0),
            "flops": EDGE_FLOPS * (it / 2 if case.get("early_stop") else it) * edges}


# ---- the same in 64 bits, in plain torch ----------------------------------------------------
def exact(case, seed):
    f = case["family"]
    if f == "decode" and case["app"]:
        bits, llr = _llrs(case["bg"], case["z"], case["n"], _sigma(case["bg"], case["ebn0"]), seed)
        return {"app": _exact_posteriors(case, llr.double())}
    if f == "train":
        return _exact_train(case, seed)
    if f == "sim":
        return {"llr": _exact_llr(case, seed)}
    return None  # bytes and counts


def _rows(bg, z):
    rows = [[] for _ in range(_shape(bg)[0])]
    for k, (r, c, v) in enumerate(_edges(bg, z)):
        rows[r].append((k, c, v))
    return rows


def _messages(q, w):
    """Weighted min-sum messages of the incoming q [D, n, z]; w: [D] or a number."""
    sign = torch.where(q < 0, -1.0, 1.0).to(q.dtype).detach()
    mag = torch.clamp(q * sign, max=1000.0)
    first = mag.detach().argmin(0, keepdim=True)
    at = torch.zeros_like(mag, dtype=torch.bool).scatter_(0, first, True)
    m1 = mag.gather(0, first)
    if q.shape[0] > 1:
        m2 = mag.masked_fill(at, 1000.0).amin(0, keepdim=True) if not mag.requires_grad else \
            mag.gather(0, mag.detach().masked_fill(at, 2000.0).argmin(0, keepdim=True))
    else:
        m2 = torch.full_like(m1, 1000.0)
    w = w.reshape(-1, 1, 1) if isinstance(w, torch.Tensor) else w
    return w * sign * sign.prod(0, keepdim=True) * torch.where(at, m2, m1)


def _iteration(rows, cols, msgs, w, layered):
    """One iteration over the posteriors (a list of columns [n, z]); msgs: the
    rows' previous messages (None at first).  Returns the new ones of both."""
    new = list(cols)
    out = []
    for r, edges in enumerate(rows):
        src = new if layered else cols
        old = msgs[r] if msgs is not None else None
        q = torch.stack([torch.roll(src[c], -v, 1) for _, c, v in edges])
        q = q if old is None else q - old
        m = _messages(q, w[edges[0][0]: edges[-1][0] + 1] if isinstance(w, torch.Tensor) else w)
        for i, (_, c, v) in enumerate(edges):
            d = m[i] if old is None else m[i] - old[i]
            new[c] = new[c] + torch.roll(d, v, 1)
        out.append(m)
    return new, out


def _exact_posteriors(case, llr):
    bg, z, n = case["bg"], case["z"], case["n"]
    rows, n_cols = _rows(bg, z), _shape(bg)[1]
    w = _weights_of(case)
    w = None if w is None else torch.from_numpy(w).to(DEV).double()
    cols = list(llr.reshape(n, n_cols, z).unbind(1))
    final, done, msgs = llr.clone(), torch.zeros(n, dtype=torch.bool, device=DEV), None
    for t in range(case["iters"]):
        cols, msgs = _iteration(rows, cols, msgs, 0.75 if w is None else w[min(t, len(w) - 1)], case["layered"])
        app = torch.stack(cols, 1).reshape(n, -1)
        final = torch.where(done.unsqueeze(1), final, app)
        if case["early_stop"]:
            hard = [(c <= 0) for c in cols]
            bad = torch.zeros(n, dtype=torch.bool, device=DEV)
            for edges in rows:
                s = torch.zeros_like(hard[0])
                for _, c, v in edges:
                    s = s ^ torch.roll(hard[c], -v, 1)
                bad |= s.any(1)
            done |= ~bad
    return final


def _exact_train(case, seed):
    bg, z, n, steps = case["bg"], case["z"], case["n"], case["iters"]
    bits, llr = _train_inputs(case, seed)
    rows, n_cols = _rows(bg, z), _shape(bg)[1]
    n_edges = sum(len(r) for r in rows)
    part = max(1, int(4e9 // (n_edges * z * 8 * steps * 8)))
    if n * n_edges * z * steps > 1.1 * 4096 * 197 * 128 * 8:
        return None
    w = _train_weights(case, seed, n_edges).double().requires_grad_(True)
    total = torch.zeros((), dtype=torch.float64, device=DEV)
    for k in range(0, n, part):
        x = llr[k: k + part].double()
        y = 1.0 - 2.0 * bits[k: k + part].double()
        cols, msgs = list(x.reshape(-1, n_cols, z).unbind(1)), None
        loss = 0.0
        for t in range(steps):
            cols, msgs = _iteration(rows, cols, msgs, w[t], case["layered"])
            loss = loss + torch.nn.functional.softplus(-y * torch.stack(cols, 1).reshape(x.shape)).sum()
        loss = loss / (steps * n * n_cols * z)
        loss.backward()
        total += loss.detach()
    # layered: 32-bit rounding decides between near-tied minima, and another
    # edge then receives the gradient, so 64 bits have no value to compare with
    return {"loss": total.reshape(1), "grad": None if case["layered"] else w.grad}


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 on int64 tensors that hold 32-bit words."""
    low = 0xFFFFFFFF

    def mul(a, b):  # high and low words of a 64-bit product of 32-bit words, in 16-bit parts
        a1, a0 = a >> 16, a & 0xFFFF
        mid = a1 * b
        p0 = a0 * b
        hi = (mid + (p0 >> 16)) >> 16
        return hi & low, ((mid << 16) + p0) & low

    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c0)
        h1, l1 = mul(0xCD9E8D57, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & low, (k1 + 0xBB67AE85) & low
    return c0, c1, c2, c3


def _exact_llr(case, seed):
    """The seeded channel: information bits and noise from Philox counters
    (block, codeword, codeword >> 32, stream), Box-Muller, LLR = 2y/sigma^2."""
    bg, z, n = case["bg"], case["z"], case["n"]
    rows, cols, kb = _shape(bg)
    cw = torch.arange(n, device=DEV, dtype=torch.int64).reshape(n, 1)
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32

    def words(count, stream):
        t = torch.arange(count, device=DEV, dtype=torch.int64).reshape(1, count).expand(n, count)
        zero = torch.zeros_like(t)
        return _philox(t, cw.expand(n, count), zero, zero + stream, k0, k1)

    o = torch.stack(words(-(-kb * z // 128), 1), 2)
    info = ((o.unsqueeze(3) >> torch.arange(32, device=DEV)) & 1).reshape(n, -1)[:, : kb * z].to(torch.uint8)
    bits = _encode(bg, z, info.reshape(n, kb, z)).reshape(n, -1)
    m = (cols - 2) * z
    o = words(-(-m // 4), 2)
    g = []
    for a, b in ((o[0], o[1]), (o[2], o[3])):
        u1, u2 = ((a >> 8) + 1).double() * 2.0 ** -24, (b >> 8).double() * 2.0 ** -24
        rad = torch.sqrt(-2.0 * torch.log(u1))
        g += [rad * torch.cos(2 * math.pi * u2), rad * torch.sin(2 * math.pi * u2)]
    noise = torch.stack(g, 2).reshape(n, -1)[:, :m]
    sigma = float(np.float32(_sigma(bg, case["ebn0"])))
    llr = torch.zeros((n, cols * z), dtype=torch.float64, device=DEV)
    llr[:, 2 * z:] = (1.0 - 2.0 * bits[:, 2 * z:].double() + sigma * noise) * (2.0 / sigma ** 2)
    return llr
