"""Speed cases: what users of this correlator have it do, through its public entry points.

A case is one pass of one of four kinds of work:

* "engine": frames already in device memory correlated into one row, which is divided by the
  frame count (FxEngine: accumulate, then scale of a complex64 row or dump of a complex128 row);
* "batch": several integration blocks of uneven length in one graph launch (corrx_batch_*);
* "frontend": the synthetic front end writing frames and their validity mask on the device;
* "abi": a row through the C ABI from the pinned staging ring to host memory (Correlator).

X-engine modes: 0 plain FP32, 1 tensor FP16, 2 tensor FP16 split.
"""

import ctypes
import importlib
import math

import numpy as np
import torch

corr = importlib.import_module("21cma_abf_correlator_gb300")
frontend = importlib.import_module("21cma_abf_correlator_gb300.frontend")

N_FREQS = [512, 1024, 2048, 4096] + list(range(6144, 32769, 2048))
PATTERNS = ["prng", "counter"]
PACKET = 1024          # samples per packet of the packet mask
BLOCK_UNIT = 16        # granularity of a batch's block starts


def _engine(name, n, nf, frames, mode, acc64=False, loss="none", chunk=1024, tune=False):
    return {"name": name, "kind": "engine", "stations": n, "n_freq": nf, "frames": frames,
            "mode": mode, "acc64": acc64, "loss": loss, "chunk": chunk, "tune": tune}


def listed():
    return [
        # The smallest runs: the reference's golden case (4 stations, 2048 channels, 300 frames)
        # on the default X-engine, and the 8-input, 1024-channel, 256-frame workload on the split
        # form. Launches and latency count here.
        _engine("golden-4in-2048-plain", 4, 2048, 300, 0),
        _engine("small-8in-1024-split", 8, 1024, 256, 2),
        # 15 stations (the reference's second golden case's count) at a channel count that is not
        # a power of two, an odd number of frames, some of them missing.
        _engine("ragged-15in-12288-plain", 15, 12288, 301, 0, acc64=True, loss="frames"),
        # The 20-input, 8192-channel workload with frame loss, split form.
        _engine("loss-20in-8192-split", 20, 8192, 2048, 2, loss="frames"),
        # The precision workload, 24 inputs at 16384 channels in 1024-frame passes: the FP16 form
        # over two passes, the split form, and the reference's numerics.
        _engine("main-24in-16384-fp16", 24, 16384, 2048, 1, acc64=True, tune=True),
        _engine("main-24in-16384-split", 24, 16384, 1024, 2, acc64=True, tune=True),
        _engine("main-24in-16384-plain", 24, 16384, 1024, 0),
        # The 40-input stream, single packets lost.
        _engine("stream-40in-16384-split", 40, 16384, 1024, 2, acc64=True, loss="packets",
                tune=True),
        # The longest frames.
        _engine("wide-24in-32768-fp16", 24, 32768, 512, 1, acc64=True),
        # Integration blocks of uneven length from a pooled ring, one graph launch.
        {"name": "batch-24in-4096-fp16", "kind": "batch", "stations": 24, "n_freq": 4096,
         "blocks": 12, "pool": 2048, "mode": 1, "chunk": 512},
        # The synthetic front end: a 512-frame slot of 24 inputs, with loss.
        {"name": "frontend-24in-16384-prng", "kind": "frontend", "stations": 24,
         "n_freq": 16384, "frames": 512, "pattern": "prng"},
        # A row through the C ABI: four slots of 128 frames, the default X-engine.
        {"name": "abi-24in-16384-plain", "kind": "abi", "stations": 24, "n_freq": 16384,
         "slot_frames": 128, "slots": 4, "mode": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["engine", "batch", "frontend", "abi"], [14, 2, 3, 1])[0]
    if kind == "frontend":
        nf = rng.choice([f for f in N_FREQS if f >= 2048])
        n = _log_int(rng, 1, 64)
        most = 24 * 16384 * 512 // (n * nf)
        return {"kind": kind, "stations": n, "n_freq": nf,
                "frames": max(1, min(2048, _log_int(rng, max(1, most // 64), most))),
                "pattern": rng.choice(PATTERNS)}
    if kind == "abi":
        nf = rng.choice([2048, 4096, 8192, 10240, 16384])
        n = rng.randint(2, 32)
        most = max(16, min(256, 24 * 16384 * 128 // (n * nf)))
        return {"kind": kind, "stations": n, "n_freq": nf,
                "slot_frames": rng.randint(max(8, most // 2), most), "slots": rng.randint(2, 4),
                "mode": rng.choice([0, 0, 2])}
    if kind == "batch":
        nf = rng.choice([1024, 2048, 4096, 8192])
        n = rng.randint(4, 24)
        return {"kind": kind, "stations": n, "n_freq": nf, "blocks": rng.randint(4, 12),
                "pool": BLOCK_UNIT * rng.randint(16, 96), "mode": rng.choice([0, 1, 2]),
                "chunk": rng.choice([128, 256, 512])}
    mode = rng.choice([0, 1, 2])
    n = _log_int(rng, 2, 64)
    nf = rng.choice(N_FREQS)
    pairs = n * (n + 1) // 2
    # at most the listed cases' samples and multiply-accumulates
    most = min(24 * 16384 * 2048 // (n * nf),
               (300 * 16384 * 1024 if mode == 0 else 820 * 16384 * 1024) // (pairs * nf), 4096)
    frames = _log_int(rng, min(64, most), most)
    loss = rng.choice(["none", "none", "frames", "packets"])
    if loss == "packets" and nf > 16384:
        loss = "frames"
    return {"kind": kind, "stations": n, "n_freq": nf, "frames": frames, "mode": mode,
            "acc64": rng.random() < 0.5, "loss": loss, "chunk": 1024, "tune": False}


# -- inputs ---------------------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _samples(n, frames, nf, seed):
    """int8 [n, frames, 2*nf]: receiver noise of sigma 24 with a common signal (correlation 0.2)
    that reaches station i delayed by a number of samples of its own."""
    dev = _device()
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    total = frames * 2 * nf
    common = torch.randn(total + 64, generator=g, device=dev)
    out = torch.empty((n, total), dtype=torch.int8, device=dev)
    for i in range(n):
        x = torch.randn(total, generator=g, device=dev)
        d = (7 * i) % 64
        x.mul_(24.0 * math.sqrt(0.8)).add_(common[d:d + total], alpha=24.0 * math.sqrt(0.2))
        out[i] = x.round_().clamp_(-128, 127).to(torch.int8)
    return out.reshape(n, frames, 2 * nf)


def _present(n, frames, seed):
    """bool [n, frames]: about one frame in twenty missing."""
    r = np.random.default_rng(seed + 1)
    return r.random((n, frames)) >= 0.05


def _packets(n, frames, nf, seed):
    """int32 words [n, frames]: bit p set where 1024-sample packet p arrived (1 % lost)."""
    r = np.random.default_rng(seed + 2)
    kept = r.random((n, frames, 32)) >= 0.01
    kept[:, :, max(1, 2 * nf // PACKET):] = True
    words = (kept.astype(np.uint64) << np.arange(32, dtype=np.uint64)).sum(axis=2)
    return words.astype(np.uint32).view(np.int32)


def _blocks(case, seed):
    r = np.random.default_rng(seed + 3)
    pool = case["pool"]
    out = []
    for _ in range(case["blocks"]):
        length = int(r.integers(max(1, pool // 16), pool // 2 + 1))
        first = int(r.integers(0, (pool - length) // BLOCK_UNIT + 1)) * BLOCK_UNIT
        out.append((first, length))
    return out


def _spec(case, seed):
    return frontend.ReplaySpec(pattern=case["pattern"], seed=seed, drop_rate=0.01, delay_stride=3)


class _Batch:
    """A captured batch and what it works on, given back when dropped."""

    def __init__(self, case, seed):
        n, nf = case["stations"], case["n_freq"]
        self.x = _samples(n, case["pool"], nf, seed)
        mask = np.packbits(_present(n, case["pool"], seed), axis=1, bitorder="little")
        self.mask = torch.from_numpy(mask).cuda()
        blocks = _blocks(case, seed)
        first = (ctypes.c_int64 * len(blocks))(*[b[0] for b in blocks])
        frames = (ctypes.c_int32 * len(blocks))(*[b[1] for b in blocks])
        self.engine = corr.FxEngine(n, nf, max_frames=case["chunk"], xmode=case["mode"])
        self.rows = torch.zeros((len(blocks), n * (n + 1) // 2, nf), dtype=torch.complex64,
                                device="cuda")
        self.lib = corr.abi.load()
        handle = ctypes.c_void_p()
        corr.abi.check(self.lib.corrx_batch_create(
            self.engine.h, ctypes.c_void_p(self.x.data_ptr()), self.x.stride(0),
            self.x.stride(1), ctypes.c_void_p(self.mask.data_ptr()), self.mask.stride(0), first,
            frames, len(blocks), ctypes.c_void_p(self.rows.data_ptr()), None,
            ctypes.byref(handle)), "corrx_batch_create")
        self.handle = handle

    def launch(self):
        corr.abi.check(self.lib.corrx_batch_launch(
            self.handle, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)),
            "corrx_batch_launch")

    def __del__(self):
        try:
            torch.cuda.synchronize()
            self.lib.corrx_batch_destroy(self.handle)
            self.engine.close()
        except Exception:
            pass


def prepare(case, seed):
    kind = case["kind"]
    n, nf = case["stations"], case["n_freq"]
    s = {"case": case}
    if kind == "frontend":
        s["spec"] = _spec(case, seed)
        s["frame0"] = s["spec"].first_full_frame(nf)
        s["x"] = torch.zeros((n, case["frames"], 2 * nf), dtype=torch.int8, device="cuda")
        s["mask"] = torch.zeros((n, (case["frames"] + 7) // 8), dtype=torch.uint8, device="cuda")
    elif kind == "batch":
        s["batch"] = _Batch(case, seed)
    elif kind == "abi":
        fps, slots = case["slot_frames"], case["slots"]
        c = corr.Correlator.new(n, nf, fps, fps, slots, 1)
        if case["mode"]:
            c.set_xengine(case["mode"])
        x = _samples(n, fps * slots, nf, seed).reshape(n, slots, fps, 2 * nf)
        for g in range(n):
            view = c.staging(g)
            torch.from_numpy(view.samples).copy_(x[g])
        s["correlator"], s["sequence"] = c, 0
        s["masks"] = [c.staging(g).mask for g in range(n)]
        s["out"] = torch.empty(c.fetch_bytes() // 8, dtype=torch.complex64).pin_memory().numpy()
    else:
        s["x"] = _samples(n, case["frames"], nf, seed)
        s["mask"] = s["packets"] = None
        if case["loss"] == "frames":
            bits = np.packbits(_present(n, case["frames"], seed), axis=1, bitorder="little")
            s["mask"] = torch.from_numpy(bits).cuda()
        elif case["loss"] == "packets":
            s["packets"] = torch.from_numpy(_packets(n, case["frames"], nf, seed)).cuda()
        e = corr.FxEngine(n, nf, max_frames=min(case["chunk"], case["frames"]),
                          xmode=case["mode"])
        if case["acc64"]:
            e.set_accumulator(corr.abi.CORRX_ACC_FP64)
        if case["tune"]:
            e.autotune()
        s["engine"], s["acc"] = e, e.new_acc()
        s["row"] = torch.empty((e.n_baseline, nf), dtype=torch.complex64, device="cuda")
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "frontend":
        frontend.fill(s["spec"], case["n_freq"], s["frame0"], s["x"], s["mask"])
        return [s["x"], s["mask"]]
    if kind == "batch":
        s["batch"].launch()
        return s["batch"].rows
    if kind == "abi":
        c, slots, fps = s["correlator"], case["slots"], case["slot_frames"]
        for k in range(slots):
            seq = s["sequence"]
            if seq >= slots:
                c.row_slot_free(seq)   # the slot's previous frames have been read
            for mask in s["masks"]:
                mask[seq % slots] = 0xFF   # the receive side marks every frame as arrived
            c.row_accumulate(seq, fps)
            s["sequence"] = seq + 1
        c.row_end(slots * fps)
        return c.rows_fetch(s["out"])
    e, acc, frames = s["engine"], s["acc"], case["frames"]
    acc.zero_()
    e.accumulate(s["x"], frames, acc, mask=s["mask"], packets=s["packets"])
    if case["acc64"]:
        return e.dump(acc, frames, out=s["row"])
    e.scale(acc, frames)
    return acc


def work(case):
    n, nf = case["stations"], case["n_freq"]
    pairs = n * (n + 1) // 2
    fft = 2.5 * 2 * nf * math.log2(2 * nf)   # one real transform
    if case["kind"] == "frontend":
        total = n * case["frames"] * 2 * nf
        return {"bytes": total + n * case["frames"] / 8, "flops": 0}
    if case["kind"] == "batch":
        # the blocks' mean length; each reads its frames and writes its row
        frames = case["blocks"] * (case["pool"] // 16 + case["pool"] // 2) / 2
        rows = case["blocks"]
    elif case["kind"] == "abi":
        frames, rows = case["slots"] * case["slot_frames"], 1
    else:
        frames, rows = case["frames"], 1
    return {"bytes": n * frames * 2 * nf + rows * pairs * nf * 8,
            "flops": n * frames * fft + 8.0 * pairs * nf * frames}


# -- the same in 64 bits --------------------------------------------------------------------

def _row64(x, present=None, packets=None):
    """complex128 [pairs, n_freq]: mean over frames of Y_j conj(Y_k), j <= k."""
    n, frames, length = x.shape
    nf = length // 2
    acc = torch.zeros((nf, n, n), dtype=torch.complex128, device=x.device)
    step = max(1, int(2 ** 27 // (n * length)))
    for f0 in range(0, frames, step):
        y = x[:, f0:f0 + step].to(torch.float64)
        if present is not None:
            y = y * torch.from_numpy(present[:, f0:f0 + step]).to(x.device)[:, :, None]
        if packets is not None:
            words = torch.from_numpy(packets[:, f0:f0 + step].astype(np.int64)).to(x.device)
            at = torch.arange(max(1, length // PACKET), device=x.device)
            kept = ((words[:, :, None] >> at) & 1).to(torch.float64)
            kept = kept.repeat_interleave(min(PACKET, length), dim=2)
            y = y * kept[:, :, :length]
        spectra = torch.fft.rfft(y, dim=2)[:, :, :nf].permute(2, 0, 1).contiguous()
        acc += spectra @ spectra.conj().transpose(1, 2)
    j, k = np.triu_indices(n)
    j, k = (torch.from_numpy(v).to(x.device) for v in (j, k))
    return (acc[:, j, k].transpose(0, 1) / frames).contiguous()


def exact(case, seed):
    n, nf = case["stations"], case["n_freq"]
    if case["kind"] == "frontend":
        return None   # whole numbers
    if case["kind"] == "batch":
        x = _samples(n, case["pool"], nf, seed)
        present = _present(n, case["pool"], seed)
        return torch.stack([_row64(x[:, a:a + m], present[:, a:a + m])
                            for a, m in _blocks(case, seed)])
    if case["kind"] == "abi":
        return _row64(_samples(n, case["slots"] * case["slot_frames"], nf, seed))[None]
    present = _present(n, case["frames"], seed) if case["loss"] == "frames" else None
    packets = _packets(n, case["frames"], nf, seed) if case["loss"] == "packets" else None
    return _row64(_samples(n, case["frames"], nf, seed), present, packets)
