"""The decode and rotary calls whose speed is measured: what they are, how their inputs are made,
and what one pass of each does.

Every case goes through the package's public calls: the decode of a batch of CRF scores into
moves, sequence and quality string (three models: fast = 64 states, hac = 256, sup = 1024), in the
flavours a basecaller uses (results in buffers of its own, results in fresh buffers as the
reference's call returns them, scores with the blank column inside, the allocation-free call), and
the rotary embedding of the transformer encoder in front of the sup model's head.
"""
import math

import torch

import openfish_b200 as of

DEV = "cuda"

# A decode case: "call" is the entry point, "state_len" the model, T timesteps, N chunks; "p_step" the
# share of timesteps at which the planted path moves on (1.0 is the benchmark's, basecalled DNA moves
# on at about 0.4 of them); "beam_cut", "temperature", "q_scale" and "q_shift" the decoder's options.
# A rotary case: packed fp16 [B][S][3][H][D], Q and K heads rotated in place in one call, "half" pairs
# of every head rotated.


def _decode(name, call, state_len, T, N, p_step=1.0, beam_cut=100.0, temperature=1.0):
    q = of.MODEL_QSCORE[state_len]
    return {"name": name, "op": "decode", "call": call, "state_len": state_len, "T": T, "N": N, "p_step": p_step,
            "beam_cut": beam_cut, "temperature": temperature, "q_scale": q["q_scale"], "q_shift": q["q_shift"]}


def _rotary(name, B, S, H, D, half):
    return {"name": name, "op": "rotary", "B": B, "S": S, "H": H, "D": D, "half": half}


def listed():
    return [
        # one short read of the fast model, decoded as it arrives: nothing but latency
        _decode("fast_one_chunk", "decode_gpu", 3, 1000, 1, p_step=0.4),
        # the CPU-sized configuration of the benchmark's list: 16 chunks of the fast model
        _decode("fast_16", "decode_gpu", 3, 1000, 16),
        # a full batch of the fast model on one GPU
        _decode("fast_1024", "decode_into", 3, 1666, 1024),
        # the tail of a run: a handful of chunks of odd length left over
        _decode("hac_7_ragged", "decode_into", 4, 833, 7, p_step=0.4),
        # what fits the allocation-free call (48 MiB of scratch): a server's small batch
        _decode("hac_static_14", "decode_static", 4, 1666, 14),
        # the headline batch, through the call that hands out fresh result buffers
        _decode("hac_512", "decode_gpu", 4, 1666, 512),
        # a batch that is no multiple of anything, DNA-like stays, tighter pruning
        _decode("hac_601_ragged", "decode_into", 4, 1201, 601, p_step=0.4, beam_cut=20.0),
        # scores as a CRF head with a blank column emits them
        _decode("hac_300_blank_column", "decode_5wide", 4, 1666, 300, p_step=0.7),
        # the whole strong-scaling job of the benchmark on one GPU
        _decode("hac_4096", "decode_into", 4, 1666, 4096),
        # a full batch of the sup model
        _decode("sup_256", "decode_into", 5, 1666, 256),
        # a small batch of short sequences: the call overhead
        _rotary("rotary_small", 2, 64, 8, 64, 32),
        # the encoder's packed QKV tensor
        _rotary("rotary_encoder", 32, 1666, 8, 64, 32),
    ]


# no drawn case decodes more states than the largest listed one
_MOST_STATES = 4096 * 1666 * 256
_STATIC_BYTES = of.STATIC_SCRATCH_BYTES


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _static_most(state_len, T):
    """Largest N that the allocation-free call takes (include/openfish_b200.h states the sizes)."""
    ns = 4 ** state_len
    per_chunk = (3 if state_len == 3 else 2) * (T + 1) * ns * 4 + (T + 1) * 32 + T * 28
    return int((_STATIC_BYTES - 16384) // (per_chunk + 64))


def draw(rng):
    if rng.random() < 0.2:
        D = rng.choice([32, 48, 64, 80, 96, 128])
        case = _rotary("", _log_int(rng, 1, 32), _log_int(rng, 16, 1666), rng.choice([4, 5, 8, 12, 16]), D,
                       rng.choice([D // 4, D // 2]))
    else:
        state_len = rng.choice([3, 4, 4, 5])
        call = rng.choice(["decode_into", "decode_into", "decode_gpu", "decode_5wide", "decode_static"])
        T = _log_int(rng, 100, 2000)
        most = _MOST_STATES // (T * 4 ** state_len)
        most = min(most, 4096 if call != "decode_5wide" else 2048)
        if call == "decode_static":
            most = min(most, _static_most(state_len, T))
        N = _log_int(rng, 1, max(1, most))
        case = _decode("", call, state_len, T, N, p_step=round(rng.uniform(0.3, 1.0), 2),
                       beam_cut=rng.choice([100.0, 100.0, 20.0]), temperature=rng.choice([1.0, 1.0, 0.9]))
    del case["name"]
    return case


def _scores(case, seed):
    """fp16 scores [T][N][4*ns]: 5*tanh(1.5*z) with +4 on the transitions of a planted path, the
    distribution of openfish_b200/synth.py, made on the GPU."""
    T, N, sl = case["T"], case["N"], case["state_len"]
    ns = 4 ** sl
    g = torch.Generator(device=DEV).manual_seed(seed)
    steps = torch.rand((T, N), generator=g, device=DEV) < case["p_step"]
    bases = torch.randint(0, 4, (T, N), generator=g, device=DEV)
    # the bases of the planted read in order, the initial k-mer's first: the k-mer after timestep t is
    # the window of sl bases that starts at the number of steps taken so far
    read = torch.randint(0, 4, (T + sl, N), generator=g, device=DEV)
    taken = steps.long().cumsum(0)
    n_idx = torch.arange(N, device=DEV).expand(T, N)
    read[(taken + sl - 1)[steps], n_idx[steps]] = bases[steps]
    kmer = torch.zeros((T, N), dtype=torch.int64, device=DEV)
    for i in range(sl):
        kmer = kmer * 4 + read.gather(0, taken + i)
    # stepping from k-mer p to q uses column 4*q + (first base of p)
    column = kmer * 4 + read.gather(0, (taken - 1).clamp_(min=0))
    out = torch.empty((T, N, 4 * ns), dtype=torch.float16, device=DEV)
    rows = max(1, (1 << 26) // (N * 4 * ns))
    for t0 in range(0, T, rows):
        t1 = min(T, t0 + rows)
        z = torch.empty((t1 - t0, N, 4 * ns), device=DEV).normal_(generator=g)
        z.mul_(1.5).tanh_().mul_(5.0)
        z.scatter_add_(2, column[t0:t1, :, None], 4.0 * steps[t0:t1, :, None].float())
        out[t0:t1] = z
    return out


class _Decode:
    """What a program that decodes batches of one shape keeps: the scores, the device buffers, the
    options and its result buffers."""

    def __init__(self, case, seed):
        T, N, sl = case["T"], case["N"], case["state_len"]
        self.call, self.state_len, self.gb = case["call"], sl, None
        self.options = of.decoder_init(beam_cut=case["beam_cut"], temperature=case["temperature"],
                                       q_scale=case["q_scale"], q_shift=case["q_shift"])
        self.scores = _scores(case, seed)
        self.tensors = {}
        if self.call == "decode_static":
            self.results = [torch.empty((N, T), dtype=torch.uint8, device=DEV) for _ in range(3)]
            return
        if self.call == "decode_5wide":
            wide = torch.empty((T, N, 4 ** sl, 5), dtype=torch.float16, device=DEV)
            wide[..., 0] = 2.0
            wide[..., 1:] = self.scores.view(T, N, 4 ** sl, 4)
            self.scores = wide.view(T, N, 5 * 4 ** sl)
        self.gb = of.gpubuf_init(T, N, sl)
        if self.call != "decode_gpu":
            self.results = [torch.empty((N, T), dtype=torch.uint8).pin_memory() for _ in range(3)]
        # the tensors a decode leaves in the device buffers (views)
        for name in ("bwd_NTC", "post_NTC", "states", "qual_data", "total_probs"):
            self.tensors[name] = torch.as_tensor(_Field(self, name), device=DEV)

    def run(self):
        if self.call == "decode_gpu":
            out = of.decode_gpu(self.scores, self.state_len, options=self.options, gpubuf=self.gb)
        else:
            if self.call == "decode_static":
                status = of.decode_static(self.scores, self.state_len, *self.results, options=self.options)
                if status != 0:
                    raise RuntimeError("decode_static returned %d" % status)
            elif self.call == "decode_5wide":
                of.decode_5wide_into(self.scores, self.state_len, self.gb, *self.results, options=self.options, clamp=9.0)
            else:
                of.decode_into(self.scores, self.state_len, self.gb, *self.results, options=self.options)
            out = dict(zip(("moves", "sequence", "qstring"), self.results))
        out.update(self.tensors)
        return out


class _Buffers:
    """Gives a batch's device buffers back when neither the batch nor a view of them is used any more."""

    def __init__(self, gb):
        self.gb = gb

    def __del__(self):
        self.gb.free()


class _Field:
    """One tensor of the device buffers, as torch.as_tensor takes it; keeps the buffers alive."""

    def __init__(self, batch, name):
        if not hasattr(batch, "buffers"):
            batch.buffers = _Buffers(batch.gb)
        self.buffers = batch.buffers
        self.__cuda_array_interface__ = batch.gb.tensor(name).__cuda_array_interface__


class _Rotary:
    def __init__(self, case, seed):
        B, S, H, D, half = (case[k] for k in ("B", "S", "H", "D", "half"))
        g = torch.Generator(device=DEV).manual_seed(seed)
        self.x = torch.randn((B, S, 3, H, D), generator=g, device=DEV).half()
        angle = torch.arange(S, device=DEV)[:, None].double() * 10000.0 ** (-torch.arange(half, device=DEV).double() / half)
        self.sin, self.cos = torch.sin(angle).float(), torch.cos(angle).float()
        self.args = (B, S, 2 * H, D, half, S * 3 * H * D, 3 * H * D, D)

    def run(self):
        of.rotary_emb_gpu(self.x, self.sin, self.cos, *self.args)
        return self.x


def prepare(case, seed):
    return (_Rotary if case["op"] == "rotary" else _Decode)(case, seed)


def run(state):
    return state.run()


def work(case):
    """Bytes: every input read once, every output written once.  Operations of a decode: both scans
    (five additions, maximum, differences, exponentials, their sum, a logarithm and an addition a
    state and timestep), the posterior, and the beam's 160 candidates a timestep."""
    if case["op"] == "rotary":
        pairs = case["B"] * case["S"] * 2 * case["H"] * case["half"]
        return {"bytes": 2 * 2 * 2 * pairs + 2 * 4 * case["S"] * case["half"], "flops": 6 * pairs}
    T, N, ns = case["T"], case["N"], 4 ** case["state_len"]
    wide = 5 if case["call"] == "decode_5wide" else 4
    read = 2 * wide * ns * T * N
    results = 3 * T * N
    # the allocation-free call hands out the three results only
    tensors = 0 if case["call"] == "decode_static" else 2 * 4 * ns * (T + 1) * N + (16 + 4 + 8) * T * N
    return {"bytes": read + results + tensors, "flops": (2 * 26 + 5) * ns * T * N + 160 * 12 * T * N}


def tolerance(case):
    """A decode's scores, posteriors and qualities are 32-bit sums of exponentials; moves and sequence
    stay the same, a quality character is a rounded logarithm of such a sum and may fall on the other
    side of a tie.  Rotary: one rounding to fp16."""
    if case["op"] == "rotary":
        return {"rel": 5e-4, "max": 2e-3}
    return {"rel": 1e-5, "differ": 1e-3}
