"""What a user of this library has it do, as cases to be measured: whole sampling runs of the diffusion
sampler through its operator entry points (cck_mk_sample, and cck_mk_sample_static for a caller without a
workspace), on device buffers that the caller owns, as the JAX side or a C caller binds them.

A case says how many tokens and samples a run has, how many sampling steps, which variant bits, and
the shape bucket that its buffers are laid out for (0: the fold's own extents). The weights are those
of one 24-block model; trunk outputs, geometry and weights are drawn with the distributions of
mkharness.synth (unit normal trunk outputs, a 3.8 A chain with 5 to 14 atoms a token, LeCun-normal
weights, Karras noise levels), here directly on the GPU.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

for _path in (os.path.abspath("colabfold-cuda-kernels_b200"),):
    if _path not in sys.path:
        sys.path.insert(0, _path)
import colabfold_cuda_kernels as cck  # noqa: E402
from mkharness import synth  # noqa: E402

BLOCKS, CS, PLC = 24, 384, 128
HEUN, REALIGN, SCFINAL, ATOB = synth.F_HEUN, synth.F_REALIGN, synth.F_SCFINAL, synth.F_ATOB
PARALLEL_QKNORM = synth.F_PARALLEL | synth.F_QKNORM
VARIANTS = (0, 0, 0, 0, HEUN, REALIGN, PARALLEL_QKNORM, SCFINAL | ATOB)


def _case(tokens, samples, steps, flags=0, bucket=0, static=False):
    return {"tokens": tokens, "samples": samples, "steps": steps, "flags": flags, "bucket": bucket, "static": static}


def listed():
    return [
        # the smallest call: one sample of a short peptide in few steps, without a workspace (from inside a graph capture)
        dict(_case(32, 1, 20, static=True), name="32x1x20 static"),
        # a small fold in the bucket above it: latency of the schedule, ragged extents told by ext
        dict(_case(61, 5, 200, bucket=64), name="61(64)x5x200"),
        # a domain, five samples a seed, the usual 200 steps
        dict(_case(256, 5, 200), name="256x5x200"),
        # one sample: a quick look, or one seed of many
        dict(_case(512, 1, 200), name="512x1x200"),
        # the headline configuration
        dict(_case(512, 5, 200), name="512x5x200"),
        # an ordinary chain in its bucket: extents that are multiples of nothing
        dict(_case(391, 5, 200, bucket=512), name="391(512)x5x200"),
        # a complex
        dict(_case(1024, 5, 200), name="1024x5x200"),
        # the largest extent, where the pair logits are the largest stream
        dict(_case(2048, 1, 200), name="2048x1x200"),
        # variants: two denoiser calls a step; another block structure with normalised q and k; the realigned step
        dict(_case(256, 1, 100, flags=HEUN), name="256x1x100 heun"),
        dict(_case(384, 1, 100, flags=PARALLEL_QKNORM), name="384x1x100 parallel qknorm"),
        dict(_case(320, 5, 50, flags=REALIGN), name="320x5x50 realign"),
    ]


def draw(rng):
    """Tokens over the logarithm of 24..2048, most often in a bucket of a multiple of 64; 1 to 8 samples,
    10 to 200 steps; no more work than the largest listed case."""
    most = max(work(c)["flops"] for c in listed())
    while True:
        tokens = int(round(math.exp(rng.uniform(math.log(24), math.log(2048)))))
        samples = rng.choice((1, 1, 2, 3, 5, 5, 5, 8))
        steps = int(round(math.exp(rng.uniform(math.log(10), math.log(200)))))
        bucket = (tokens + 63) // 64 * 64 if rng.random() < 0.6 else 0
        c = _case(tokens, samples, steps, flags=rng.choice(VARIANTS), bucket=bucket if bucket != tokens else 0)
        if work(c)["flops"] <= 0.8 * most and tokens * samples <= 5120:
            return c


def _extents(case):
    """(tokens, subsets) of the fold and of its bucket: 8 atoms a token on average, the last subset partly filled."""
    n, nb = case["tokens"], case["bucket"] or case["tokens"]
    return n, (8 * n + 31) // 32, nb, (8 * nb + 31) // 32


def _calls(case):
    return 2 if case["flags"] & HEUN and not case["flags"] & REALIGN else 1


def work(case):
    n, ns, nb, nsb = _extents(case)
    flags = case["flags"]
    tw1, aw1 = (4608, 768) if flags & ATOB else (3072, 512)
    per_eval = synth.flops_per_eval(n, 8 * n, case["samples"], nb=BLOCKS, cs=CS, tw1=tw1, aw1=aw1)
    flops = case["samples"] * case["steps"] * _calls(case) * per_eval + 2 * n * n * PLC * 16 * BLOCKS
    weights = 2 * BLOCKS * (768 * (3072 + 768 + tw1 + 1536) + 6 * 768 * CS) + 2 * 2 * (4 + 2) * CS * CS + 2 * 768 * CS
    weights += 2 * 6 * 128 * (512 + 128 + aw1 + 256) + 2 * 2 * 768 * 128
    pair = n * n * (2 * PLC + 8)
    atoms = 8 * n * 4 * (128 + 6 * 8 * 128) + 6 * ns * 4 * 32 * 128 * 4 + ns * 128 * 8
    out = case["samples"] * nb * 24 * 3 * 4
    return {"bytes": weights + pair + atoms + n * CS * 4 + out, "flops": flops}


def tolerance(case):
    # f32 coordinates at the end of up to 200 evaluations of a bf16 network, each of which other roundings
    # of the same precision move by a few 1e-3
    return {"rel": 1e-2}


def _inputs(case, seed):
    """The operator's 74 inputs on the GPU, laid out for the bucket: zeros, masks 0 and index -1 in the padding."""
    n, ns, nb, nsb = _extents(case)
    flags, dev = case["flags"], "cuda"
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    rng = np.random.default_rng(seed)
    atoms, slots_b, rows_b = 8 * n, nb * synth.SLOTS, nsb * synth.SUBSET
    x = {}

    def normal(*shape, std=1.0, mean=0.0, dtype=torch.float32):
        a = torch.randn(shape, generator=g, device=dev)
        return a.mul_(std).add_(mean).to(dtype)

    def lecun(*shape):
        return normal(*shape, std=shape[-1] ** -0.5, dtype=torch.bfloat16)

    def padded(a, rows, fill=0.0, dim=0):
        shape = list(a.shape)
        shape[dim] = rows
        b = torch.full(shape, fill, dtype=a.dtype, device=dev)
        b.narrow(dim, 0, a.shape[dim]).copy_(a)
        return b

    # geometry and index maps
    count = synth.atoms_per_token(n, rng, False)
    token = np.repeat(np.arange(n), count)
    slot = (token * synth.SLOTS + np.arange(atoms) - np.repeat(np.cumsum(count) - count, count)).astype(np.int32)
    tok2q = np.full(rows_b, -1, dtype=np.int32)
    tok2q[:atoms] = slot
    q2ta = np.full(slots_b, -1, dtype=np.int32)
    q2ta[slot] = np.arange(atoms, dtype=np.int32)
    q2k = (np.arange(nsb)[:, None] * synth.SUBSET - 48 + np.arange(synth.NK)[None, :]).astype(np.int32)
    q2k[(q2k < 0) | (q2k >= atoms)] = -1
    q2k[ns:] = -1
    x["TOK2Q"], x["Q2TA"], x["Q2K"] = (torch.from_numpy(a).to(dev) for a in (tok2q, q2ta, q2k))
    x["QMASK"] = (torch.arange(rows_b, device=dev) < atoms).float()
    x["KMASK"] = (x["Q2K"] >= 0).float()
    x["ATOM_MASK"] = (x["Q2TA"] >= 0).float()
    x["TAM"] = x["ATOM_MASK"].clone()
    x["TMASK"] = (torch.arange(nb, device=dev) < n).float()
    way = normal(n, 3)
    way /= way.norm(dim=1, keepdim=True)
    ref = torch.cumsum(3.8 * way, 0)[torch.from_numpy(token).to(dev)] + normal(atoms, 3, std=1.5)

    # schedule and conditioning
    x["SIGMA"] = torch.from_numpy(synth.karras_sigmas(case["steps"])).to(dev)
    x["MISC"] = torch.tensor([0.8, 1.0, 1.003, 1.5, float(flags), 0.4], device=dev)
    x["SC_BASE"] = padded(normal(n, CS), nb)
    x["FOURIER_W"], x["FOURIER_B"] = normal(256), torch.rand(256, generator=g, device=dev)
    x["NOISE_LN"], x["NOISE_LNO"], x["WN"] = normal(256, std=0.1, mean=1.0), normal(256, std=0.1), normal(256, CS, std=1 / 16)
    for i in range(2):
        x["ST%d_S" % i], x["ST%d_O" % i] = normal(CS, std=0.1, mean=1.0), normal(CS, std=0.1)
        x["ST%d_W1" % i], x["ST%d_W2" % i] = lecun(4 * CS, CS), lecun(CS, 2 * CS)
    x["WM1"], x["BM1"] = lecun(BLOCKS * 4 * 768, CS), normal(BLOCKS * 4 * 768, std=0.1)
    x["WM2"], x["BM2"] = lecun(BLOCKS * 2 * 768, CS), normal(BLOCKS * 2 * 768, std=0.1, mean=-2.0)
    x["WSE"], x["SE_B"] = lecun(768, CS), normal(768, std=0.1)
    x["SCF"] = torch.cat([normal(CS, std=0.2, mean=1.0), normal(CS, std=0.2)])

    # token transformer and pair representation (with the row statistics of its folded LayerNorm)
    x["WQKVG"], x["BQ"], x["WO"] = lecun(BLOCKS, 3072, 768), normal(BLOCKS, 768, std=0.1), lecun(BLOCKS, 768, 768)
    x["W1"], x["W2"] = lecun(BLOCKS, (3 if flags & ATOB else 2) * 1536, 768), lecun(BLOCKS, 768, 1536)
    x["WTB"], x["TB_B"], x["WAGGR"] = lecun(128, 768), normal(128, std=0.1), lecun(768, 128)
    x["PC"] = torch.zeros(nb, nb, PLC, dtype=torch.bfloat16, device=dev)
    x["PCS"] = torch.zeros(nb, nb, 2, device=dev)
    for r in range(0, n, 256):
        z = normal(min(256, n - r), n, PLC, dtype=torch.bfloat16)
        x["PC"][r:r + 256][:z.shape[0], :n] = z
        var, mean = torch.var_mean(z.float(), -1, correction=0)
        x["PCS"][r:r + 256][:z.shape[0], :n] = torch.stack([mean, (var + 1e-5).rsqrt()], -1)
    x["PLW"] = lecun(BLOCKS, 16, PLC)
    x["PLWS"], x["PLB"] = x["PLW"].float().sum(-1).reshape(-1), normal(BLOCKS * 16, std=0.1)
    x["PLX"] = torch.zeros(2, dtype=torch.bfloat16, device=dev)  # absent

    # atom path
    x["WPOS"] = normal(3, 128, std=3 ** -0.5)
    feat = torch.cat([ref / 10.0, normal(atoms, 13)], 1)
    x["SCQ"] = padded(feat @ normal(16, 128, std=0.25), rows_b)
    x["WUPD"], x["UPD_B"] = normal(3, 128, std=128 ** -0.5), normal(3, std=0.1)
    keys = x["Q2K"][:ns].long()
    where = padded(ref, 32 * ns)
    dist2 = ((where.view(ns, 32, 1, 3) - where[keys.clamp(min=0)].view(ns, 1, synth.NK, 3)) ** 2).sum(-1)
    near = 1.0 / (1.0 + dist2 / 16.0)
    no_key = (keys < 0)[:, None, None, :]
    for side in ("ENC", "DEC"):
        lin = torch.einsum("af,bsfc->basc", feat, normal(3, 8, 16, 128, std=0.25))
        for s, shift in ((0, 0.0), (2, 0.0), (4, 0.0), (6, 2.0), (7, 2.0)):  # scales, and the gates after their sigmoid
            lin[:, :, s] = torch.sigmoid(lin[:, :, s] - shift)
        x[side + "_AMODS"] = padded(lin, rows_b, dim=1)
        head = normal(3, 4)
        apl = torch.zeros(3, nsb, 4, 2, 8, 256, device=dev)
        for b in range(3):
            v = head[b].view(1, 4, 1, 1) * near[:, None] + normal(ns, 4, 32, synth.NK, std=0.5)
            v = v.masked_fill(no_key, -1e9)
            # tiles of 16 x 16 in the order the atom attention reads: [lane = (row % 8, column pair)][column half, row half, column]
            v = v.view(ns, 4, 2, 2, 8, 8, 2, 4, 2).permute(0, 1, 2, 5, 4, 7, 6, 3, 8)
            apl[b, :ns] = v.reshape(ns, 4, 2, 8, 256)
        x[side + "_APL"] = apl
        x[side + "_WQG"], x[side + "_BQ"], x[side + "_WKV"] = lecun(3, 256, 128), normal(3, 128, std=0.1), lecun(3, 256, 128)
        x[side + "_WO"], x[side + "_W1"], x[side + "_W2"] = lecun(3, 128, 128), lecun(3, 768 if flags & ATOB else 512, 128), lecun(3, 128, 256)

    # what only variants read
    def qk_norm(blocks, width):
        t = normal(blocks, 4, width, std=0.2)
        t[:, 0::2] += 1.0
        return t

    x["TQKN"], x["EQKN"], x["DQKN"] = qk_norm(BLOCKS, 768), qk_norm(3, 128), qk_norm(3, 128)
    x["ROPE"] = torch.zeros(rows_b, 32, device=dev)
    x["CHIR_W"], x["CHIR_A"] = torch.zeros(3, 128, device=dev), torch.zeros(1, device=dev)
    x["CHIR_C"] = torch.zeros(1, 4, dtype=torch.int32, device=dev)
    x["CHIR_PTR"] = torch.zeros(slots_b + 1, dtype=torch.int32, device=dev)
    x["CHIR_IDX"] = torch.zeros(1, dtype=torch.int32, device=dev)
    return [x[name].contiguous() for name in synth.IN_NAMES]


_LIB = None


def _library():
    global _LIB
    if _LIB is None:
        lib = ctypes.CDLL(cck.library_path("diffusion", 100))
        p, i, z = ctypes.c_void_p, ctypes.c_int, ctypes.c_size_t
        lib.cck_mk_sample.argtypes = [p, p, p, p, i, p, i, p, z, i, i, i]
        lib.cck_mk_sample_static.argtypes = [p, p, p, p, i, p, i, i, i, i]
        lib.mk_workspace_bytes.argtypes = [i] * 5 + [p]
        lib.mk_workspace_bytes.restype = z
        lib.cck_last_error.restype = ctypes.c_char_p
        _LIB = lib
    return _LIB


def prepare(case, seed):
    lib = _library()
    n, ns, nb, nsb = _extents(case)
    inputs = _inputs(case, seed)
    ptrs = (ctypes.c_void_p * 74)(*[t.data_ptr() for t in inputs])
    sizes = (ctypes.c_size_t * 74)(*[t.numel() * t.element_size() for t in inputs])
    s = {"lib": lib, "inputs": inputs, "ptrs": ptrs, "sizes": sizes, "tokens": nb}
    s["call"] = (case["samples"], case["steps"], case["flags"])
    s["ext"] = torch.tensor([n, ns, 1, seed & 0x7FFFFFFF, 0], dtype=torch.int32, device="cuda")
    s["out"] = torch.zeros(case["samples"], nb, 24, 3, device="cuda")
    s["ws"] = None
    if not case["static"]:
        need = lib.mk_workspace_bytes(case["samples"], nb, nsb, case["steps"], case["flags"], sizes)
        if need == 0:
            raise RuntimeError(lib.cck_last_error().decode())
        s["ws"] = torch.empty(need, dtype=torch.uint8, device="cuda")
    return s


def run(s):
    """One sampling run: every step of every sample, enqueued on the current stream."""
    stream = torch.cuda.current_stream().cuda_stream
    args = (stream, s["ext"].data_ptr(), s["ptrs"], s["sizes"], 74, s["out"].data_ptr(), s["tokens"])
    if s["ws"] is None:
        rc = s["lib"].cck_mk_sample_static(*args, *s["call"])
    else:
        rc = s["lib"].cck_mk_sample(*args, s["ws"].data_ptr(), s["ws"].numel(), *s["call"])
    if rc:
        raise RuntimeError(s["lib"].cck_last_error().decode())
    return s["out"]
