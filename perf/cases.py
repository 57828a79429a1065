"""Timed cases of the codec: what its users call, over the sizes they call it with.

Each case goes through the Python binding (bpc_paco) on data already where such
a program keeps it: device tensors for the device calls, a pinned host buffer for
the host call.  Images are the seeded synthetic ones of bpc_synth (sinusoids,
blurred noise of amplitude `amp`, sharp rectangles; 5/3 DWT), with the committed
probability tables.

Fields of a case: `op`; X, Y, levels, passes (2 or 3), cb (codeblock side), `amp`
and `rects` of the image; `sched` (the work-ordered device calls).  Ops:

  encode   coefficients -> slot stream, device to device
  decode   slot stream -> coefficients
  codec    encode, then decode of what it wrote
  batch    `images` images of mixed size, levels, passes and codeblock size, encoded
           into one compact container and decoded from it
  dwt      8-bit samples (pixel - 128) -> int32 -> forward 5/3 DWT in place
  restore  slot stream -> coefficients -> inverse 5/3 DWT in place
  host     the host-buffer call, encode and decode in place in a pinned buffer
"""
import math
import os
import random
import sys

import torch

_PKG = os.path.join(os.getcwd(), "cuda_bpc-paco_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import bpc_paco  # noqa: E402
import bpc_synth  # noqa: E402

_LUTS = os.path.join(os.getcwd(), "tests", "golden", "luts")

# the largest image of a drawn case; the listed ones go to 16384 x 16384
_DRAW_MAX = 96 * 1024 * 1024


def listed():
    return [
        # a thumbnail or preview: 64 codeblocks, a fraction of the GPU; launch
        # latency and the serial time of one codeblock count
        {"name": "thumb_512", "op": "codec", "X": 512, "Y": 512, "levels": 5, "passes": 3, "cb": 64, "amp": 20.0,
         "rects": 30, "sched": False},
        # one photograph-sized image with the plain calls and 2 coding passes
        {"name": "encode_2048_2pass", "op": "encode", "X": 2048, "Y": 2048, "levels": 5, "passes": 2, "cb": 64,
         "amp": 20.0, "rects": 30, "sched": False},
        {"name": "decode_2048_2pass", "op": "decode", "X": 2048, "Y": 2048, "levels": 5, "passes": 2, "cb": 64,
         "amp": 20.0, "rects": 30, "sched": False},
        # one large image with 3 coding passes through the work-ordered calls:
        # the workload the benchmark reports
        {"name": "encode_4096_3pass", "op": "encode", "X": 4096, "Y": 4096, "levels": 5, "passes": 3, "cb": 64,
         "amp": 40.0, "rects": 60, "sched": True},
        {"name": "decode_4096_3pass", "op": "decode", "X": 4096, "Y": 4096, "levels": 5, "passes": 3, "cb": 64,
         "amp": 40.0, "rects": 60, "sched": True},
        # a scan or satellite tile of a quarter gigapixel, noisy: many waves
        {"name": "encode_16384_3pass", "op": "encode", "X": 16384, "Y": 16384, "levels": 5, "passes": 3, "cb": 64,
         "amp": 80.0, "rects": 400, "sched": True},
        {"name": "decode_16384_3pass", "op": "decode", "X": 16384, "Y": 16384, "levels": 5, "passes": 3, "cb": 64,
         "amp": 80.0, "rects": 400, "sched": True},
        # small codeblocks and a ragged size (95 x 55 codeblocks, an odd count)
        {"name": "codec_3040x1760_cb32", "op": "codec", "X": 3040, "Y": 1760, "levels": 4, "passes": 2, "cb": 32,
         "amp": 30.0, "rects": 40, "sched": False},
        # a folder of pictures coded in one call, autotuning left out
        {"name": "batch_24_mixed", "op": "batch", "images": 24, "mix": 3, "amp": 30.0, "rects": 40},
        # the transform before an encode and after a decode
        {"name": "dwt_8192x6144", "op": "dwt", "X": 8192, "Y": 6144, "levels": 5, "amp": 30.0, "rects": 100},
        {"name": "restore_3072x2048", "op": "restore", "X": 3072, "Y": 2048, "levels": 5, "passes": 3, "cb": 64,
         "amp": 30.0, "rects": 40, "sched": True},
        # the drop-in user, whose image lives in host memory
        {"name": "host_2048_2pass", "op": "host", "X": 2048, "Y": 2048, "levels": 5, "passes": 2, "cb": 64,
         "amp": 20.0, "rects": 30},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    op = rng.choice(["encode", "encode", "decode", "decode", "codec", "batch", "dwt", "restore", "host"])
    case = {"op": op, "amp": round(_log_uniform(rng, 8.0, 80.0), 1), "rects": rng.randint(20, 400)}
    if op == "batch":
        case.update(images=rng.randint(4, 32), mix=rng.randint(0, 1 << 20))
        return case
    cb = 64 if rng.random() < 0.7 else 32
    top = {"host": 4096 * 4096, "dwt": _DRAW_MAX, "restore": 8192 * 8192}.get(op, _DRAW_MAX)
    area = _log_uniform(rng, 256 * 256, top)
    aspect = _log_uniform(rng, 0.5, 2.0)

    def side(v):
        return max(2, min(16384 // cb, round(v / cb))) * cb

    X, Y = side(math.sqrt(area * aspect)), side(math.sqrt(area / aspect))
    case.update(X=X, Y=Y, levels=rng.randint(3, 5))
    if op != "dwt":
        case.update(passes=rng.choice([2, 3]), cb=cb)
    if op in ("encode", "decode", "codec", "restore"):
        case["sched"] = rng.random() < 0.6
    return case


def _pixels(case, seed, X=None, Y=None, amp=None):
    """Y x X int32 pixels 0..255: the top-left part of a square synthetic image."""
    X, Y = X or case["X"], Y or case["Y"]
    img = bpc_synth.make_image_gpu(max(X, Y), seed, amp or case["amp"], case["rects"])
    return img if X == Y else img[:Y, :X].contiguous()


def _coefficients(case, seed, levels=None, X=None, Y=None):
    img = _pixels(case, seed, X, Y) - 128
    bpc_paco.dwt53(img, case["levels"] if levels is None else levels)
    return img


def _lut_dir(passes):
    return os.path.join(_LUTS, f"{passes}_coding_pass")


def _mixed(case):
    """The batch's images: (X, Y, levels, passes, cb)."""
    r = random.Random(case["mix"])
    out = []
    for _ in range(case["images"]):
        cb = 64 if r.random() < 0.7 else 32
        X, Y = (round(_log_uniform(r, 512, 4096) / 64) * 64 for _ in range(2))
        out.append((X, Y, r.randint(3, 5), r.choice([2, 3]), cb))
    return out


def prepare(case, seed):
    op = case["op"]
    s = {"op": op, "case": case}
    if op == "batch":
        specs = _mixed(case)
        s["in"] = [_coefficients(case, seed * 1000 + k, lv, X, Y) for k, (X, Y, lv, _, _) in enumerate(specs)]
        s["batch"] = bpc_paco.Batch(specs, {2: _lut_dir(2), 3: _lut_dir(3)})
        s["compact"] = torch.zeros(s["batch"].words, dtype=torch.int32, device="cuda")
        s["offsets"] = torch.zeros(s["batch"].codeblocks + 1, dtype=torch.int64, device="cuda")
        s["out"] = [torch.empty_like(t) for t in s["in"]]
        s["status"] = torch.zeros(1, dtype=torch.int32, device="cuda")
        return s
    X, Y, levels = case["X"], case["Y"], case["levels"]
    if op == "dwt":
        s["samples"] = (_pixels(case, seed) - 128).to(torch.int8)
        s["out"] = torch.empty((Y, X), dtype=torch.int32, device="cuda")
        s["tmp"] = torch.empty_like(s["out"])
        return s
    s["lut"] = bpc_paco.DeviceLut(_lut_dir(case["passes"]), case["passes"], levels)
    coeffs = _coefficients(case, seed)
    if op == "host":
        s["buf"] = torch.empty((Y, X), dtype=torch.int32, pin_memory=True)
        s["buf"].copy_(coeffs)
        return s
    s["status"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    s["sched"] = bpc_paco.sched_buffer(X, Y, case["cb"]) if case["sched"] else None
    s["stream"] = torch.empty(X * Y, dtype=torch.int32, device="cuda")
    if op in ("encode", "codec"):
        s["coeffs"] = coeffs
    else:
        bpc_paco.encode_device(coeffs, s["stream"], s["lut"], case["cb"])
    if op != "encode":
        s["out"] = torch.empty((Y, X), dtype=torch.int32, device="cuda")
    if op == "restore":
        s["tmp"] = torch.empty_like(s["out"])
    return s


def run(s):
    op, case = s["op"], s["case"]
    if op == "batch":
        s["batch"].encode(s["in"], s["compact"], s["offsets"], s["status"])
        s["batch"].decode(s["compact"], s["offsets"], s["out"], s["status"])
        return {"compact": s["compact"], "offsets": s["offsets"], "out": s["out"], "status": s["status"]}
    if op == "dwt":
        s["out"].copy_(s["samples"])
        bpc_paco.dwt53(s["out"], case["levels"], tmp=s["tmp"])
        return s["out"]
    lut, cb = s["lut"], case["cb"]
    if op == "host":
        L, buf = bpc_paco.lib(), s["buf"]
        a = (buf.data_ptr(), case["X"], case["Y"], lut.ptr, lut.n, lut.passes, lut.levels, cb)
        st_enc = L.bpc_code_host(bpc_paco.CODE, *a)
        st_dec = L.bpc_code_host(bpc_paco.DECODE, *a)
        return {"coeffs": buf, "status": [st_enc, st_dec]}
    got = {"status": s["status"]}
    if op in ("encode", "codec"):
        bpc_paco.encode_device(s["coeffs"], s["stream"], lut, cb, status=s["status"], sched=s["sched"])
        got["stream"] = s["stream"]
    if op != "encode":
        bpc_paco.decode_device(s["stream"], s["out"], lut, cb, status=s["status"], sched=s["sched"])
        got["out"] = s["out"]
    if op == "restore":
        bpc_paco.dwt53(s["out"], case["levels"], inverse=True, tmp=s["tmp"])
    return got


def work(case):
    """Bytes read and written once; there is no floating-point work."""
    op = case["op"]
    if op == "batch":
        n = sum(X * Y for (X, Y, _, _, _) in _mixed(case))
        # coefficients in, container out (about a sixth of them), and back
        return {"bytes": 2 * (4 + 4 / 6) * n, "flops": 0}
    n = case["X"] * case["Y"]
    per = {"encode": 8, "decode": 8, "codec": 16, "dwt": 5, "restore": 8, "host": 16}[op]
    return {"bytes": per * n, "flops": 0}
