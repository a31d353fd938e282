"""The work that programs have this library do, as cases to be timed.

Each case is one call chain of a program that uses the library: decoding
batches of frame-path pictures (records and levels in, filtered planes out),
P pictures of the multi-tool stream, coding-tree pictures of the general
decoder, the frame encoder, and the function-level stages an encoder or
another decoder calls (motion compensation, transforms, the CTU search and
the CNN that prunes it). Inputs are value-noise content coded by the
library's own encoder, or records of the distributions in synth.py.
"""
import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

HERE = os.path.dirname(os.path.abspath(__file__))


def _pkg():
    """The package directory's name has a hyphen: it is imported by path."""
    if "rustmpeg_next_b200" not in sys.modules:
        d = os.path.join(os.path.dirname(HERE), "rustmpeg-next_b200")
        spec = importlib.util.spec_from_file_location("rustmpeg_next_b200", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["rustmpeg_next_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["rustmpeg_next_b200"]


pkg = _pkg()
from rustmpeg_next_b200 import cnn, synth  # noqa: E402

QPS = (22, 27, 32, 37)  # the quantisers of the full-frame configuration
_STREAM = None


def _stream():
    """The program's one CUDA stream; every context's kernels run on it."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


# ------------------------------------------------------------------- cases --

def listed():
    return [
        # a live decoder's smallest call: one 416x240 8-bit picture, host buffers in and out
        dict(name="decode_240p8_host", kind="decode", w=416, h=240, bd=8, cf=1, ctu_log2=5, n=1, sparse=True, io="host"),
        # the lowest latency at the ordinary size: one 1080p 10-bit picture, planes stay on the device
        dict(name="decode_1080p10", kind="decode", w=1920, h=1080, bd=10, cf=1, ctu_log2=5, n=1, sparse=True, io="device"),
        # bulk decoding: the full-frame configuration's batch of 128 pictures
        dict(name="decode_1080p10_x128", kind="decode", w=1920, h=1080, bd=10, cf=1, ctu_log2=5, n=128, sparse=True,
             io="device"),
        # studio material: 12-bit 4:4:4, 64x64 CTUs, a width that is no multiple of them, dense levels
        dict(name="decode_480p12_444_x6", kind="decode", w=854, h=480, bd=12, cf=3, ctu_log2=6, n=6, sparse=False,
             io="device"),
        # many streams of the multi-tool coder: 8 x (reference, P, P, P) at 1080p
        dict(name="p_1080p_x24", kind="p", w=1920, h=1088, streams=8, chain=3, sparse=True, deblock=True),
        # the frame encoder on four 1080p 10-bit frames from host memory
        dict(name="encode_1080p10_x4", kind="encode", w=1920, h=1080, bd=10, cf=1, n=4),
        # coding-tree pictures (4x4..64x64 blocks) of the general decoder, host buffers in and out
        dict(name="general_240p10_x4", kind="general", w=416, h=240, bd=10, ctu=64, n=4),
        # bi-prediction of every block of a 1080p 10-bit 4:2:0 picture
        dict(name="mc_1080p10_bi", kind="mc", w=1920, h=1080, bd=10, bi=True),
        # an encoder's transform round trip: residual -> levels -> residual of 16,000 mixed units
        dict(name="tu_16k", kind="tu", n=16000, seed_shape=1),
        # the pruner's inference on one 1080p frame
        dict(name="cnn_forward_1980", kind="cnn_forward", n=1980, bd=10, qp=32),
        # one training step of the pruner
        dict(name="cnn_train_1024", kind="cnn_train", n=1024, bd=10, qp=27, soft=True),
        # the encoder's full candidate search on one 1080p frame
        dict(name="search_1980", kind="search", n=1980, bd=10, qp=32, pruned=False),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "p", "encode", "general", "mc", "tu", "cnn_forward", "cnn_train",
                       "search"])
    if kind == "decode":
        io = rng.choice(["device", "device", "host"])
        w, h = _log(rng, 64, 1920) & ~1, _log(rng, 64, 1080) & ~1
        n = max(1, min(128 if io == "device" else 8, _log(rng, 1, 128), int(128 * 1920 * 1080 // (w * h))))
        return dict(kind=kind, w=w, h=h, bd=rng.choice([8, 10, 10, 12]), cf=rng.choice([1, 1, 1, 2, 3, 0]),
                    ctu_log2=rng.choice([5, 5, 6, 7]), n=n, sparse=rng.random() < 0.7, io=io)
    if kind == "p":
        return dict(kind=kind, w=32 * rng.randint(2, 60), h=32 * rng.randint(2, 34), streams=rng.randint(1, 8),
                    chain=rng.randint(1, 3), sparse=rng.random() < 0.7, deblock=rng.random() < 0.5)
    if kind == "encode":
        return dict(kind=kind, w=_log(rng, 64, 1920) & ~1, h=_log(rng, 64, 1080) & ~1, bd=rng.choice([8, 10, 12]),
                    cf=rng.choice([1, 1, 3]), n=rng.randint(1, 4))
    if kind == "general":
        return dict(kind=kind, w=8 * rng.randint(8, 52), h=8 * rng.randint(8, 30), bd=rng.choice([8, 10]),
                    ctu=rng.choice([32, 64, 128]), n=rng.randint(1, 4))
    if kind == "mc":
        return dict(kind=kind, w=_log(rng, 64, 1920) & ~1, h=_log(rng, 64, 1080) & ~1, bd=rng.choice([8, 10, 12]),
                    bi=rng.random() < 0.6)
    if kind == "tu":
        return dict(kind=kind, n=_log(rng, 50, 16000), seed_shape=rng.randint(2, 1 << 20))
    n = _log(rng, 16, 1980)
    if kind == "cnn_forward":
        return dict(kind=kind, n=n, bd=rng.choice([8, 10]), qp=rng.randint(22, 37))
    if kind == "cnn_train":
        return dict(kind=kind, n=min(n, 1024), bd=rng.choice([8, 10]), qp=rng.randint(22, 37), soft=rng.random() < 0.5)
    return dict(kind=kind, n=n, bd=rng.choice([8, 10]), qp=rng.randint(22, 37), pruned=rng.random() < 0.5)


# ------------------------------------------------------------------ inputs --

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _noise_plane(g, w, h, lo, hi):
    """Four octaves of value noise and some finely textured rectangles, as int16 CUDA samples in lo..hi."""
    acc = torch.zeros((1, 1, h, w), device="cuda")
    for o, gain in enumerate((1.0, 0.5, 0.25, 0.125)):
        cell = 128 >> o
        lat = torch.rand((1, 1, h // cell + 3, w // cell + 3), generator=g, device="cuda")
        acc += gain * torch.nn.functional.interpolate(lat, size=(h + cell, w + cell), mode="bicubic")[..., :h, :w]
    acc /= 1.875
    for k in range(8):
        s = min(64, w, h)
        lat = torch.rand((1, 1, s // 4 + 2, s // 4 + 2), generator=g, device="cuda")
        at = torch.rand(2, generator=g, device="cuda").tolist()
        y, x = int(at[0] * (h - s)), int(at[1] * (w - s))
        acc[..., y:y + s, x:x + s] = torch.nn.functional.interpolate(lat, size=(s, s), mode="bicubic")
    return (lo + acc[0, 0].clamp(0, 1) * (hi - lo)).round().to(torch.int16)


def _frame(g, w, h, cw, ch, bd, cf):
    """Coded-size (cw x ch) planes of one w x h frame, edges repeated below and right of the visible part."""
    mx = (1 << bd) - 1
    out = []
    for c in range(3 if cf else 1):
        sx, sy = (2 if c and cf in (1, 2) else 1), (2 if c and cf == 1 else 1)
        p = _noise_plane(g, (w + sx - 1) // sx, (h + sy - 1) // sy, 0 if c == 0 else int(mx * 0.375),
                         mx if c == 0 else int(mx * 0.625))
        pw, ph = cw // sx, ch // sy
        p = torch.nn.functional.pad(p[None, None].float(), (0, pw - p.shape[1], 0, ph - p.shape[0]), mode="replicate")
        out.append(p[0, 0].to(torch.int16).contiguous())
    return out + [None] * (3 - len(out))


def _encoder_pics(w, h, bd, cf, ctu_log2, qps):
    ctu = 1 << ctu_log2
    pics = np.zeros(len(qps), pkg.PIC_DTYPE)
    pics["width"], pics["height"] = -(-w // ctu) * ctu, -(-h // ctu) * ctu
    pics["visible_width"], pics["visible_height"] = w, h
    pics["bit_depth"], pics["chroma_format"], pics["ctu_log2"] = bd, cf, ctu_log2
    pics["slice_qp"] = qps
    pics["chroma_qp_scaled"] = [synth.chroma_qp_scaled(q, bd) for q in qps]
    pics["tools"] = synth.ENC_TOOLS if cf else synth.ENC_TOOLS & ~pkg.TOOL_ENC_CCLM
    pics["alf_aps"] = -1
    return pics


def _pinned(a):
    """A pinned host copy of a numpy array (asynchronous copies), as a numpy array."""
    t = torch.empty(max(a.nbytes, 1), dtype=torch.uint8, pin_memory=True)
    v = t.numpy()[:a.nbytes].view(a.dtype).reshape(a.shape)
    v[...] = a
    return v


def _decode_batch(ctx, c, seed):
    """Decoder records of c["n"] pictures: up to 8 different ones, coded by the library's encoder at the four
    quantisers, in turn; each picture with SAO and ALF parameters of its own."""
    g = _gen(seed)
    n, m = c["n"], min(c["n"], 8)
    qps = [QPS[i % 4] for i in range(m)]
    pics = _encoder_pics(c["w"], c["h"], c["bd"], c["cf"], c["ctu_log2"], qps)
    cw, ch = int(pics[0]["width"]), int(pics[0]["height"])
    cus, levels = ctx.encode_batch(pics, [_frame(g, c["w"], c["h"], cw, ch, c["bd"], c["cf"]) for _ in range(m)])
    ncu = len(cus) // m
    parts = []
    for i in range(m):
        k, lv = synth.compact_levels(pics[i], cus[i * ncu:(i + 1) * ncu], levels)
        p = pics[i:i + 1].copy()
        p["cu_offset"] = 0
        if c["sparse"]:
            p, k, lv = synth.sparsify(p, k, lv)
        parts.append((p[0], k, lv))
    rng = np.random.default_rng(seed)
    full = []
    for i in range(n):
        p, k, lv = parts[i % m]
        p = p.copy()
        p["tools"] = synth.DEC_TOOLS | (pkg.TOOL_SPARSE_LEVELS if c["sparse"] else 0)
        p["alf_aps"] = 0
        full.append((p, k, lv, synth.random_ctu_params(rng, cw, ch, 1 << c["ctu_log2"], c["bd"], c["cf"])))
    pics, cus, levels, ctus, aps = synth.assemble(full, synth.workload_aps(seed))
    return pkg.Batch(pics, _pinned(cus), torch.from_numpy(_pinned(levels)), _pinned(ctus), _pinned(aps))


class _View:
    """A device plane (or equally spaced planes of several pictures) of the library as torch sees it; it keeps the
    context alive, which owns the memory."""

    def __init__(self, ctx, ptr, shape, strides):
        self.ctx = ctx
        self.__cuda_array_interface__ = dict(shape=tuple(shape), strides=tuple(strides), typestr="<i2",
                                             data=(ptr, False), version=3)


def _views(ctx, where, n, dims):
    """int16 CUDA views of n pictures' planes, one per component where the pictures lie equally spaced, else one
    per plane. where(i, comp): (address, row pitch in samples); dims: (height, width) per component."""
    out = []
    for comp, (h, w) in enumerate(dims):
        if not h:
            continue
        at = [where(i, comp) for i in range(n)]
        step = {b[0] - a[0] for a, b in zip(at, at[1:])}
        if len(step) <= 1 and len({s for _, s in at}) == 1 and (not step or min(step) > 0):
            views = [_View(ctx, at[0][0], (n, h, w), (step.pop() if step else h * at[0][1] * 2, at[0][1] * 2, 2))]
        else:
            views = [_View(ctx, p, (h, w), (s * 2, 2)) for p, s in at]
        out += [torch.as_tensor(v, device="cuda") for v in views]
    return out


def _chroma(c):
    w, h = pkg.chroma_dims(c["w"], c["h"], c["cf"])
    return [(c["h"], c["w"]), (h, w), (h, w)]


def _prepare_decode(c, seed):
    ctx = pkg.Context(0)
    if c["io"] == "device":
        ctx.set_stream(_stream())
    batch = _decode_batch(ctx, c, seed)
    st = dict(ctx=ctx, batch=batch, io=c["io"])
    if c["io"] == "host":
        st["outs"] = [tuple(torch.zeros(d, dtype=torch.int16, pin_memory=True) if d[0] else None for d in _chroma(c))
                      for _ in range(c["n"])]
        return st
    ctx.prepare(batch)
    st["planes"] = _views(ctx, ctx.plane, c["n"], _chroma(c))
    return st


def _run_decode(st):
    ctx = st["ctx"]
    if st["io"] == "host":
        return [[p for p in planes if p is not None] for planes in ctx.decode_batch(st["batch"], st["outs"])]
    # the records and levels of every step go up, the planes stay on the device for their consumer
    ctx.upload(st["batch"])
    ctx.run()
    return st["planes"]


def _prepare_p(c, seed):
    w, h, s, chain = c["w"], c["h"], c["streams"], c["chain"]
    n, gw, gh = s * chain, w // 32, h // 32
    rng = np.random.default_rng(seed)
    m = min(n, 4)
    spec = [dict(width=w, height=h, bit_depth=8, chroma_format=1, ctu_log2=5, qp=QPS[i % 4]) for i in range(m)]
    pics, cus, levels, _, _ = synth.random_records(spec, seed=seed, tools=0)
    if c["sparse"]:
        pics, cus, levels = synth.sparsify(pics, cus, levels)
    cus = cus.reshape(m, gw * gh)
    rec = np.zeros((n, gw * gh), pkg.INTER_CU_DTYPE)
    pp = np.zeros(n, pkg.P_PIC_DTYPE)
    for i in range(n):
        rec[i]["cbf"], rec[i]["level_off"] = cus[i % m]["cbf"], cus[i % m]["level_off"]
        # global motion of the picture and, for a third of the units, their own; quarter samples
        mv = np.repeat(rng.integers(-48, 49, (1, 2)), gw * gh, 0)
        own = rng.random(gw * gh) < 0.33
        mv[own] = rng.integers(-160, 161, (int(own.sum()), 2))
        rec[i]["mv"][:, 0] = mv * 4
        rec[i]["ref_idx"] = (0, -1)
        rec[i]["inter_dir"], rec[i]["bcw_idx"], rec[i]["flags"] = 1, 2, pkg.INTER_CU_MERGE
        st, k = divmod(i, chain)
        pp[i]["width"], pp[i]["height"], pp[i]["qp"] = w, h, QPS[(i % m) % 4]
        pp[i]["options"] = pkg.SLICE_DEBLOCK if c["deblock"] else 0
        pp[i]["sparse"], pp[i]["num_refs"], pp[i]["cu_offset"] = int(c["sparse"]), 1, i * gw * gh
        pp[i]["ref_slot"][:] = s * k + st  # slots 0..s-1: the references; then the pictures, in order of depth
        pp[i]["out_slot"] = s * (k + 1) + st
    ctx = pkg.Context(0)
    ctx.set_stream(_stream())
    ctx.dpb_reserve(s * (chain + 1), w, h)
    g = _gen(seed)
    for i in range(s):
        ctx.dpb_upload(i, [p.cpu().numpy().astype(np.uint16) for p in _frame(g, w, h, w, h, 8, 1)])

    def where(i, comp):
        p, stride = ctypes.c_void_p(), ctypes.c_uint32()
        if pkg.lib().vvcg_dpb_plane(ctx._h, s + i, comp, ctypes.byref(p), ctypes.byref(stride)):
            raise RuntimeError("no such picture-buffer plane")
        return p.value, stride.value

    return dict(ctx=ctx, pics=pp, cus=_pinned(rec.reshape(-1)), levels=_pinned(levels),
                planes=_views(ctx, where, n, [(h, w), (h // 2, w // 2), (h // 2, w // 2)]))


def _run_p(st):
    st["ctx"].decode_p_batch(st["pics"], st["cus"], st["levels"])
    return st["planes"]


def _prepare_encode(c, seed):
    pics = _encoder_pics(c["w"], c["h"], c["bd"], c["cf"], 5, [QPS[i % 4] for i in range(c["n"])])
    g = _gen(seed)
    cw, ch = int(pics[0]["width"]), int(pics[0]["height"])
    srcs = [[p.cpu().pin_memory() for p in _frame(g, c["w"], c["h"], cw, ch, c["bd"], c["cf"]) if p is not None]
            for _ in range(c["n"])]
    ctx = pkg.Context(0)
    ctx.set_stream(_stream())
    return dict(ctx=ctx, pics=pics, srcs=srcs)


def _run_encode(st):
    cus, levels = st["ctx"].encode_batch(st["pics"], st["srcs"])
    return dict(cus=cus.view(np.uint8), levels=levels)


def _prepare_general(c, seed):
    # two different pictures, in turn: building their trees here is what takes the time
    m = min(c["n"], 2)
    parts = [synth.random_general_picture(c["w"], c["h"], ctu=c["ctu"], bd=c["bd"], qp=QPS[(i + 1) % 4], seed=seed + i,
                                          dep_quant=bool(i & 1)) for i in range(m)]
    batch = pkg.GenBatch(**synth.general_batch([parts[i % m] for i in range(c["n"])]))
    dims = _chroma(dict(c, cf=1))
    outs = [tuple(torch.zeros(d, dtype=torch.int16, pin_memory=True) for d in dims) for _ in range(c["n"])]
    return dict(ctx=pkg.Context(0), batch=batch, outs=outs)


def _run_general(st):
    return [list(p) for p in st["ctx"].decode_general(st["batch"], st["outs"])]


def _mc_blocks(rng, w, h, sub, bi):
    """The blocks of a picture (64x64 areas, each cut into equal blocks of 8..64 luma samples a side) with motion of
    up to 24 samples in 1/16 steps; coordinates and sizes in samples of the plane, which `sub` halves."""
    rows = []
    for y in range(0, h, 64):
        for x in range(0, w, 64):
            bw, bh = 1 << int(rng.integers(3, 7)), 1 << int(rng.integers(3, 7))
            for yy in range(y, min(y + 64, h), bh):
                for xx in range(x, min(x + 64, w), bw):
                    rows.append((xx, yy, min(bw, w - xx), min(bh, h - yy)))
    r = np.array(rows)
    b = np.zeros((2, len(r)), pkg.MC_BLOCK_DTYPE)
    for k in range(2):
        b[k]["x"], b[k]["y"], b[k]["w"], b[k]["h"] = r[:, 0], r[:, 1], r[:, 2], r[:, 3]
        b[k]["mv_x"], b[k]["mv_y"] = rng.integers(-384, 385, len(r)), rng.integers(-384, 385, len(r))
        whole = rng.random(len(r)) < 0.15
        b[k]["mv_x"][whole] &= ~15
        b[k]["mv_y"][whole] &= ~15
        b[k]["flags"] = pkg.MC_BI if bi else 0
    out = []
    for div in (1, 2):
        d = b.copy()
        for f in ("x", "y", "w", "h"):
            d[f] //= div
        size = d[0]["w"].astype(np.int64) * d[0]["h"]
        d["out_offset"] = np.cumsum(size) - size
        out.append(([torch.from_numpy(x.view(np.uint8).reshape(-1).copy()).cuda() for x in d], int(size.sum())))
    return out


def _prepare_mc(c, seed):
    rng = np.random.default_rng(seed)
    g = _gen(seed)
    refs = [_frame(g, c["w"], c["h"], c["w"], c["h"], c["bd"], 1) for _ in range(2)]
    if c["bd"] == 8:
        refs = [[p.to(torch.uint8) for p in r] for r in refs]
    luma, chroma = _mc_blocks(rng, c["w"], c["h"], 2, c["bi"])
    plans = []
    for comp in range(3):
        blocks, n = luma if comp == 0 else chroma
        plans.append(dict(comp=comp, blocks=blocks, pred=[torch.empty(n, dtype=torch.int32, device="cuda")
                                                          for _ in range(2 if c["bi"] else 1)],
                          out=torch.empty(n, dtype=torch.int16, device="cuda")))
    ctx = pkg.Context(0)
    ctx.set_stream(_stream())
    return dict(ctx=ctx, refs=refs, plans=plans, bd=c["bd"], bi=c["bi"])


def _run_mc(st):
    ctx, bd = st["ctx"], st["bd"]
    res = []
    for p in st["plans"]:
        for k, pred in enumerate(p["pred"]):
            ref, blocks = st["refs"][k][p["comp"]], p["blocks"][k]
            if bd == 8:
                (ctx.mc_chroma_420_8 if p["comp"] else ctx.mc_luma_8)(ref, blocks, pred)
            elif p["comp"]:
                ctx.mc_chroma(ref, bd, pkg.CHROMA_420, blocks, pred)
            else:
                ctx.mc_luma(ref, bd, blocks, pred)
        if st["bi"]:
            ctx.mc_bi_average(p["pred"][0], p["pred"][1], 2, bd, p["out"])
            res.append(p["out"])
        else:
            res.append(p["pred"][0])
    return res


def _prepare_tu(c, seed):
    """Units of 4x4..64x64 (and the narrow shapes) with every tool, repeating a set of up to 1,000; residuals of a
    Laplacian around each unit's own level."""
    n, m = c["n"], min(c["n"], 1000)
    recs, _, total = synth.random_tu_records(m, seed=c["seed_shape"], forward=True)
    k = -(-n // m)
    recs = np.tile(recs, k).reshape(k, m)
    recs["in_off"] += (np.arange(k, dtype=np.uint32) * total)[:, None]
    recs = recs.reshape(-1)[:n]
    size = 1 << (recs["log2_w"].astype(np.int64) + recs["log2_h"])
    recs["out_off"] = recs["in_off"]
    total = int(recs["in_off"][-1]) + int(size[-1])
    g = _gen(seed)
    level = torch.randn(n, generator=g, device="cuda") * 24
    u = torch.rand(total, generator=g, device="cuda") - 0.5
    data = torch.repeat_interleave(level, torch.from_numpy(size).cuda()) - 14 * u.sign() * torch.log1p(-2 * u.abs() + 1e-6)
    data = data.round().clamp(-250, 250).to(torch.int16)
    ctx = pkg.Context(0)
    ctx.set_stream(_stream())
    return dict(ctx=ctx, recs=recs, data=data, levels=torch.empty_like(data), out=torch.empty_like(data))


def _run_tu(st):
    st["ctx"].tu_forward(st["recs"], st["data"], st["levels"])
    st["ctx"].tu_inverse(st["recs"], st["levels"], st["out"])
    return dict(levels=st["levels"], residual=st["out"])


def _blocks_plane(c, seed):
    """A frame whose whole 32x32 blocks are the case's n blocks: 60 in a row at 1080p."""
    cols = min(60, c["n"])
    rows = -(-c["n"] // cols)
    w, h = cols * 32, rows * 32
    plane = _frame(_gen(seed), w, h, w, h, c["bd"], 0)[0]
    k = torch.arange(c["n"], device="cuda", dtype=torch.int32)
    return plane, torch.stack([k % cols * 32, k // cols * 32], 1).contiguous()


def _cnn_state(c, seed):
    plane, xy = _blocks_plane(c, seed)
    ctx = pkg.Context(0)
    ctx.set_stream(_stream())
    ctx.torch_stream = _stream()
    params = torch.from_numpy(cnn.init_params(seed)).cuda()
    return dict(ctx=ctx, plane=plane, xy=xy, params=params, bd=c["bd"], qp=c["qp"])


def _run_cnn_forward(st):
    with st["ctx"].torch_stream_scope():
        logits, gap, _ = st["ctx"].cnn_forward(st["plane"], st["bd"], st["xy"], st["params"], st["qp"], sync=False)
    return dict(logits=logits, gap=gap)


def _prepare_cnn_train(c, seed):
    st = _cnn_state(c, seed)
    g = _gen(seed + 1)
    labels = torch.stack([torch.randint(0, 67, (c["n"],), generator=g, device="cuda"),
                          torch.randint(0, 6, (c["n"],), generator=g, device="cuda")], 1).to(torch.uint8)
    soft = torch.softmax(3 * torch.randn((c["n"], 67), generator=g, device="cuda"), 1) if c["soft"] else None
    z = torch.zeros_like(st["params"])
    st.update(labels=labels, soft=soft, m=z.clone(), v=z.clone(), step=0)
    return st


def _run_cnn_train(st):
    st["step"] += 1
    with st["ctx"].torch_stream_scope():
        loss, grads = st["ctx"].cnn_train_step(st["plane"], st["bd"], st["qp"], st["xy"], st["labels"], st["params"],
                                               st["m"], st["v"], st["step"], 1e-3, sync=False, soft=st["soft"])
    return dict(loss=loss, grads=grads, params=st["params"])


def _prepare_search(c, seed):
    st = _cnn_state(c, seed)
    # logits as confident as a trained pruner's
    st["logits"] = 2.5 * torch.randn((c["n"], pkg.CNN_OUT), generator=_gen(seed + 1), device="cuda") if c["pruned"] else None
    st["lam"] = cnn.search_lambda_q8(c["qp"], c["bd"])
    st["out"] = torch.zeros(c["n"] * pkg.CTU_SEARCH_RES_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    return st


def _run_search(st):
    st["ctx"].ctu_search_xy(st["plane"], st["bd"], st["lam"], st["xy"], st["logits"], 6, 3, 0.79, out=st["out"],
                            sync=False)
    return st["out"]


_PREPARE = dict(decode=_prepare_decode, p=_prepare_p, encode=_prepare_encode, general=_prepare_general, mc=_prepare_mc,
                tu=_prepare_tu, cnn_forward=_cnn_state, cnn_train=_prepare_cnn_train, search=_prepare_search)
_RUN = dict(decode=_run_decode, p=_run_p, encode=_run_encode, general=_run_general, mc=_run_mc, tu=_run_tu,
            cnn_forward=_run_cnn_forward, cnn_train=_run_cnn_train, search=_run_search)


def prepare(case, seed):
    st = _PREPARE[case["kind"]](case, seed)
    st["kind"] = case["kind"]
    torch.cuda.synchronize()
    return st


def run(state):
    return _RUN[state["kind"]](state)


# -------------------------------------------------------------------- work --

_CHROMA_SHARE = (0.0, 0.5, 1.0, 2.0)  # chroma samples per luma sample
_FWD_MACS = 1024 * (18 * 32 + 3 * 9 * 32 * 32) + 73 * 32  # of the pruner on one 32x32 block


def work(case):
    kind, n = case["kind"], case.get("n", 1)
    if kind in ("decode", "encode", "general"):
        # one 16-bit write of every sample; the levels and records: about 0.1 byte per sample in the sparse form
        # and two in the dense one, or the source samples read and the dense levels written by the encoder
        samples = case["w"] * case["h"] * n * (1 + _CHROMA_SHARE[case.get("cf", 1)])
        per = {"decode": 2 + (0.1 if case.get("sparse") else 2), "encode": 4, "general": 4}[kind]
        return {"bytes": samples * per, "flops": 0}
    if kind == "p":  # a reference sample read and a sample written, and the levels
        samples = case["w"] * case["h"] * 1.5 * case["streams"] * case["chain"]
        return {"bytes": samples * (4 + (0.3 if case["sparse"] else 1.2)), "flops": 0}
    if kind == "mc":
        samples = case["w"] * case["h"] * 1.5
        ref = 1 if case["bd"] == 8 else 2
        return {"bytes": samples * (2 * ref + 2 if case["bi"] else ref + 4), "flops": 0}
    if kind == "tu":  # about 520 coefficients a unit: residual in, levels out, levels in, residual out
        return {"bytes": n * 520 * 8, "flops": 0}
    if kind == "cnn_forward":
        return {"bytes": n * (2048 + 4 * (73 + 32)), "flops": 2 * n * _FWD_MACS}
    if kind == "cnn_train":
        return {"bytes": n * 2048 + 30761 * 4 * 8, "flops": 6 * n * _FWD_MACS}
    # 67 predictions of each of the six splits' blocks, and their 8x8 Hadamard sums (6 butterflies a sample)
    return {"bytes": n * (2048 + 36), "flops": n * 1024 * 6 * 67 * 14 * (0.2 if case["pruned"] else 1)}


# ------------------------------------------------------------------- exact --

def _network(c, seed, params, plane, xy):
    """The pruner in 64 bits: (logits, gap) as plain torch gives them."""
    d = plane.double()
    blocks = torch.stack([d[y:y + 32, x:x + 32] for x, y in xy.tolist()])[:, None] / ((1 << c["bd"]) - 1)
    x = torch.cat([blocks, torch.full_like(blocks, c["qp"] / 63.0)], 1)
    w1, b1, convs, wi, bi, ws, bs = cnn.unpack(params)
    x = torch.relu(torch.nn.functional.conv2d(x, w1, b1, padding=1))
    for w, b in convs:
        x = torch.relu(torch.nn.functional.conv2d(x, w, b, padding=1))
    gap = x.mean((2, 3))
    return torch.cat([gap @ wi.T + bi, gap @ ws.T + bs], 1), gap


def exact(case, seed):
    if case["kind"] not in ("cnn_forward", "cnn_train"):
        return None  # whole numbers
    st = prepare(case, seed)
    params = st["params"].double().requires_grad_(case["kind"] == "cnn_train")
    logits, gap = [], []
    if case["kind"] == "cnn_forward":
        with torch.no_grad():
            for a in range(0, case["n"], 256):
                lo, ga = _network(case, seed, params, st["plane"], st["xy"][a:a + 256])
                logits.append(lo)
                gap.append(ga)
        return dict(logits=torch.cat(logits), gap=torch.cat(gap))
    n = case["n"]
    loss = 0.0
    for a in range(0, n, 128):
        b = min(n, a + 128)
        lo, _ = _network(case, seed, params, st["plane"], st["xy"][a:b])
        lm, ls = torch.log_softmax(lo[:, :67], 1), torch.log_softmax(lo[:, 67:], 1)
        lab = st["labels"][a:b].long()
        mode = -(st["soft"][a:b].double() * lm).sum() if case["soft"] else -lm.gather(1, lab[:, :1]).sum()
        part = (mode - ls.gather(1, lab[:, 1:]).sum()) / n
        part.backward()
        loss += float(part)
    g = params.grad
    # the first Adam step from zero moments (0.9, 0.999, 1e-8)
    new = params.detach() - 1e-3 * g / (g.abs() + 1e-8)
    return dict(loss=torch.tensor([loss], dtype=torch.float64), grads=g, params=new)
