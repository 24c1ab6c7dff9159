"""The work a program has this framework do, as cases that can be timed: textures encoded, decoded, mip-mapped and packed
through the public Python calls, at the sizes and contents of the benchmark, the tests and the tools around them.

listed() gives the cases, draw(rng) one more of the same ranges, prepare(case, seed) the inputs and handles a program
holds before the call, run(state) one pass, work(case) the bytes and operations a pass cannot do without. All outputs are
blocks, texels or files: bytes, which are either equal or wrong, so no case has an output that a wider type would hold
more exactly.

A case's "kind":
  encode   bc_encode_dev / astc_encode_dev / bc6h_encode_dev on a texture in device memory
  decode   the decoders on blocks in device memory (the blocks are this encoder's own)
  mips     mip_chain_dev: every level below a texture
  batch    Batch.run: many textures with their mip chains and mixed formats, one graph launch
  rdo      bc_encode_rdo_dev in bands of 8 block rows, as a tool encodes for a later compressor
  host     bc_encode on an image in ordinary host memory, the call that replaces the CPU encoder's
"""
import numpy as np
import torch

import zap_b200 as zt
import zap_b200.synth as synth

FMT = {"bc1": zt.BC1, "bc3": zt.BC3, "bc4": zt.BC4, "bc5": zt.BC5, "bc7": zt.BC7, "bc6h": zt.BC6H, "astc": zt.ASTC4X4}
# palette entries each texel is compared with in one fit, and the channels compared
FIT = {"bc1": (4, 3), "bc3": (12, 2), "bc4": (8, 1), "bc5": (16, 1), "bc7": (16, 4), "bc6h": (16, 3), "astc": (16, 4)}


def listed():
    return [
        # the headline: an albedo texture with an alpha channel, as an asset pipeline bakes it
        {"name": "bc7_2048_alpha", "kind": "encode", "fmt": "bc7", "src": "rgba8", "content": "alpha", "w": 2048, "h": 2048},
        # a screenshot-sized opaque image whose sides are not multiples of four and whose rows are not 16-byte aligned
        {"name": "bc7_1918x1077_opaque", "kind": "encode", "fmt": "bc7", "src": "rgba8", "content": "opaque", "w": 1918, "h": 1077},
        # an icon or a small atlas tile encoded while a program runs: latency and launches
        {"name": "bc7_64_alpha", "kind": "encode", "fmt": "bc7", "src": "rgba8", "content": "alpha", "w": 64, "h": 64},
        # the benchmark's small opaque texture
        {"name": "bc1_512_opaque", "kind": "encode", "fmt": "bc1", "src": "rgba8", "content": "opaque", "w": 512, "h": 512},
        # a tangent-space normal map from its two channels
        {"name": "bc5_2048_normal", "kind": "encode", "fmt": "bc5", "src": "rg8", "content": "normal", "w": 2048, "h": 2048},
        # an HDR environment or light map in half floats
        {"name": "bc6h_2048_hdr", "kind": "encode", "fmt": "bc6h", "src": "rgb16f", "content": "hdr", "w": 2048, "h": 2048},
        # the mobile build of an opaque texture
        {"name": "astc_1024_opaque", "kind": "encode", "fmt": "astc", "src": "rgba8", "content": "opaque", "w": 1024, "h": 1024},
        # blocks back to texels on the device, for quality checks and previews
        {"name": "bc7_decode_2048_alpha", "kind": "decode", "fmt": "bc7", "content": "alpha", "w": 2048, "h": 2048},
        # the mip chain of a large colour texture, averaged in linear light
        {"name": "mips_4096_srgb", "kind": "mips", "srgb": True, "content": "opaque", "w": 4096, "h": 4096},
        # an asset bundle: textures of uneven sizes, full chains, 40 % BC1, 20 % BC3, 40 % BC7
        {"name": "batch_64_textures", "kind": "batch", "n": 64, "lo": 6, "hi": 11, "bundle": 1},
        # rate-distortion encode of a ragged texture with alpha for an archive, in the bands a tool's threads take
        {"name": "rdo_bc3_1021x767", "kind": "rdo", "fmt": "bc3", "content": "alpha", "w": 1021, "h": 767, "rdo": 30.0},
        # the drop-in call on a host image: copy in, encode, copy out
        {"name": "host_bc1_1024_opaque", "kind": "host", "fmt": "bc1", "content": "opaque", "w": 1024, "h": 1024},
    ]


def _side(rng, lo, hi):
    """A side between lo and hi, spread over its logarithm; four in ten are any number, the others powers of two or
    multiples of four, as textures mostly are."""
    v = lo * (hi / lo) ** rng.random()
    u = rng.random()
    if u < 0.4:
        return max(lo, min(hi, int(v)))
    if u < 0.7:
        return max(lo, min(hi, 1 << round(np.log2(v))))
    return max(lo, min(hi, 4 * round(v / 4)))


def _size(rng, lo, hi):
    w = _side(rng, lo, hi)
    h = w if rng.random() < 0.4 else max(lo, min(hi, _side(rng, max(lo, w // 4), min(hi, 4 * w))))
    return {"w": int(w), "h": int(h)}


def draw(rng):
    kind = rng.choices(("encode", "decode", "mips", "batch", "rdo", "host"), (6, 2, 1, 1, 1, 1))[0]
    if kind == "encode":
        fmt = rng.choice(("bc1", "bc3", "bc4", "bc5", "bc7", "bc7", "bc6h", "astc"))
        if fmt == "bc6h":
            src, content = rng.choice((("rgb16f", "hdr"), ("rgba32f", "hdr")))
        elif fmt == "bc5":
            src, content = rng.choice((("rg8", "normal"), ("rgba8", "alpha")))
        elif fmt == "bc4":
            src, content = rng.choice((("r8", "opaque"), ("rgba8", "opaque")))
        else:
            src, content = "rgba8", "alpha" if fmt == "bc3" else rng.choice(("alpha", "opaque"))
        return {"kind": kind, "fmt": fmt, "src": src, "content": content, **_size(rng, 16, 2048)}
    if kind == "decode":
        fmt = rng.choice(("bc1", "bc3", "bc4", "bc5", "bc7", "bc7", "bc6h", "astc"))
        content = {"bc6h": "hdr", "bc3": "alpha"}.get(fmt) or rng.choice(("alpha", "opaque"))
        return {"kind": kind, "fmt": fmt, "content": content, **_size(rng, 64, 2048)}
    if kind == "mips":
        return {"kind": kind, "srgb": rng.random() < 0.6, "content": rng.choice(("alpha", "opaque")), **_size(rng, 64, 4096)}
    if kind == "batch":
        return {"kind": kind, "n": rng.randint(8, 64), "lo": 6, "hi": rng.randint(8, 11), "bundle": rng.randint(1, 999)}
    if kind == "rdo":
        fmt = rng.choice(("bc1", "bc3", "bc7"))
        content = "alpha" if fmt == "bc3" else rng.choice(("alpha", "opaque"))
        return {"kind": kind, "fmt": fmt, "content": content, "rdo": rng.choice((10.0, 30.0, 60.0)), **_size(rng, 64, 1024)}
    fmt = rng.choice(("bc1", "bc3", "bc7", "astc"))
    return {"kind": kind, "fmt": fmt, "content": "alpha" if fmt == "bc3" else rng.choice(("alpha", "opaque")), **_size(rng, 64, 2048)}


def _texture(content, src, w, h, seed):
    """The texture on the GPU in the layout a program holds it in."""
    if content == "normal":
        return synth.normal_map(w, h, seed, "cuda")
    if content == "hdr":
        t = synth.hdr_texture(w, h, seed, "cuda")
        if src == "rgba32f":
            t = torch.cat((t.float(), torch.ones(h, w, 1, device="cuda")), 2).contiguous()
        return t
    t = synth.colour_texture(w, h, seed, "noise" if content == "alpha" else "opaque", "cuda")
    return t[..., :1].contiguous() if src == "r8" else t


def _encode(t, fmt):
    return zt.bc6h_encode_dev(t) if fmt == "bc6h" else zt.bc_encode_dev(t, FMT[fmt])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        sizes = synth.batch_sizes(case["n"], case["bundle"], case["lo"], case["hi"])  # "bundle": its textures' sizes and formats
        textures = [synth.colour_texture(w, h, seed * 1000 + i, "noise" if i % 2 else "opaque", "cuda") for i, (w, h) in enumerate(sizes)]
        return {"kind": kind, "batch": zt.Batch(textures, synth.batch_formats(case["n"], case["bundle"]))}
    w, h, content = case["w"], case["h"], case["content"]
    fmt = case.get("fmt")
    state = {"kind": kind, "fmt": fmt, "w": w, "h": h, "rdo": case.get("rdo"), "srgb": case.get("srgb")}
    t = _texture(content, case.get("src", "rgb16f" if content == "hdr" else "rgba8"), w, h, seed)
    if kind == "decode":
        state["blocks"] = _encode(t, fmt)
    elif kind == "host":
        state["image"] = t.cpu().numpy()
    else:
        state["texture"] = t
    return state


def run(s):
    kind, fmt = s["kind"], s.get("fmt")
    if kind == "encode":
        return _encode(s["texture"], fmt)
    if kind == "decode":
        if fmt == "bc6h":
            return zt.bc6h_decode_dev(s["blocks"], s["w"], s["h"])
        if fmt == "astc":
            return zt.astc_decode_dev(s["blocks"], s["w"], s["h"])
        return zt.bc_decode_dev(s["blocks"], s["w"], s["h"], FMT[fmt])
    if kind == "mips":
        return zt.mip_chain_dev(s["texture"], s["srgb"])
    if kind == "batch":
        s["batch"].run()
        return s["batch"].outputs
    if kind == "rdo":
        return zt.bc_encode_rdo_dev(s["texture"], FMT[fmt], s["rdo"], band_rows=8)
    return zt.astc_encode(s["image"]) if fmt == "astc" else zt.bc_encode(s["image"], FMT[fmt])


def work(case):
    """bytes: the source read once and the result written once. flops: the arithmetic of the least a result takes: one palette
    fit per block for an encoder, one interpolation per texel channel for a decoder, one average for a mip."""
    kind = case["kind"]

    def one(fmt, w, h, texel):
        blocks = ((w + 3) // 4) * ((h + 3) // 4)
        entries, channels = FIT[fmt]
        return w * h * texel + blocks * zt.block_bytes(FMT[fmt]), blocks * 16 * entries * (3 * channels + 1)

    if kind == "batch":
        nbytes = flops = 0
        names = {v: k for k, v in FMT.items()}
        for (w, h), f in zip(synth.batch_sizes(case["n"], case["bundle"], case["lo"], case["hi"]), synth.batch_formats(case["n"], case["bundle"])):
            nbytes += w * h * 4 / 3  # the levels below are written once, and read from where they were just written
            texel = 4
            for k in range(zt.mip_levels(w, h)):
                b, n = one(names[f], max(1, w >> k), max(1, h >> k), texel)
                nbytes, flops, texel = nbytes + b, flops + n, 0
        return {"bytes": nbytes, "flops": flops}
    w, h = case["w"], case["h"]
    if kind == "mips":
        return {"bytes": w * h * 4 * 4 / 3, "flops": w * h / 3 * 4 * 4}
    fmt = case["fmt"]
    if kind == "decode":
        blocks = ((w + 3) // 4) * ((h + 3) // 4)
        return {"bytes": w * h * (8 if fmt == "bc6h" else 4) + blocks * zt.block_bytes(FMT[fmt]), "flops": w * h * 4 * 4}
    nbytes, flops = one(fmt, w, h, {"rgba8": 4, "rg8": 2, "r8": 1, "rgb16f": 6, "rgba32f": 16}[case.get("src", "rgba8")])
    return {"bytes": nbytes, "flops": flops}
