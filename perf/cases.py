"""The framework's work as its users have it done, for timing and for comparing outputs.

Four kinds of case, each through the public entry points (the processor classes, and the C ABI of
include/rd_gpu.h where the caller's own buffers are passed in):

  develop  one photograph: develop (normalize, highlight, demosaic, capture sharpening), spatial pass
           (optics, area reduction, white balance, matrix), render (adjustments, sRGB8, histogram);
           the mosaic in pinned host memory, as a decoder leaves it, or resident on the device, as an
           open image keeps it; the picture and its histogram come back to pinned host memory.
  batch    several photographs of uneven sizes and settings through rd_develop_batch.
  edit     the re-render of a resident preview base for one slider event (rd_render_device_noalloc).
  export   a full-resolution base to its output rows (rd_render_output_device) and, for a file, the
           rows to PNG or JPEG on the device (rd_encode_png_device, rd_encode_jpeg_device).

Sizes, levels, lenses and settings are those of the repository's benchmark workloads and tests; the
drawn cases spread over the ranges between them.
"""

import ctypes
import math

import numpy as np
import torch

from rohditor_gb300 import (CaptureContract, ColorContract, Device, GpuSensorProcessor, GpuSpatialProcessor,
                            OpticsExecution, OutputSpec, SensorDescription, capture_ceilings, clip_levels,
                            light_tone_lut, opposed_levels, standard_base_lut)
from rohditor_gb300 import _ffi
from rohditor_gb300.workloads import CAMERA_TO_REC2020, hsl_bands, preview_dimensions, sixteen_knot_curve

AS_SHOT = (2.0, 1.0, 1.6)
ICC = bytes(range(256)) * 12  # a profile's worth of bytes for the file headers
LENSES = {
    "none": None,
    "poly5": dict(distortion="poly5", distortion_k=(-0.02, 0.005, 0.0), tca="linear", tca_red=(1.0003, 0.0, 0.0),
                  tca_blue=(0.9997, 0.0, 0.0)),
    "ptlens": dict(distortion="ptlens", distortion_k=(0.01, -0.03, 0.02)),
    "poly3": dict(distortion="poly3", distortion_k=(-0.01, 0.0, 0.0)),
}
# What an adjustment set switches on: the plain rendering, the benchmark's edit, every slider.
EDITS = ("plain", "tone", "full")


def _develop(name, width, height, bits=14, black=512.0, cfa="RGGB", crop=0, highlight="opposed", demosaic="amaze",
             iterations=10, radius=0.7, lens="poly5", long_edge=2560, edit="tone", resident=True, hot=0.0):
    return dict(name=name, kind="develop", width=width, height=height, bits=bits, black=black, cfa=cfa, crop=crop,
                highlight=highlight, demosaic=demosaic, iterations=iterations, radius=radius, lens=lens,
                long_edge=long_edge, edit=edit, resident=resident, hot=hot)


def _export(name, width, height, format="srgb8", primaries="srgb", policy="clip", dither="none", orientation="normal",
            headroom=1.0, file="rows", quality=90, edit="tone"):
    return dict(name=name, kind="export", width=width, height=height, format=format, primaries=primaries,
                policy=policy, dither=dither, orientation=orientation, headroom=headroom, file=file, quality=quality,
                edit=edit)


def listed():
    return [
        # A tile or thumbnail sized frame from the decoder to the screen: launches and host work count.
        _develop("develop_small", 512, 344, bits=12, black=256.0, highlight="clip", iterations=8, long_edge=256,
                 resident=False),
        # The plain development of a 6 MP frame at its own size (the plain_3mp workload).
        _develop("develop_plain", 3008, 2008, highlight="clip", iterations=0, lens="none", long_edge=3008,
                 edit="plain"),
        # The headline workload: 24 MP, every stage, an image that is open already.
        _develop("develop_24mp", 6048, 4024),
        # A 12-bit 12 MP frame with masked borders, the faster demosaic, from the decoder.
        _develop("develop_12mp_rcd", 4000, 3000, bits=12, black=128.0, cfa="GRBG", crop=8, demosaic="rcd",
                 iterations=5, resident=False),
        # A quick look at a 45 MP frame: interpolation only, through a Poly3 lens.
        _develop("develop_45mp_mhc", 8256, 5504, cfa="BGGR", highlight="clip", demosaic="mhc", iterations=0,
                 lens="poly3", edit="plain", resident=False),
        # The largest configured sensor: 102 MP, 16 bits, hot pixels, 20 iterations.
        _develop("develop_102mp", 11648, 8736, bits=16, black=1024.0, iterations=20, hot=0.005),
        # A short import queue of uneven frames.
        dict(name="batch_uneven", kind="batch", count=5, lanes=3, iterations=5, largest=45),
        # One slider event on the 24 MP image's preview, every adjustment on.
        dict(name="edit_preview", kind="edit", width=2560, height=1703, edit="full"),
        # The wide-gamut HDR export of the export stream.
        _export("export_f16_p3", 6048, 4024, format="extended_f16", primaries="display_p3", policy="chroma_compress",
                headroom=4.0),
        # A linear archive of an odd sized portrait, turned upright.
        _export("export_f32_turned", 4001, 2667, format="extended_f32", orientation="rotate90", headroom=2.0,
                edit="exposure"),
        # 16-bit print file.
        _export("export_png16", 6048, 4024, format="srgb16", policy="chroma_compress", dither="ordered8x8", file="png"),
        # 8-bit file for the web, from an odd sized frame.
        _export("export_jpeg", 5999, 4001, file="jpeg"),
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("develop", "develop", "develop", "edit", "export", "export", "batch"))
    long = _spread(rng, 480, 9504)
    short = max(320, int(long * rng.uniform(0.55, 0.8)))
    width, height = (long, short) if rng.random() < 0.8 else (short, long)
    if kind == "develop":
        bits = rng.choice((12, 14, 14, 16))
        c = _develop("", width, height, bits=bits, black=rng.uniform(0.015, 0.06) * (1 << bits),
                     cfa=rng.choice(("RGGB", "BGGR", "GRBG", "GBRG")), crop=rng.choice((0, 0, 8, 13, 30)),
                     highlight=rng.choice(("opposed", "opposed", "clip")),
                     demosaic=rng.choice(("amaze", "amaze", "rcd", "mhc", "bilinear")),
                     iterations=rng.choice((0, 5, 8, 10, 20)), radius=round(rng.uniform(0.5, 1.2), 3),
                     lens=rng.choice(tuple(LENSES)), long_edge=rng.choice((640, 1280, 2560, 9504)),
                     edit=rng.choice(EDITS), resident=rng.random() < 0.5, hot=rng.choice((0.0, 0.0, 0.005)))
    elif kind == "edit":
        long = _spread(rng, 320, 3840)
        c = dict(kind="edit", width=long, height=max(2, int(long * rng.uniform(0.5, 1.5))), edit=rng.choice(EDITS))
    elif kind == "export":
        fmt = rng.choice(("srgb8", "srgb8", "srgb16", "extended_f16", "extended_f32"))
        file = rng.choice({"srgb8": ("rows", "png", "jpeg"), "srgb16": ("rows", "png")}.get(fmt, ("rows",)))
        c = _export("", width, height, format=fmt, primaries=rng.choice(("srgb", "display_p3")),
                    policy=rng.choice(("clip", "chroma_compress")),
                    dither=rng.choice(("none", "ordered8x8")) if fmt.startswith("srgb") else "none",
                    orientation=rng.choice(("normal", "normal", "rotate90", "rotate180", "transpose")),
                    headroom=rng.choice((1.0, 2.0, 4.0)) if fmt.startswith("ext") else 1.0, file=file,
                    quality=rng.randint(60, 98), edit=rng.choice(EDITS + ("exposure",)))
    else:
        c = dict(kind="batch", count=rng.randint(2, 5), lanes=rng.randint(1, 4), iterations=rng.choice((5, 8)),
                 largest=rng.choice((12, 24, 45)), at=rng.randint(0, 99))
    c.pop("name", None)
    return c


# ---------------------------------------------------------------- what a program keeps
_device = None


def _dev():
    global _device
    if _device is None:
        _device = Device(0)
    return _device


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _color(edit, rng, wb=AS_SHOT, cam=CAMERA_TO_REC2020):
    seed = int(rng.integers(1 << 30))
    ev = float(rng.uniform(-0.5, 0.8))
    kw = dict(wb_gains=wb, camera_to_rec2020=cam)
    if edit == "exposure":
        return ColorContract(exposure_ev=ev, **kw)
    kw["base_lut"] = standard_base_lut()
    if edit == "tone":
        kw.update(exposure_ev=ev, tone_lut=sixteen_knot_curve(seed), hsl=hsl_bands(seed))
    if edit == "full":
        kw.update(exposure_ev=ev, tone_lut=sixteen_knot_curve(seed), hsl=hsl_bands(seed), saturation=1.15,
                  vibrance=0.2, light_tone_lut=light_tone_lut(0.3, -0.4, 0.5, 0.2, -0.2),
                  grading=np.random.default_rng(seed).uniform(-0.15, 0.15, (3, 3)).astype(np.float32))
    return ColorContract(**kw)


def _optics(lens, width, height, rng):
    if LENSES[lens] is None:
        return None
    vig = tuple(float(v) for v in (-rng.uniform(0.2, 0.4), rng.uniform(0.02, 0.08), -rng.uniform(0.0, 0.02)))
    return OpticsExecution(width=width, height=height, vignetting_k=vig, **LENSES[lens])


def _mosaic(width, height, bits, black, cfa, seed, blobs, hot, pinned):
    """The seeded scene's samples: a pinned host array, as a decoder fills it, or a device array."""
    d = _ffi.SynthDesc()
    d.width, d.height, d.cfa, d.bits = width, height, _ffi.CFA[cfa], bits
    d.black, d.white, d.clip_fraction = black, float((1 << bits) - 1), 0.05 if blobs else 0.02
    for c in range(3):
        d.gains[c] = min(AS_SHOT) / AS_SHOT[c]
    d.seed, d.highlight_blobs, d.hot_pixel_fraction = seed, 1 if blobs else 0, hot
    dev = _dev()
    on = torch.empty((height, width), dtype=torch.int16, device="cuda")
    torch.cuda.synchronize()  # the context has a stream of its own
    dev.check(dev.lib.rd_synth_mosaic_device(dev.handle, ctypes.byref(d), _ptr(on)))
    dev.synchronize()
    if not pinned:
        return on
    return torch.empty((height, width), dtype=torch.int16, pin_memory=True).copy_(on)


def _sensor(c, wb=AS_SHOT):
    white = float((1 << c["bits"]) - 1)
    m = c["crop"]
    crop = (m, m, c["width"] - 2 * m, c["height"] - 2 * m) if m else None
    kw = dict(sensor_width=c["width"], sensor_height=c["height"], cfa=c["cfa"], crop=crop, black=(c["black"],),
              white=(white,), highlight=c["highlight"], demosaic=c["demosaic"], demosaic_balance=AS_SHOT)
    if c["highlight"] == "opposed":
        kw["detection_levels"], kw["neutral_ceiling"] = opposed_levels(1.0, AS_SHOT)
    else:
        kw["clip_levels"] = clip_levels(1.0, wb)
    return SensorDescription(**kw)


def _capture(c, wb=AS_SHOT):
    if not c["iterations"]:
        return None
    return CaptureContract(amount=0.5, radius=c["radius"], noise_protection=0.5, iterations=c["iterations"],
                           ceilings=capture_ceilings(c["highlight"], 1.0, wb))


def _outputs(width, height):
    return (torch.empty((height, 3 * width), dtype=torch.uint8, pin_memory=True),
            torch.empty(1024, dtype=torch.int64, pin_memory=True))


def _batch_images(case):
    """The uneven batch's photographs: the four configured sensors up to the largest asked for."""
    sensors = [s for s in ((4000, 3000, 12, 12), (6048, 4024, 14, 24), (8256, 5504, 14, 45))
               if s[3] <= case["largest"]]
    out = []
    for k in range(case["count"]):
        w, h, bits, _ = sensors[(k + case.get("at", 0)) % len(sensors)]
        out.append(_develop("", w, h, bits=bits, black=128.0 if bits == 12 else 512.0,
                            cfa=("RGGB", "BGGR", "GRBG", "GBRG")[(k + case.get("at", 0)) % 4],
                            iterations=case["iterations"]))
    return out


def _base(width, height, seed):
    """A developed and white-balanced full-size base, resident on the device."""
    dev = _dev()
    c = _develop("", width, height, highlight="clip", demosaic="mhc")
    mosaic = _mosaic(width, height, 14, 512.0, "RGGB", seed, True, 0.0, False)
    source = GpuSensorProcessor(dev).develop_device(mosaic.data_ptr(), width, _sensor(c))
    base = GpuSpatialProcessor(dev).reduce_preview(source, None, (width, height), AS_SHOT, CAMERA_TO_REC2020)
    source.release()
    return base


# ---------------------------------------------------------------- prepare and run
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    s = {"case": case, "kind": case["kind"]}
    if case["kind"] == "develop":
        s["sensor"] = _sensor(case)
        w, h = s["sensor"].crop_size
        s["mosaic"] = _mosaic(case["width"], case["height"], case["bits"], case["black"], case["cfa"], seed, True,
                              case["hot"], not case["resident"])
        s["capture"], s["optics"] = _capture(case), _optics(case["lens"], w, h, rng)
        if s["optics"] is not None:
            s["optics"].to_c()
        s["target"] = preview_dimensions(w, h, case["long_edge"])
        s["color"] = _color(case["edit"], rng).to_c()
        s["srgb"], s["hist"] = _outputs(*s["target"])
    elif case["kind"] == "batch":
        images = _batch_images(case)
        s["items"], s["out"], s["keep"] = (_ffi.BatchItem * len(images))(), [], []
        for k, c in enumerate(images):
            w, h = c["width"], c["height"]
            mosaic = _mosaic(w, h, c["bits"], c["black"], c["cfa"], seed * 64 + k, True, 0.0, True)
            target = preview_dimensions(w, h, 2560)
            srgb, hist = _outputs(*target)
            it = s["items"][k]
            it.mosaic = ctypes.cast(mosaic.data_ptr(), ctypes.POINTER(ctypes.c_uint16))
            it.row_stride = w
            it.sensor, it.detail = _sensor(c).to_c(), _capture(c).to_c()
            it.optics = _optics("poly5", w, h, rng).to_c()
            it.target_width, it.target_height = target
            for i in range(3):
                it.wb_gains[i] = AS_SHOT[i]
            for i in range(9):
                it.camera_to_rec2020[i] = CAMERA_TO_REC2020[i]
            it.color = _color("tone", rng).to_c()
            it.srgb_out = ctypes.cast(srgb.data_ptr(), ctypes.POINTER(ctypes.c_uint8))
            it.hist = ctypes.cast(hist.data_ptr(), ctypes.POINTER(ctypes.c_uint64))
            s["out"].append((srgb, hist))
            s["keep"].append(mosaic)
    elif case["kind"] == "edit":
        base = _base(case["width"], case["height"], seed)
        rgb = torch.from_numpy(base.download()).view(case["height"], case["width"], 3)
        s["base"] = rgb.permute(2, 0, 1).contiguous().cuda()
        base.release()
        s["color"] = _color(case["edit"], rng).to_c()
        s["srgb"] = torch.empty((case["height"], 3 * case["width"]), dtype=torch.uint8, device="cuda")
        s["hist"] = torch.empty(1024, dtype=torch.int64, device="cuda")
    else:
        s["base"] = _base(case["width"], case["height"], seed)
        s["color"] = _color(case["edit"], rng).to_c()
        spec = OutputSpec(format=case["format"], primaries=case["primaries"], policy=case["policy"],
                          dither=case["dither"], orientation=case["orientation"], headroom=case["headroom"])
        s["spec"] = spec.to_c()
        w, h = s["size"] = spec.dimensions(case["width"], case["height"])
        kind = {"srgb8": torch.uint8, "srgb16": torch.int16, "extended_f16": torch.float16,
                "extended_f32": torch.float32}[case["format"]]
        s["rows"] = torch.empty((h, 3 * w), dtype=kind, device="cuda")
        s["gamut"] = torch.empty(5, dtype=torch.int64, device="cuda")
        if case["file"] != "rows":
            s["depth"] = 16 if case["format"] == "srgb16" else 8
            room = _dev().lib.rd_png_bound(w, h, s["depth"], len(ICC), 0) if case["file"] == "png" else \
                _dev().lib.rd_jpeg_bound(w, h, len(ICC), 0)
            s["file"] = torch.zeros(int(room), dtype=torch.uint8, device="cuda")
            s["bytes"] = torch.empty(1, dtype=torch.int64, device="cuda")
            s["icc"] = np.frombuffer(ICC, dtype=np.uint8)
    return s


def run(s):
    case, dev = s["case"], _dev()
    lib = dev.lib
    if s["kind"] == "develop":
        m = s["mosaic"]
        if case["resident"]:
            source = GpuSensorProcessor(dev).develop_device(m.data_ptr(), case["width"], s["sensor"], s["capture"])
        else:
            source = GpuSensorProcessor(dev).develop(m.numpy().view(np.uint16), s["sensor"], s["capture"])
        base = GpuSpatialProcessor(dev).reduce_preview(source, s["optics"], s["target"], AS_SHOT, CAMERA_TO_REC2020)
        source.release()
        dev.check(lib.rd_render(dev.handle, base.handle, ctypes.byref(s["color"]),
                                ctypes.cast(s["srgb"].data_ptr(), ctypes.POINTER(ctypes.c_uint8)),
                                ctypes.cast(s["hist"].data_ptr(), ctypes.POINTER(ctypes.c_uint64)), None, None))
        base.release()
        return {"srgb": s["srgb"], "hist": s["hist"]}
    if s["kind"] == "batch":
        rc = lib.rd_develop_batch(0, s["items"], len(s["items"]), case["lanes"], None)
        if rc:
            raise RuntimeError(lib.rd_status_name(rc).decode())
        return s["out"]
    if s["kind"] == "edit":
        rc = lib.rd_render_device_noalloc(_ptr(s["base"]), case["width"], case["height"], ctypes.byref(s["color"]),
                                          _ptr(s["srgb"]), _ptr(s["hist"]),
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError(lib.rd_status_name(rc).decode())
        return {"srgb": s["srgb"], "hist": s["hist"]}
    dev.check(lib.rd_render_output_device(dev.handle, s["base"].handle, ctypes.byref(s["color"]),
                                          ctypes.byref(s["spec"]), _ptr(s["rows"]), None, _ptr(s["gamut"]), None))
    out = {"rows": s["rows"], "gamut": s["gamut"]}
    if case["file"] != "rows":
        w, h = s["size"]
        icc = s["icc"].ctypes.data_as(_ffi.U8P)
        if case["file"] == "png":
            dev.check(lib.rd_encode_png_device(dev.handle, _ptr(s["rows"]), w, h, 3 * w, s["depth"], icc, len(ICC),
                                               None, 0, _ptr(s["file"]), s["file"].numel(), _ptr(s["bytes"])))
        else:
            dev.check(lib.rd_encode_jpeg_device(dev.handle, _ptr(s["rows"]), w, h, 3 * w, case["quality"], icc,
                                                len(ICC), None, 0, _ptr(s["file"]), s["file"].numel(),
                                                _ptr(s["bytes"])))
        out["file"], out["bytes"] = s["file"], s["bytes"]
    return out


# ---------------------------------------------------------------- what a pass cannot do without
DEMOSAIC_FLOPS = {"amaze": 478, "rcd": 200, "mhc": 26, "bilinear": 8}  # per pixel
EDIT_FLOPS = {"exposure": 30, "plain": 60, "tone": 150, "full": 220}


def work(case):
    if case["kind"] == "batch":
        parts = [work(c) for c in _batch_images(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = case["width"] * case["height"]
    if case["kind"] == "develop":
        w, h = _sensor(case).crop_size
        n = w * h
        tw, th = preview_dimensions(w, h, case["long_edge"])
        per = DEMOSAIC_FLOPS[case["demosaic"]] + (6 if case["highlight"] == "opposed" else 2)
        if case["iterations"]:
            per += 58 * case["iterations"] + 60
        if case["lens"] != "none":
            per += 330
        return {"bytes": 2 * n + 3 * tw * th + 8192, "flops": per * n + EDIT_FLOPS[case["edit"]] * tw * th}
    if case["kind"] == "edit":
        return {"bytes": 15 * n + 8192, "flops": EDIT_FLOPS[case["edit"]] * n}
    out = {"srgb8": 3, "srgb16": 6, "extended_f16": 6, "extended_f32": 12}[case["format"]]
    flops = EDIT_FLOPS[case["edit"]] * n
    if case["file"] == "jpeg":
        flops += 3 * 32 * n
    return {"bytes": (12 + out) * n + (out * n // 2 if case["file"] != "rows" else 0), "flops": flops}


# CIE xy of the primaries and the white of Rec.2020, sRGB and Display P3 (ITU-R BT.2020, BT.709, SMPTE RP 431-2).
_XY = {"rec2020": ((0.708, 0.292), (0.170, 0.797), (0.131, 0.046)), "srgb": ((0.64, 0.33), (0.30, 0.60), (0.15, 0.06)),
       "display_p3": ((0.680, 0.320), (0.265, 0.690), (0.150, 0.060))}


def _to_xyz(space):
    xyz = np.array([[x / y, 1.0, (1.0 - x - y) / y] for x, y in _XY[space]], dtype=np.float64).T
    white = np.array([0.3127 / 0.3290, 1.0, (1.0 - 0.3127 - 0.3290) / 0.3290])
    return xyz * np.linalg.solve(xyz, white)


def exact(case, seed):
    """The linear export of a base that no adjustment but exposure touches, in 64 bits; the other outputs are bytes
    and whole numbers, or follow an adjustment chain that is defined in 32 bits."""
    if case["kind"] != "export" or case["edit"] != "exposure" or case["format"] != "extended_f32" or \
            case["policy"] != "clip":
        return None
    s = prepare(case, seed)
    base = torch.from_numpy(s["base"].download()).cuda().double().view(case["height"], case["width"], 3)
    m = torch.from_numpy(np.linalg.solve(_to_xyz(case["primaries"]), _to_xyz("rec2020"))).cuda()
    x = base * 2.0 ** float(s["color"].exposure_ev)
    x = (x @ m.T).clamp(0.0, case["headroom"])
    turn = {"normal": lambda t: t, "rotate180": lambda t: t.flip(0, 1), "transpose": lambda t: t.transpose(0, 1),
            "rotate90": lambda t: t.transpose(0, 1).flip(1)}[case["orientation"]]
    x = turn(x).contiguous()
    s["base"].release()
    return {"rows": x.view(x.shape[0], -1), "gamut": None}
