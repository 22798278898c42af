"""The rendering work this backend is timed on: one pass is one public call sequence on one scene.

A case names a scene generator of `blend2d_gb300.scenes` with its size, how the frame is run and
where its pixels go:

  entry  "frame"   Context.begin / submit_stream / end: record, upload, render (what an application
                   or a request handler does for every frame);
         "batch"   Runtime.render_batch over many canvases;
         "replay"  Runtime.replay of the frame kept on the device (inputs resident there).
  target "device"  a CUDA tensor the frame is drawn into;
         "host"    a page-locked host image it is read back into.
  graph  frames run as launches of one captured graph (LaunchConfig.graph_frames), as a program
         that renders frame after frame of a like size sets it.

Every scene begins with a fill of the whole canvas, so a pass gives the same pixels each time. The
pixels are whole numbers, the same whatever computes them.
"""
import math

import numpy as np
import torch

import blend2d_gb300 as bg
from blend2d_gb300 import scenes


def _case(name, scene, width, height, count, entry="frame", target="device", graph=False, canvases=1):
    case = {"scene": scene, "width": width, "height": height, "count": count, "entry": entry,
            "target": target, "graph": graph, "canvases": canvases}
    return {"name": name, **case} if name else case


def listed():
    return [
        # An icon or thumbnail: the smallest call a program makes, all launches and latency.
        _case("icon_64", "mixed", 64, 64, 12),
        # What a render server hands a worker: a batch of requests of uneven sizes (up to
        # width x height, up to `count` paths each), read back to the host.
        _case("serving_batch", "serving", 1024, 1024, 2000, entry="batch", target="host", canvases=32),
        # Plain polygons in solid colours on a small canvas, frame after frame.
        _case("polygons_512", "polygons", 512, 512, 2000, graph=True),
        # An application window of odd size: boxes, rectangles, polygons and paths in every style,
        # with transforms and alphas, into an XRGB32 image on the host.
        _case("ui_xrgb_1023x767", "ui_xrgb", 1023, 767, 900, target="host", graph=True),
        # Shapes drawn into an 8-bit mask.
        _case("mask_a8_1281x719", "mask_a8", 1281, 719, 600),
        # Image composition: aligned, fractional and scaled blits, nearest and bilinear.
        _case("blits_1280x720", "blits", 1280, 720, 1500),
        # Curved paths with dithered gradients, the high-quality gradient option.
        _case("dither_1600x900", "curves_dither", 1600, 900, 4000),
        # The curves-and-gradients workload at full size with its inputs on the device.
        _case("curves_1080p", "curves", 1920, 1080, 20000, entry="replay"),
        # Affine image patterns on the largest canvas.
        _case("patterns_4096", "patterns", 4096, 4096, 20000),
        # Stroked curves with every kind of join and cap.
        _case("strokes_1080p", "strokes", 1920, 1080, 10000),
        # The largest request a server takes: 4096 x 4096 with 20,000 mixed paths.
        _case("request_4096", "mixed", 4096, 4096, 20000),
        # The batched workload: canvases of 32 to 2048 px a side with 10 to 5,000 paths, one
        # pipeline for all of them, inputs on the device.
        _case("batch_512", "batch", 2048, 2048, 5000, entry="replay", canvases=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    scene = rng.choice(["mixed", "mixed", "serving", "polygons", "ui_xrgb", "mask_a8", "blits", "shapes",
                        "curves_dither", "curves", "patterns", "strokes", "batch"])
    graph = rng.random() < 0.4
    target = rng.choice(["device", "host"])
    if scene == "serving":
        return _case(None, scene, 1024, 1024, _log(rng, 64, 2000), "batch", "host", graph, _log(rng, 2, 32))
    if scene == "batch":
        return _case(None, scene, 2048, 2048, 5000, rng.choice(["batch", "replay"]), "device", graph,
                     _log(rng, 8, 256))
    if scene == "mixed":
        side = _log(rng, 64, 4096)
        return _case(None, scene, side, side, _log(rng, 1, 16000), "frame", target, graph)
    if scene in ("curves", "curves_dither", "strokes"):
        most = 16000 if scene == "curves" else 5000
        # strokes are sized by a pass of their own before each upload: those frames never run as graphs
        return _case(None, scene, _log(rng, 320, 1920), _log(rng, 200, 1080), _log(rng, 50, most),
                     rng.choice(["frame", "replay"]), "device", graph and scene != "strokes")
    if scene == "patterns":
        side = _log(rng, 512, 4096)
        return _case(None, scene, side, side - rng.randrange(1, 60), _log(rng, 20, 10000), "frame", target, graph)
    if scene == "polygons":
        return _case(None, scene, _log(rng, 128, 2048), _log(rng, 128, 2048), _log(rng, 50, 8000), "frame", target,
                     graph)
    return _case(None, scene, _log(rng, 130, 1920), _log(rng, 100, 1080), _log(rng, 20, 1500), "frame", target, graph)


def _specs(case):
    """(width, height, paths) of a case's canvases: the sizes of a batch are the case's, whatever its inputs."""
    w, h, n, k = case["width"], case["height"], case["count"], case["canvases"]
    if case["scene"] == "serving":
        return [(s, s, p) for s, p in scenes.serving_request_specs(5, k, max_side=w, max_paths=n)]
    if case["scene"] == "batch":
        return scenes.batch_canvas_specs(4, k, max_side=w, max_paths=n)
    return [(w, h, n)]


def _streams(case, seed):
    scene, w, h, n = case["scene"], case["width"], case["height"], case["count"]
    if scene in ("mixed", "serving", "batch"):
        made = [scenes._mixed_canvas(np.random.Generator(np.random.PCG64([seed, i])), *spec)
                for i, spec in enumerate(_specs(case))]
    elif scene == "polygons":
        made = [scenes.polygons(seed, w, h, n)]
    elif scene == "ui_xrgb":
        made = [scenes.random_mix(seed, w, h, n, format=scenes.FORMAT_XRGB32)]
    elif scene == "mask_a8":
        made = [scenes.random_mix(seed, w, h, n, format=scenes.FORMAT_A8,
                                  commands=("box_d", "polygon", "path_quad", "path_cubic"))]
    elif scene == "blits":
        made = [scenes.blits(seed, w, h, n)]
    elif scene == "shapes":
        made = [scenes.shapes(seed, w, h, n)]
    elif scene in ("curves", "curves_dither"):
        made = [scenes.curves(seed, w, h, n, dither=scene == "curves_dither")]
    elif scene == "patterns":
        made = [scenes.patterns(seed, w, h, n)]
    else:
        made = [scenes.stroked_paths(seed, w, h, n)]
    return [sw.to_bytes() for sw in made]


def _canvases(streams, target):
    """One buffer with a canvas for each stream, every canvas at a 256-byte boundary, and the canvases."""
    a8 = bg.stream_format(streams[0]) == bg.FORMAT_A8
    align = 256 if a8 else 64                  # pixels
    sizes = [bg.stream_size(s) for s in streams]
    first, end = [], 0
    for w, h in sizes:
        first.append(end)
        end += -(-w * h // align) * align
    dtype = torch.uint8 if a8 else torch.int32
    pool = torch.zeros(end, dtype=dtype, device="cuda") if target == "device" else torch.zeros(end, dtype=dtype).pin_memory()
    return pool, [pool[o:o + w * h].view(h, w) for o, (w, h) in zip(first, sizes)]


def prepare(case, seed):
    streams = _streams(case, int(seed))
    pool, targets = _canvases(streams, case["target"])
    torch.cuda.synchronize()                   # the runtime's stream does not wait for torch's fills
    rt = bg.Runtime(0)
    config = rt.launch_config()
    config.graph_frames = int(case["graph"])
    rt.set_launch_config(config)
    state = {"case": case, "streams": streams, "targets": targets, "pool": pool, "runtime": rt}
    if case["entry"] == "frame" or len(streams) == 1:
        state["context"] = bg.Context(rt)
        state["format"] = bg.stream_format(streams[0])
    if case["entry"] == "replay":
        _render(state)                         # the frame the runtime keeps on the device
    return state


def _render(state):
    if "context" in state:
        ctx = state["context"]
        ctx.begin(state["targets"][0], state["format"])
        ctx.submit_stream(state["streams"][0])
        ctx.end()
    else:
        state["runtime"].render_batch(state["streams"], state["targets"])


def run(state):
    if state["case"]["entry"] == "replay":
        state["runtime"].replay()
        state["runtime"].synchronize()         # its result and its errors are this call's
    else:
        _render(state)
    return state["pool"]


# Bytes of one drawing record of each scene (its style, options and geometry, on average) and the
# pixels it covers: sides log-uniform in 8..256 px have a mean square of 9,400 px, about 0.4 of it
# inside the path and 0.8 of that on the canvas.
_RECORD = {"mixed": (460, 3000), "serving": (460, 3000), "batch": (460, 3000), "polygons": (192, 1500),
           "ui_xrgb": (200, None), "mask_a8": (200, None), "blits": (100, 3000), "shapes": (128, 3000),
           "curves": (680, 3000), "curves_dither": (680, 3000), "patterns": (240, 55000), "strokes": (610, 2000)}
_PIXEL_OPS = 24          # SrcOver of four channels: three products and sums each


def work(case):
    record, covered = _RECORD[case["scene"]]
    bpp = 1 if case["scene"] == "mask_a8" else 4
    size = flops = 0
    for w, h, n in _specs(case):
        size += n * record + w * h * bpp
        flops += n * (w * h / 12 if covered is None else min(covered, w * h)) * _PIXEL_OPS
    return {"bytes": size, "flops": flops}


def exact(case, seed):
    """Pixels are whole numbers: every correct renderer gives the same ones."""
    return None
