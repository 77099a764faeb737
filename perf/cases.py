"""What the framework's users have it do, as cases that can be timed and compared.

A case is a dict of plain values.  Its "kind" says which public entry point
it goes through:

  cull      lh_cull_instances_noalloc: one view's instance cull + prefix sum
            with no allocation (engines under a fixed memory budget)
  frame     one frame of a main view and its four cascades; "api" is the
            call: "launches" (lh_frame), "graph" (lh_frame_graph) or
            "readback" (lh_frame_readback, the image in pinned host memory)
  batched   lh_frame_graph with probe views beside the main view
  train     lh_frame_graph_backward: a frame and the adjoint of its lighting
            (a differentiable renderer's step; gradients zeroed before)
  adjoint   lh_resolve_backward of the last frame (several losses of one
            frame; gradients zeroed before)
  display   lh_display_transform of the last frame through a caller's LUT

Scenes are the repository's seeded synthetic configurations (1: a few
spheres in a box, 2 and 3: clustered instances of eight meshes, 4: the
differentiable workload, 5: the stress workload); the seed places meshes,
materials and camera.  "view" is the configuration's own camera ("own") or
the same camera lifted over the scene and looking down ("above").  Launch
shapes are the library's defaults.
"""
import ctypes as C
import math

import numpy as np
import torch

import lighthugger_gb300 as lh

LUT = 48


def _case(kind, config, width, height, **more):
    case = {"kind": kind, "config": config, "width": width, "height": height, "shadow": 1024, "instances": 0,
            "detail": 1.0, "quantized": False, "alpha": False, "half": False, "view": "own", "api": "graph",
            "probes": 0}
    case.update(more)
    return case


def listed():
    return [
        # a fixed-budget engine's cull of the reference's instance capacity: latency alone
        dict(_case("cull", 5, 1920, 1080, instances=1024, detail=0.05), name="cull 1k"),
        # the same call over an open world, near the call's limit of 2^20 instances
        dict(_case("cull", 5, 1920, 1080, instances=700001, detail=0.05), name="cull 700k"),
        # a small scene rendered call by call: what launches and their gaps cost
        dict(_case("frame", 1, 1280, 720, api="launches"), name="frame 720p small scene"),
        # the reference's asset formats, alpha-clip foliage and RGBA16F, in a window of odd size
        dict(_case("frame", 2, 1279, 719, instances=1500, detail=0.4, quantized=True, alpha=True, half=True,
                   api="launches"), name="frame odd window, foliage"),
        # the benchmark's frame
        dict(_case("frame", 2, 1920, 1080), name="frame 1080p"),
        # the same scene from the air: many meshlets in view instead of a few walls
        dict(_case("frame", 2, 1920, 1080, view="above"), name="frame 1080p from above"),
        # an application that reads every frame back to the host
        dict(_case("frame", 2, 1920, 1080, api="readback"), name="frame 1080p read back"),
        # light probes or reflection captures beside the main view
        dict(_case("batched", 3, 1920, 1080, shadow=2048, probes=32), name="batched 32 probes"),
        # the stress workload: 100,000 instances at 4K
        dict(_case("frame", 5, 3840, 2160, instances=100000), name="frame 4K stress"),
        # a step of an inverse-rendering fit
        dict(_case("train", 4, 512, 512), name="train 512"),
        # the adjoint alone at a full frame's size
        dict(_case("adjoint", 2, 1920, 1080, view="above"), name="adjoint 1080p"),
        # presenting a 4K frame
        dict(_case("display", 2, 3840, 2160, view="above"), name="display 4K"),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["cull", "frame", "frame", "frame", "batched", "train", "adjoint", "display"])
    if kind == "cull":
        return _case("cull", 5, 1920, 1080, instances=_log(rng, 600, 1000000), detail=0.05)
    if kind == "batched":
        return _case("batched", 3, _log(rng, 320, 1920), _log(rng, 240, 1080), shadow=rng.choice([512, 1024, 2048]),
                     instances=_log(rng, 500, 4096), detail=round(rng.uniform(0.2, 1.0), 2), probes=_log(rng, 1, 32),
                     quantized=rng.random() < 0.25, alpha=rng.random() < 0.25)
    if kind == "train":
        return _case("train", 4, _log(rng, 128, 1024), _log(rng, 128, 1024), instances=_log(rng, 200, 2048),
                     detail=round(rng.uniform(0.3, 1.0), 2), alpha=rng.random() < 0.25)
    if kind == "adjoint":
        return _case("adjoint", rng.choice([2, 4]), _log(rng, 256, 1920), _log(rng, 256, 1080),
                     instances=_log(rng, 200, 2048), view=rng.choice(["own", "above"]))
    if kind == "display":
        return _case("display", 2, _log(rng, 320, 3840), _log(rng, 240, 2160), instances=_log(rng, 200, 2048),
                     half=rng.random() < 0.5, view="above")
    config = rng.choice([1, 2, 2, 2, 5])
    more = {"shadow": rng.choice([512, 1024, 1024, 2048]), "view": rng.choice(["own", "above"]),
            "api": rng.choice(["launches", "graph", "graph", "readback"]), "half": rng.random() < 0.33,
            "quantized": rng.random() < 0.33, "alpha": rng.random() < 0.33}
    if config == 1:
        return _case("frame", 1, _log(rng, 320, 1920), _log(rng, 240, 1080), instances=_log(rng, 16, 256),
                     **dict(more, view="own"))
    if config == 2:
        return _case("frame", 2, _log(rng, 320, 3840), _log(rng, 240, 2160), instances=_log(rng, 300, 6000),
                     detail=round(rng.uniform(0.2, 1.0), 2), **more)
    return _case("frame", 5, _log(rng, 1280, 3840), _log(rng, 720, 2160), instances=_log(rng, 10000, 100000),
                 detail=round(rng.uniform(0.3, 0.9), 2), **dict(more, view="own", alpha=False))


class _Device:
    """Device memory of the context as an array torch can view; keeps `owner`
    (the state that owns the memory) alive as long as the view is."""

    def __init__(self, address, shape, dtype, owner, strides=None):
        self.owner = owner
        self.__cuda_array_interface__ = {"version": 3, "shape": tuple(shape), "typestr": dtype,
                                         "data": (int(address), False), "strides": strides}


def _view(address, shape, dtype, owner, strides=None):
    return torch.as_tensor(_Device(address, shape, dtype, owner, strides), device="cuda")


def _scene(case, seed):
    return lh.Scene(case["config"], seed=1000003 + int(seed), width=case["width"], height=case["height"],
                    n_instances=case["instances"], n_probes=case["probes"], detail=case["detail"],
                    quantized=int(case["quantized"]), alpha_clip_materials=int(case["alpha"])).upload(0)


def _uniforms(case, scene):
    u = scene.uniforms
    if case["view"] == "own":
        return u
    f = lh.uniforms_fields(u)
    inverse = f["view_inverse"]  # columns: the camera looks along -z
    x, _, z = (float(v) for v in f["camera_pos"])
    yaw = math.atan2(-float(inverse[2][2]), -float(inverse[2][0]))
    return lh.make_uniforms((x, 40.0, z), yaw, -0.5, 60.0, case["width"], case["height"], scene.desc.n_instances)


class _Owner:
    """A scene and its renderer, destroyed together once nothing views them."""


def _renderer(case, scene, probes, n_probes):
    sizes = [lh.uniforms_fields(probes[p])["window_size"] for p in range(n_probes)]
    packed = [(w * h + 31) // 32 * 32 for w, h in sizes]
    d = scene.desc
    o = _Owner()
    o.scene, o.sizes, o.packed = scene, sizes, packed
    o.renderer = lh.Renderer(lh.Config(
        width=case["width"], height=case["height"], shadow_size=case["shadow"], max_instances=max(1024, d.n_instances),
        max_draws=min(d.total_meshlets + 1024, 1 << 23), max_big_triangles=1 << (23 if case["config"] == 5 else 21),
        max_probes=n_probes, max_probe_pixels=sum(packed), device=0,
        flags=lh.CONFIG_HDR_RGBA16F if case["half"] else 0))
    o.renderer.set_scene(scene)
    return o


def _frame_outputs(case, o, n_probes):
    """Everything a frame leaves behind: views of the context's own buffers."""
    r = o.renderer
    w, h, s, n = case["width"], case["height"], case["shadow"], 5 + n_probes
    lh._check(lh.lib().lh_get_outputs(r.ctx, C.byref(r.out)), "lh_get_outputs", r.ctx)
    f = r.out
    out = {
        "visibility": _view(f.visibility, (h, w), "<i8", o),
        "hdr": _view(f.hdr, (h, w, 4), "<f2" if case["half"] else "<f4", o),
        "shadow_maps": _view(f.shadow_maps, (4, s, s), "<f4", o),
        "cascades": _view(f.misc_storage, (196,), "<f4", o),
        "depth_range": _view(f.misc_storage + 784, (2,), "<i4", o),
        "instance_counters": _view(f.prefix_sums, (n,), "<i8", o, (f.prefix_sector_bytes,)),
        "draw_counts": _view(f.draw_calls, (n, 2), "<i4", o, (f.draw_call_section_bytes, 4)),
    }
    first = 0
    for p, ((pw, ph), size) in enumerate(zip(o.sizes, o.packed)):
        out["probe %02d" % p] = _view(f.probe_visibility + 8 * first, (ph, pw), "<i8", o)
        first += size
    return out


def _gradients(case, o, seed):
    """One flat gradient buffer, the tables lh_grad_targets points at, and the
    loss's gradient of the image."""
    from lighthugger_gb300.diff import _scene_records
    records, of_instance = _scene_records(o.scene)
    d = o.scene.desc
    vertices = {}
    for m in records:
        vertices[m.mesh] = m.vertices
    first, total = {}, 0
    for mesh in sorted(vertices):
        first[mesh] = total
        total += vertices[mesh]
    texels = [int(d.host_textures[i].width) * int(d.host_textures[i].height) for i in range(d.n_textures)]
    sizes = {"positions": 3 * total, "normals": 3 * total, "uvs": 2 * total, "factors": 4 * len(records),
             "textures": 4 * sum(texels), "light": 8}
    flat = torch.zeros(sum((n + 3) // 4 * 4 for n in sizes.values()), device="cuda")
    g, at = {}, 0
    for name, n in sizes.items():
        g[name] = flat[at:at + n]
        at += (n + 3) // 4 * 4
    rows = [[g["positions"].data_ptr() + 12 * first[m.mesh], g["normals"].data_ptr() + 12 * first[m.mesh],
             g["uvs"].data_ptr() + 8 * first[m.mesh], g["factors"].data_ptr() + 16 * k] for k, m in enumerate(records)]
    table = torch.from_numpy(np.array(rows, np.uint64).view(np.int64)).cuda()
    per_instance = torch.from_numpy(table.data_ptr() + 32 * of_instance.astype(np.int64)).cuda()
    starts = np.concatenate([[0], np.cumsum(texels)])[:-1].astype(np.int64)
    per_texture = torch.from_numpy(g["textures"].data_ptr() + 16 * starts).cuda()
    upstream = torch.randn(case["height"], case["width"], 4, device="cuda",
                           generator=torch.Generator(device="cuda").manual_seed(int(seed)))
    targets = lh.GradTargets(instance_grads=per_instance.data_ptr(), texture_grads=per_texture.data_ptr(),
                             light_dir=g["light"].data_ptr(), light_color=g["light"].data_ptr() + 16)
    return {"flat": flat, "named": g, "tables": (table, per_instance, per_texture), "upstream": upstream,
            "targets": targets}


def prepare(case, seed):
    scene = _scene(case, seed)
    u = _uniforms(case, scene)
    stream = torch.cuda.current_stream().cuda_stream
    s = {"kind": case["kind"], "api": case["api"], "uniforms": u, "stream": stream}
    if case["kind"] == "cull":
        n = scene.desc.n_instances
        s.update(scene=scene, n=n, sector=torch.zeros(1 + n, dtype=torch.int64, device="cuda"),
                 flags=torch.zeros(1, dtype=torch.int32, device="cuda"))
        return s
    probes, n_probes = scene.probe_uniforms()
    o = _renderer(case, scene, probes, n_probes)
    s.update(owner=o, probes=probes, n_probes=n_probes, outputs=_frame_outputs(case, o, n_probes))
    if case["api"] == "readback":
        shape, dtype = (case["height"], case["width"], 4), torch.float16 if case["half"] else torch.float32
        s.update(host=[torch.empty(shape, dtype=dtype, pin_memory=True) for _ in range(2)], turn=0)
    if case["kind"] in ("train", "adjoint"):
        s["gradients"] = _gradients(case, o, seed)
    if case["kind"] == "display":
        lut = torch.rand(LUT, LUT, LUT, 4, device="cuda",
                         generator=torch.Generator(device="cuda").manual_seed(int(seed)))
        s.update(lut=lut, image=torch.empty(case["height"], case["width"], 4, dtype=torch.uint8, device="cuda"))
    if case["kind"] in ("adjoint", "display"):
        o.renderer.frame(u, stream=stream)
    return s


def run(s):
    kind, u, stream = s["kind"], s["uniforms"], s["stream"]
    if kind == "cull":
        lh._check(lh.lib().lh_cull_instances_noalloc(s["scene"].desc.device_instances, s["n"], C.addressof(u),
                                                     s["sector"].data_ptr(), s["n"], s["flags"].data_ptr(), stream),
                  "lh_cull_instances_noalloc")
        return {"sector": s["sector"], "flags": s["flags"]}
    r = s["owner"].renderer
    if kind == "frame" and s["api"] == "launches":
        r.frame(u, stream=stream)
        return s["outputs"]
    if kind == "frame" and s["api"] == "readback":
        host = s["host"][s["turn"]]
        s["turn"] ^= 1
        r.frame_readback(u, host.data_ptr(), stream=stream)
        return dict(s["outputs"], hdr=host)
    if kind in ("frame", "batched"):
        r.frame_graph(u, s["probes"], s["n_probes"], stream=stream)
        return s["outputs"]
    if kind == "display":
        r.display_transform(s["image"].data_ptr(), s["lut"].data_ptr(), stream=stream)
        return {"image": s["image"]}
    g = s["gradients"]
    g["flat"].zero_()
    if kind == "train":
        r.frame_graph_backward(u, None, 0, g["upstream"].data_ptr(), g["targets"], stream=stream)
        return dict(s["outputs"], **g["named"])
    lh._check(lh.lib().lh_resolve_backward(r.ctx, g["upstream"].data_ptr(), C.byref(g["targets"]), stream),
              "lh_resolve_backward", r.ctx)
    return dict(g["named"])


def work(case):
    """Each input read once and each output written once.  Of a scene's
    geometry only the instance records are counted (which triangles have to
    be read depends on the view); operations are the cull's and the
    lighting's (about 100 an instance, 400 a pixel, and twice those again for
    the adjoint)."""
    pixels = case["width"] * case["height"]
    instances = case["instances"] or {1: 64, 2: 4096, 3: 4096, 4: 2048, 5: 100000}[case["config"]]
    if case["kind"] == "cull":
        return {"bytes": 112 * instances + 8 * instances // 2, "flops": 100 * instances}
    hdr = 8 if case["half"] else 16
    if case["kind"] == "display":
        return {"bytes": pixels * (hdr + 4) + 16 * LUT ** 3, "flops": 100 * pixels}
    if case["kind"] == "adjoint":
        return {"bytes": pixels * (8 + 16) + 4 * 4 * case["shadow"] ** 2, "flops": 1200 * pixels}
    probes = case["probes"] * 208 * 208  # sides spread over 64 .. 512 by their logarithm
    frame = {"bytes": 112 * instances + pixels * (8 + hdr) + 8 * probes + 4 * 4 * case["shadow"] ** 2,
             "flops": 400 * pixels + 100 * instances * (5 + case["probes"])}
    if case["kind"] == "train":
        frame["bytes"] += 16 * pixels
        frame["flops"] += 1200 * pixels
    return frame


def exact(case, seed):
    """None for every case.  The outputs are integers (visibility IDs, depth
    bits, counters, display bytes), or floats that hang on the float32
    decisions that made them -- the depth test between triangles, the shadow
    compare of a texel: a 64-bit evaluation of a frame takes other branches
    at edges, and a whole frame in plain numpy takes far longer than it may."""
    return None
