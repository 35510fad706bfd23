"""Performance cases: the calls a program makes into gjxl_b200, over the range
of sizes, efforts, precisions and forms it offers.

Every case is a dict of plain values; `kind` names the entry point:

  session      AnalysisSession.analyze: an image already on the device
  host         AnalysisSession.analyze_host: pinned host pixels in, results and
               token streams in pinned host memory out
  batch        BatchAnalyzer.analyze with host input: many uneven images
  stages       the provider-level calls of the front half, one after another
  butteraugli  Butteraugli.prepare and .compare of one image pair
  sections     entropy.write_sections: token streams into coded sections
  train        ProposalNetwork.train_step on one batch of tiles

The analysis restates its CPU counterpart to the bit (its floating-point
planes included), and its decisions, coefficients and tokens follow from
comparisons of those values, so every kind but `train` is compared exactly.
"""

from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from gjxl_b200 import _lib, stages
from gjxl_b200.batch import BatchAnalyzer
from gjxl_b200.entropy import ANS, PREFIX, EntropyCode, write_sections
from gjxl_b200.learned import QF_WEIGHT, ProposalNetwork
from gjxl_b200.session import AnalysisSession

AC_CONTEXTS = 4 * 495          # contexts of the default block-context map
CLUSTERS = 40                  # entropy-code clusters of the section cases


def listed() -> list[dict]:
    return [
        # A thumbnail: the smallest analysis in real use, where launches and
        # the serial stages' latency are all there is.
        {"name": "session_256", "kind": "session", "width": 256, "height": 256, "channels": 3,
         "effort": 7, "precision": 0, "distance": 1.0, "learned": False},
        # A web image of odd size with an alpha channel, at a lower effort and
        # a coarser distance.
        {"name": "session_odd_rgba", "kind": "session", "width": 1021, "height": 767,
         "channels": 4, "effort": 6, "precision": 0, "distance": 2.0, "learned": False},
        # A 12 MP photograph at the default effort: the headline workload.
        {"name": "session_12mp", "kind": "session", "width": 4032, "height": 3024,
         "channels": 3, "effort": 7, "precision": 0, "distance": 1.0, "learned": False},
        # A 24 MP photograph, fast costs, four field updates: the largest call.
        {"name": "session_24mp_fast", "kind": "session", "width": 6000, "height": 4000,
         "channels": 3, "effort": 9, "precision": 1, "distance": 1.0, "learned": False},
        # The learned form, with the shipped proposal network.
        {"name": "learned_2048", "kind": "session", "width": 2048, "height": 2048,
         "channels": 3, "effort": 7, "precision": 0, "distance": 1.0, "learned": True},
        # An encoder's whole call on host memory: copies and tokens included.
        {"name": "host_2048x1536", "kind": "host", "width": 2048, "height": 1536, "channels": 3,
         "effort": 7, "precision": 0, "distance": 1.0},
        # A service's batch of uneven uploads through concurrent lanes.
        {"name": "batch_12", "kind": "batch", "images": 12, "low": 256, "high": 1600,
         "layout": 7, "lanes": 4, "effort": 7},
        # Single providers called one by one by a host encoder, odd size.
        {"name": "stages_900x675", "kind": "stages", "width": 900, "height": 675,
         "distance": 1.0, "precision": 0},
        # Quality measurement of a decoded image against its original.
        {"name": "butteraugli_2048x1536", "kind": "butteraugli", "width": 2048, "height": 1536},
        # Entropy-coded AC sections of a 3 MP frame at distance 1, ANS.
        {"name": "sections_ans", "kind": "sections", "mode": ANS, "tokens": 1500000,
         "sections": 48},
        # The same with prefix codes, a 12 MP frame.
        {"name": "sections_prefix", "kind": "sections", "mode": PREFIX, "tokens": 6000000,
         "sections": 192},
        # One training step of the proposal network at its default batch.
        {"name": "train_256", "kind": "train", "tiles": 256},
    ]


def _log_uniform(rng, low: float, high: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _extent(rng, low: int, high: int, pixels: int) -> tuple[int, int]:
    """An image extent: log-uniform width, aspect ratio 0.5 to 2, any parity."""
    while True:
        w = _log_uniform(rng, low, high)
        h = int(round(w * 2.0 ** rng.uniform(-1.0, 1.0)))
        if low <= h <= high and w * h <= pixels:
            return w, h


def draw(rng) -> dict:
    kind = rng.choice(["session", "session", "session", "host", "batch", "stages",
                       "butteraugli", "sections", "train"])
    if kind == "session":
        w, h = _extent(rng, 64, 4096, 12_200_000)
        return {"kind": kind, "width": w, "height": h, "channels": rng.choice([3, 3, 4]),
                "effort": rng.choice([5, 6, 7, 7, 8, 9]), "precision": rng.choice([0, 0, 1]),
                "distance": round(rng.uniform(0.5, 3.0), 2),
                "learned": rng.random() < 0.2}
    if kind == "host":
        w, h = _extent(rng, 64, 3000, 6_000_000)
        return {"kind": kind, "width": w, "height": h, "channels": rng.choice([3, 4]),
                "effort": rng.choice([5, 6, 7, 8]), "precision": rng.choice([0, 1]),
                "distance": round(rng.uniform(0.5, 3.0), 2)}
    if kind == "batch":
        return {"kind": kind, "images": rng.randint(3, 12), "low": 256,
                "high": rng.randint(600, 1600), "layout": rng.randint(0, 10**6),
                "lanes": rng.choice([2, 4, 8]), "effort": rng.choice([6, 7])}
    if kind == "stages":
        w, h = _extent(rng, 64, 2500, 4_000_000)
        return {"kind": kind, "width": w, "height": h,
                "distance": round(rng.uniform(0.5, 3.0), 2), "precision": rng.choice([0, 1])}
    if kind == "butteraugli":
        w, h = _extent(rng, 64, 4096, 12_200_000)
        return {"kind": kind, "width": w, "height": h}
    if kind == "sections":
        tokens = _log_uniform(rng, 20_000, 4_000_000)
        return {"kind": kind, "mode": rng.choice([ANS, PREFIX]), "tokens": tokens,
                "sections": max(1, tokens // rng.randint(15_000, 60_000))}
    return {"kind": "train", "tiles": _log_uniform(rng, 16, 512)}


# ---------------------------------------------------------------- inputs


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _uniform(g: torch.Generator, low: float, high: float) -> float:
    return float(low + (high - low) * torch.rand((), generator=g, device="cuda",
                                                 dtype=torch.float64).item())


def _noise_planes(g: torch.Generator, planes: int, height: int, width: int,
                  alpha: float) -> torch.Tensor:
    """1/f^alpha noise (exponent of the power spectrum), about [0, 1]."""
    fy = torch.fft.fftfreq(height, device="cuda")[:, None]
    fx = torch.fft.rfftfreq(width, device="cuda")[None, :]
    f = torch.sqrt(fx * fx + fy * fy)
    f[0, 0] = 1.0
    amplitude = f ** (-alpha / 2.0)
    amplitude[0, 0] = 0.0
    out = []
    for _ in range(planes):
        re = torch.randn(amplitude.shape, generator=g, device="cuda")
        im = torch.randn(amplitude.shape, generator=g, device="cuda")
        plane = torch.fft.irfft2(torch.complex(re, im) * amplitude, s=(height, width))
        out.append((0.5 + plane / (5.0 * plane.std())).clamp(0.0, 1.0))
    return torch.stack(out, -1)


def _image(seed: int, width: int, height: int, channels: int) -> torch.Tensor:
    """(height, width, channels) uint8: colour noise of natural spectra with a
    gradient, soft blobs, hard-edged flat polygons and a little sensor noise,
    at a random saturation."""
    g = _generator(seed)
    image = _noise_planes(g, 3, height, width, _uniform(g, 1.5, 2.5))
    yy = torch.arange(height, device="cuda", dtype=torch.float32)[:, None]
    xx = torch.arange(width, device="cuda", dtype=torch.float32)[None, :]
    angle = _uniform(g, 0.0, 2.0 * math.pi)
    t = (math.cos(angle) * xx / width + math.sin(angle) * yy / height + 1.5) / 3.0
    colours = torch.rand((2, 3), generator=g, device="cuda")
    weight = _uniform(g, 0.2, 0.6)
    image = (1 - weight) * image + weight * (colours[0] + t[..., None] * (colours[1] - colours[0]))
    side = min(width, height)
    for _ in range(6):
        cx, cy = _uniform(g, 0, width), _uniform(g, 0, height)
        sigma = _uniform(g, 0.02, 0.2) * side
        blob = torch.exp(-0.5 * (((xx - cx) / sigma) ** 2 + ((yy - cy) / sigma) ** 2))
        blob = blob[..., None] * _uniform(g, 0.3, 0.9)
        image = image + blob * (torch.rand(3, generator=g, device="cuda") - image)
    for _ in range(12):
        cx, cy = _uniform(g, 0, width), _uniform(g, 0, height)
        radius = _uniform(g, 0.02, 0.2) * side
        inside = torch.ones((height, width), dtype=torch.bool, device="cuda")
        for k in range(4):
            a = _uniform(g, 0.0, 1.5) + k * math.pi / 2
            inside &= (xx - cx) * math.cos(a) + (yy - cy) * math.sin(a) < radius
        image = torch.where(inside[..., None], torch.rand(3, generator=g, device="cuda"), image)
    luma = image @ torch.tensor([0.2126, 0.7152, 0.0722], device="cuda")
    image = luma[..., None] + _uniform(g, 0.0, 1.0) * (image - luma[..., None])
    image = image * 255.0
    image = image + _uniform(g, 0.5, 2.0) * torch.randn(image.shape, generator=g, device="cuda")
    pixels = image.round().clamp(0, 255).to(torch.uint8)
    if channels == 4:
        alpha = torch.full((height, width, 1), 255, dtype=torch.uint8, device="cuda")
        pixels = torch.cat([pixels, alpha], -1)
    return pixels.contiguous()


def _srgb_to_linear(pixels: torch.Tensor, dtype=torch.float32) -> torch.Tensor:
    """(3, height, width) linear light of 8-bit sRGB."""
    v = pixels[..., :3].to(torch.float64) / 255.0
    v = torch.where(v <= 0.04045, v / 12.92, ((v + 0.055) / 1.055) ** 2.4)
    return v.permute(2, 0, 1).contiguous().to(dtype)


def _pad_columns(planes: torch.Tensor) -> torch.Tensor:
    """Row stride a multiple of four."""
    extra = -planes.shape[-1] % 4
    return torch.nn.functional.pad(planes, (0, extra)).contiguous()


def _tokens(seed: int, tokens: int, sections: int):
    """Token values, contexts and section offsets with the skew of AC streams:
    few frequent contexts, geometric values, uneven sections, rare large
    values."""
    g = _generator(seed)
    contexts = (torch.rand(tokens, generator=g, device="cuda") ** 3 * AC_CONTEXTS).to(torch.int64)
    contexts.clamp_(max=AC_CONTEXTS - 1)
    p = 0.25 + 0.7 * (contexts % 61).to(torch.float64) / 61.0
    u = torch.rand(tokens, generator=g, device="cuda", dtype=torch.float64).clamp_(min=1e-12)
    values = (torch.log(u) / torch.log1p(-p)).floor().to(torch.int64)
    large = torch.rand(tokens, generator=g, device="cuda") < 0.002
    values = torch.where(large, torch.randint(0, 1 << 12, (tokens,), generator=g, device="cuda"),
                         values)
    share = torch.exp(0.4 * torch.randn(sections, generator=g, device="cuda",
                                        dtype=torch.float64))
    ends = (torch.cumsum(share, 0) / share.sum() * tokens).round().to(torch.int64)
    ends[-1] = tokens
    offsets = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), ends])
    return values.to(torch.int32), contexts.to(torch.int16), offsets.to(torch.int32)


def _symbols(values: torch.Tensor) -> torch.Tensor:
    """Hybrid-uint symbols of the {4, 2, 0} configuration."""
    v = values.to(torch.int64)
    n = torch.floor(torch.log2(v.clamp(min=1).to(torch.float64))).to(torch.int64)
    coded = 16 + (n - 4) * 4 + ((v - (1 << n)) >> (n - 2).clamp(min=0))
    return torch.where(v < 16, v, coded)


def _entropy_tables(mode: int, values: torch.Tensor, contexts: torch.Tensor, seed: int) -> dict:
    """A code for the tokens: contexts in CLUSTERS equal runs, frequencies of
    the tokens' own symbols normalised to 4096 (ANS), or code lengths from
    them (prefix, at most 12 bits)."""
    context_map = (np.arange(AC_CONTEXTS) * CLUSTERS // AC_CONTEXTS).astype(np.uint8)
    cluster = torch.from_numpy(context_map.astype(np.int64)).cuda()[contexts.to(torch.int64)]
    counts = torch.bincount(cluster * 128 + _symbols(values), minlength=CLUSTERS * 128)
    counts = counts.reshape(CLUSTERS, 128).cpu().numpy().astype(np.float64)
    counts[:, 0] = np.maximum(counts[:, 0], 1.0)
    share = counts * 4096.0 / counts.sum(1, keepdims=True)
    freq = np.where(counts > 0, np.maximum(np.floor(share), 1.0), 0.0).astype(np.int64)
    freq[np.arange(CLUSTERS), freq.argmax(1)] += 4096 - freq.sum(1)
    tables = {"mode": mode, "context_count": AC_CONTEXTS, "cluster_count": CLUSTERS,
              "context_map": context_map,
              "configs": np.tile(np.array([[4, 2, 0]], np.uint8), (CLUSTERS, 1))}
    if mode == ANS:
        padded = np.zeros((CLUSTERS, 256), np.int64)
        padded[:, :128] = freq
        starts = np.cumsum(padded, 1) - padded
        rng = np.random.default_rng(seed)
        slots = np.stack([rng.permutation(4096) for _ in range(CLUSTERS)])
        return tables | {"frequencies": padded.astype(np.uint16),
                         "reverse_offsets": starts.astype(np.uint16),
                         "reverse_map": slots.astype(np.uint16)}
    depths = np.zeros((CLUSTERS, 128), np.uint8)
    bits = np.zeros((CLUSTERS, 128), np.uint16)
    degenerate = np.full(CLUSTERS, 128, np.uint16)
    for c in range(CLUSTERS):
        present = np.nonzero(freq[c])[0]
        if present.size == 1:
            degenerate[c] = present[0]
            continue
        lengths = np.maximum(1, np.ceil(np.log2(4096.0 / freq[c, present]))).astype(int)
        code, previous = 0, 0
        for k in np.argsort(lengths, kind="stable"):
            code <<= lengths[k] - previous
            previous = lengths[k]
            depths[c, present[k]] = previous
            bits[c, present[k]] = int(format(code, f"0{previous}b")[::-1], 2)
            code += 1
    return tables | {"depths": depths, "bits": bits, "degenerate": degenerate}


# ---------------------------------------------------------------- states


class _DeviceView:
    """Device memory a session owns, keeping the session alive."""

    def __init__(self, owner, pointer: int, shape, dtype):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(int(n) for n in shape),
                                         "typestr": np.dtype(dtype).str,
                                         "data": (int(pointer), False), "version": 3,
                                         "strides": None}


def _device_outputs(s: AnalysisSession) -> dict:
    """The results a device-resident encoder reads after analyze()."""
    o = s.outputs
    blocks, tiles = (o.blocks_y, o.blocks_x), (o.tiles_y, o.tiles_x)
    views = {
        "cells": (o.strategy_cells, blocks, np.uint8),
        "quant_field": (o.quant_field, blocks, np.float32),
        "raw_quant": (o.raw_quant_field, blocks, np.int32),
        "y_to_x": (o.y_to_x, tiles, np.int8),
        "y_to_b": (o.y_to_b, tiles, np.int8),
        "quantized_ac": (o.quantized_ac, (3, o.padded_height, o.padded_width), np.int32),
        "quantized_dc": (o.quantized_dc, (3,) + blocks, np.int32),
        "distance_map": (o.distance_map, (s.height, s.width), np.float32),
        "block_distance": (o.block_distance, blocks, np.float32),
        "score_history": (o.score_history, (o.iterations + 1,), np.float64),
        "pnorm_history": (o.pnorm_history, (o.iterations + 1,), np.float64),
        "quantizer": (o.quantizer_params, (2,), np.int32),
        "group_offsets": (o.group_offsets, (o.groups + 1,), np.int32),
        "token_histogram": (o.token_histogram, (AC_CONTEXTS, 128), np.int32),
        "dc_tokens": (o.dc_tokens, (3 * blocks[0] * blocks[1], 2), np.int32),
        "dc_group_info": (o.dc_group_info, (o.dc_groups, 5), np.int32),
        "dc_histogram": (o.dc_histogram, (45, 128), np.int32),
        "error": (o.device_error, (3,), np.int32),
    }
    return {k: torch.as_tensor(_DeviceView(s, *v), device="cuda") for k, v in views.items()}


def _host_view(owner, pointer: int, shape, dtype) -> np.ndarray:
    count = int(np.prod(shape))
    buffer = (ctypes.c_uint8 * (count * np.dtype(dtype).itemsize)).from_address(pointer)
    buffer.owner = owner
    return np.frombuffer(buffer, dtype, count).reshape(shape)


def _host_outputs(s: AnalysisSession, owner) -> dict:
    """The fixed-size pinned host results an encoder reads after
    analyze_host()."""
    o = s.outputs
    blocks = (o.blocks_y, o.blocks_x)
    views = {
        "cells": (o.host_strategy_cells, blocks, np.uint8),
        "raw_quant": (o.host_raw_quant_field, blocks, np.int32),
        "quantized_dc": (o.host_quantized_dc, (3,) + blocks, np.int32),
        "score_history": (o.host_score_history, (o.iterations + 1,), np.float64),
        "dc_tokens": (o.host_dc_tokens, (3 * blocks[0] * blocks[1], 2), np.uint32),
    }
    return {k: _host_view(owner, *v) for k, v in views.items()}


def _host_streams(s: AnalysisSession) -> dict:
    """The rest: maps, the field, and the token streams at their capacity."""
    o = s.outputs
    tiles = (o.tiles_y, o.tiles_x)
    tokens = _lib.load().gjxl_b200_ac_token_capacity(o.blocks_x, o.blocks_y)
    sizes = [ctypes.c_size_t() for _ in range(4)]
    _lib.call("gjxl_b200_dc_token_sizes", o.blocks_x, o.blocks_y,
              *[ctypes.addressof(v) for v in sizes])
    views = {
        "quant_field": (o.host_quant_field, (o.blocks_y, o.blocks_x), np.float32),
        "y_to_x": (o.host_y_to_x, tiles, np.int8),
        "y_to_b": (o.host_y_to_b, tiles, np.int8),
        "token_values": (o.host_token_values, (tokens,), np.uint32),
        "token_contexts": (o.host_token_contexts, (tokens,), np.uint16),
        "group_offsets": (o.host_group_offsets, (o.groups + 1,), np.uint32),
        "meta_tokens": (o.host_meta_tokens, (sizes[1].value, 2), np.uint32),
        "dc_group_info": (o.host_dc_group_info, (o.dc_groups, 5), np.uint32),
        "dc_histogram": (o.host_dc_histogram, (45, 128), np.uint32),
    }
    return {k: _host_view(s, *v) for k, v in views.items()}


def _batch_extents(case: dict) -> list[tuple[int, int, float]]:
    rng = np.random.default_rng(case["layout"])
    low, high = math.log(case["low"]), math.log(case["high"])
    out = []
    for _ in range(case["images"]):
        w = int(math.exp(rng.uniform(low, high)))
        h = int(np.clip(w * 2.0 ** rng.uniform(-1, 1), case["low"], case["high"]))
        out.append((w, h, float(rng.uniform(0.5, 3.0))))
    return out


def _pinned(pixels: torch.Tensor) -> torch.Tensor:
    host = torch.empty(pixels.shape, dtype=pixels.dtype, pin_memory=True)
    host.copy_(pixels)
    return host


def _prepare_session(case: dict, seed: int) -> dict:
    network = ProposalNetwork.load() if case["learned"] else None
    s = AnalysisSession(case["width"], case["height"], butteraugli_target=case["distance"],
                        effort=case["effort"], precision=case["precision"],
                        proposal_weights=network.params.data_ptr() if network else 0)
    s.network = network
    pixels = _image(seed, case["width"], case["height"], case["channels"])
    return {"session": s, "pixels": pixels, "outputs": _device_outputs(s)}


def _prepare_host(case: dict, seed: int) -> dict:
    s = AnalysisSession(case["width"], case["height"], butteraugli_target=case["distance"],
                        effort=case["effort"], precision=case["precision"])
    pixels = _pinned(_image(seed, case["width"], case["height"], case["channels"]))
    # A server's session has served a request before; past a pass's own tokens
    # the stream arrays hold nothing.
    s.analyze_host(np.zeros(tuple(pixels.shape), np.uint8),
                   torch.cuda.current_stream().cuda_stream)
    streams = _host_streams(s)
    for name in ("token_values", "token_contexts", "meta_tokens"):
        streams[name][...] = 0
    return {"session": s, "pixels": pixels, "outputs": _host_outputs(s, s) | streams}


def _prepare_batch(case: dict, seed: int) -> dict:
    extents = _batch_extents(case)
    pixels = [_pinned(_image(seed * 1000 + i, w, h, 3)) for i, (w, h, _) in enumerate(extents)]
    batch = BatchAnalyzer(case["lanes"], effort=case["effort"])
    batch.set_schedule(case["lanes"], True)
    requests = batch.requests([(p.data_ptr(), w, h, d)
                               for p, (w, h, d) in zip(pixels, extents)])
    return {"batch": batch, "pixels": pixels, "extents": extents, "requests": requests}


def _prepare_stages(case: dict, seed: int) -> dict:
    w, h = case["width"], case["height"]
    pw, ph = stages.padded_extent(w, h)
    tiles = ((ph + 63) // 64, (pw + 63) // 64)
    f32 = {"dtype": torch.float32, "device": "cuda"}
    return {
        "pixels": _image(seed, w, h, 3),
        "linear": torch.zeros((3, h, (w + 3) // 4 * 4), **f32),
        "opsin": torch.zeros((3, ph, pw), **f32),
        "pre": torch.zeros((3, ph, pw), **f32),
        "stats": torch.zeros(3, **f32),
        "quant": torch.zeros((ph // 8, pw // 8), **f32),
        "strategy_mask": torch.zeros((ph // 8, pw // 8), **f32),
        "pixel_mask": torch.zeros((ph, pw), **f32),
        "scratch": torch.empty(stages.initial_quant_scratch_bytes(pw, ph), dtype=torch.uint8,
                               device="cuda"),
        "y_to_x": torch.zeros(tiles, dtype=torch.int8, device="cuda"),
        "y_to_b": torch.zeros(tiles, dtype=torch.int8, device="cuda"),
        "costs": torch.empty(stages.ac_strategy_cost_bytes(pw, ph) // 4, **f32),
        "cells": torch.zeros((ph // 8, pw // 8), dtype=torch.uint8, device="cuda"),
        "error": torch.zeros(1, dtype=torch.int32, device="cuda"),
    }


def _prepare_butteraugli(case: dict, seed: int) -> dict:
    w, h = case["width"], case["height"]
    pixels = _image(seed, w, h, 3)
    g = _generator(seed + 1)
    # What a lossy coder does to an image: noise in proportion to a slowly
    # varying strength, and flat 8x8 blocks here and there.
    strength = _noise_planes(g, 1, h, w, 3.0) * 10.0
    changed = pixels + strength * torch.randn(pixels.shape, generator=g, device="cuda")
    small = torch.nn.functional.avg_pool2d(changed.permute(2, 0, 1)[None], 8, ceil_mode=True)
    flat = torch.repeat_interleave(torch.repeat_interleave(small[0], 8, 1), 8, 2)[:, :h, :w]
    pick = torch.rand((h // 8 + 1, w // 8 + 1), generator=g, device="cuda") < 0.1
    pick = pick.repeat_interleave(8, 0).repeat_interleave(8, 1)[:h, :w]
    changed = torch.where(pick[..., None], flat.permute(1, 2, 0), changed)
    changed = changed.round().clamp(0, 255).to(torch.uint8)
    return {
        "handle": stages.Butteraugli(w, h),
        "reference": _pad_columns(_srgb_to_linear(pixels)),
        "distorted": _pad_columns(_srgb_to_linear(changed)),
        "map": torch.zeros((h, w), dtype=torch.float32, device="cuda"),
        "score": torch.zeros(1, dtype=torch.float64, device="cuda"),
    }


def _prepare_sections(case: dict, seed: int) -> dict:
    values, contexts, offsets = _tokens(seed, case["tokens"], case["sections"])
    code = EntropyCode(_entropy_tables(case["mode"], values, contexts, seed))
    return {"code": code, "values": values, "contexts": contexts, "offsets": offsets,
            "tokens": case["tokens"]}


def _train_inputs(case: dict, seed: int):
    """Tiles of XYB with their log distance (BF16 bits), labels, targets."""
    tiles = case["tiles"]
    g = _generator(seed)
    y = torch.rand((tiles, 1, 1, 1), generator=g, device="cuda") * 0.6 + 0.1
    y = y + 0.05 * torch.randn((tiles, 80, 80, 1), generator=g, device="cuda")
    x = 0.01 * torch.randn((tiles, 80, 80, 1), generator=g, device="cuda")
    b = y + 0.03 * torch.randn((tiles, 80, 80, 1), generator=g, device="cuda")
    d = torch.log2(0.5 + 2.5 * torch.rand((tiles, 1, 1, 1), generator=g, device="cuda"))
    inputs = torch.cat([x, y, b, d.expand(tiles, 80, 80, 1)], -1).to(torch.bfloat16)
    searched = torch.tensor([0, 6, 7, 4, 10, 11, 5], device="cuda")
    pick = torch.randint(0, 7, (tiles, 64), generator=g, device="cuda")
    labels = searched[pick].to(torch.uint8)
    targets = 0.3 * torch.randn((tiles, 64), generator=g, device="cuda")
    weights = (torch.rand((tiles, 64), generator=g, device="cuda") < 0.97).to(torch.float32)
    return inputs.contiguous(), labels, targets, weights


def _prepare_train(case: dict, seed: int) -> dict:
    network = ProposalNetwork.load()
    network.ensure(case["tiles"])
    inputs, labels, targets, weights = _train_inputs(case, seed)
    return {"network": network, "initial": network.params.clone(),
            "inputs": inputs.view(torch.int16), "labels": labels, "targets": targets,
            "weights": weights, "tiles": case["tiles"]}


_PREPARE = {"session": _prepare_session, "host": _prepare_host, "batch": _prepare_batch,
            "stages": _prepare_stages, "butteraugli": _prepare_butteraugli,
            "sections": _prepare_sections, "train": _prepare_train}


def prepare(case: dict, seed: int) -> dict:
    return _PREPARE[case["kind"]](case, seed) | {"case": case}


# ---------------------------------------------------------------- passes


def _run_session(s: dict):
    c = s["case"]
    s["session"].analyze(s["pixels"].data_ptr(), c["width"] * c["channels"], c["channels"],
                         torch.cuda.current_stream().cuda_stream)
    return s["outputs"]


def _run_host(s: dict):
    s["session"].analyze_host(s["pixels"].numpy(), torch.cuda.current_stream().cuda_stream)
    return s["outputs"]


def _run_batch(s: dict):
    results, _ = s["batch"].analyze(s["requests"], host_input=True)
    return [_host_outputs(s["batch"].session(r, w, h), s["batch"])
            for r, (w, h, _) in zip(results, s["extents"])]


def _run_stages(s: dict):
    c = s["case"]
    w, h, d = c["width"], c["height"], c["distance"]
    pw, ph = stages.padded_extent(w, h)
    stages.prepare_input(s["pixels"], w, h, 3 * w, 3, s["linear"], s["opsin"],
                         device_error=s["error"])
    stages.matrix_scale_stats(s["opsin"], w, h, s["stats"])
    stages.initial_quant_field(s["opsin"], pw, ph, d, 1.0, s["quant"], s["strategy_mask"],
                               s["pixel_mask"], s["scratch"], s["error"])
    stages.gaborish_inverse(s["opsin"], s["pre"], pw, ph, device_error=s["error"])
    stages.initial_cfl(s["pre"], s["y_to_x"], s["y_to_b"])
    stages.ac_strategy_search(s["pre"], s["quant"], s["pixel_mask"], s["y_to_x"], s["y_to_b"],
                              s["costs"], s["cells"], d, device_error=s["error"],
                              precision=c["precision"])
    return {k: s[k] for k in ("linear", "opsin", "stats", "quant", "strategy_mask", "pixel_mask",
                              "pre", "y_to_x", "y_to_b", "cells", "error")}


def _run_butteraugli(s: dict):
    s["handle"].prepare(s["reference"])
    s["handle"].compare(s["distorted"], s["map"], s["score"])
    return {"map": s["map"], "score": s["score"]}


def _run_sections(s: dict):
    out = write_sections(s["code"], s["offsets"], values=s["values"], contexts=s["contexts"],
                         tokens=s["tokens"])
    return {k: out[k] for k in ("packed", "byte_offsets", "bit_counts", "error")}


def _run_train(s: dict):
    network, tiles = s["network"], s["tiles"]
    # The first step of a training run, so that every pass starts alike.
    network.params.copy_(s["initial"])
    network.m.zero_()
    network.v.zero_()
    network.step = 0
    network.inputs(tiles).copy_(s["inputs"])
    loss = network.train_step(tiles, s["labels"], s["targets"], s["weights"], 2e-3)
    return {"loss": loss, "grads": network.grads, "m": network.m, "v": network.v,
            "params": network.params}


_RUN = {"session": _run_session, "host": _run_host, "batch": _run_batch, "stages": _run_stages,
        "butteraugli": _run_butteraugli, "sections": _run_sections, "train": _run_train}


def run(state: dict):
    return _RUN[state["case"]["kind"]](state)


# ---------------------------------------------------------------- work

_UPDATES = {5: 0, 6: 1, 7: 2, 8: 3, 9: 4}
# Operations per pixel: the seven transform families' candidates (forward and
# inverse separable transforms of three channels), and one evaluation
# (reconstruction, loop filters, both scales of the distance's blurs and
# oriented line sums).
_SEARCH_OPS, _EVALUATION_OPS = 5800, 2500


def _analysis_work(pixels: int, channels: int, updates: int, learned: bool) -> dict:
    # In: packed pixels. Out: quantized AC and distance map (16 B/px), block
    # fields, about one 6-byte token per two pixels.
    share = 0.65 if learned else 1.0
    return {"bytes": pixels * (channels + 16 + 1 + 3),
            "flops": pixels * (_SEARCH_OPS * share + _EVALUATION_OPS * (updates + 1))}


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("session", "host"):
        learned = case.get("learned", False)
        return _analysis_work(case["width"] * case["height"], case["channels"],
                              1 if learned else _UPDATES[case["effort"]], learned)
    if kind == "batch":
        parts = [_analysis_work(w * h, 3, _UPDATES[case["effort"]], False)
                 for w, h, _ in _batch_extents(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "stages":
        # In: packed pixels. Out: linear, XYB and sharpened XYB, pixel mask.
        pixels = case["width"] * case["height"]
        return {"bytes": pixels * (3 + 40), "flops": pixels * (_SEARCH_OPS + 200)}
    if kind == "butteraugli":
        pixels = case["width"] * case["height"]
        return {"bytes": pixels * 28, "flops": pixels * 4000}
    if kind == "sections":
        # Six bytes read per token and about one byte of stream written.
        return {"bytes": case["tokens"] * 7, "flops": case["tokens"] * 10}
    # Multiply-adds of the four convolutions and the head; backward twice that.
    macs = 40 * 40 * 36 * 32 + 20 * 20 * 288 * 32 + 10 * 10 * 288 * 32 * 2 + 64 * 32 * 28
    return {"bytes": case["tiles"] * (80 * 80 * 8 + 64 * 9) + 4 * 30000,
            "flops": case["tiles"] * macs * 2 * 3}


# ---------------------------------------------------------------- comparison


def tolerance(case: dict):
    # The training step rounds weights and activations to BF16 and sums in 32
    # bits; every other result is a whole number or a restated 32-bit value.
    return {"rel": TRAIN_REL} if case["kind"] == "train" else "exact"


# A forward sum in another order moves a few activations to the next BF16
# value. Between the SIMT and the tensor-core forward, 16 to 512 tiles, the
# gradients differed by up to 8e-4 (their squares 1.1e-3); about four times.
TRAIN_REL = 4e-3


def exact(case: dict, seed: int):
    """64-bit values of the training step and of the stages that are plain
    formulas. The other kinds' results are decisions, coefficients and tokens,
    or long chains of restated 32-bit operations that are compared exactly."""
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "stages":
        return _exact_stages(case, seed)
    return None


def _exact_train(case: dict, seed: int) -> dict:
    """Loss and gradients in 64 bits from the BF16 inputs: unrounded weights
    and activations."""
    inputs, labels, targets, weights = _train_inputs(case, seed)
    flat = ProposalNetwork.load().params.to(torch.float64).requires_grad_(True)
    x = inputs.to(torch.float64).permute(0, 3, 1, 2)
    offset = 0
    for cin, out_size, stride in ((4, 40, 2), (32, 20, 2), (32, 10, 2), (32, 10, 1)):
        n = 32 * 9 * cin
        w = flat[offset:offset + n].reshape(32, 3, 3, cin).permute(0, 3, 1, 2)
        bias = flat[offset + n:offset + n + 32]
        offset += n + 32
        x = torch.nn.functional.pad(x, (1, 1, 1, 1))
        patches = torch.nn.functional.unfold(x, 3, stride=stride)
        size = (x.shape[-1] - 3) // stride + 1
        x = torch.einsum("ok,nkp->nop", w.reshape(32, -1), patches) + bias[:, None]
        x = torch.relu(x).reshape(x.shape[0], 32, size, size)[:, :, :out_size, :out_size]
    head_w = flat[offset:offset + 28 * 32].reshape(28, 32)
    head_b = flat[offset + 28 * 32:offset + 28 * 33]
    centre = x[:, :, 1:9, 1:9].permute(0, 2, 3, 1).reshape(x.shape[0], 64, 32)
    head = centre @ head_w.T + head_b
    entropy = torch.nn.functional.cross_entropy(head[..., :27].reshape(-1, 27),
                                                labels.reshape(-1).long(), reduction="none")
    error = head[..., 27] - targets
    loss = (weights * (entropy.reshape(error.shape) + QF_WEIGHT * error * error)).mean()
    loss.backward()
    # The first step's weights move by the gradients' signs alone, which these
    # values do not settle where a gradient is about zero.
    return {"loss": loss.detach().reshape(1), "grads": flat.grad, "m": 0.1 * flat.grad,
            "v": 0.001 * flat.grad ** 2, "params": None}


# Opsin absorbance and its bias, and the normalised 5x5 sharpening kernel that
# undoes the decoder's smoothing.
_OPSIN = ((0.30, 0.622, 0.078), (0.23, 0.692, 0.078),
          (0.24342268924547819, 0.20476744424496821, 0.55180986650955360))
_OPSIN_BIAS = 0.0037930732552754493


def _exact_stages(case: dict, seed: int) -> dict:
    w, h = case["width"], case["height"]
    pw, ph = stages.padded_extent(w, h)
    linear = _srgb_to_linear(_image(seed, w, h, 3), torch.float64)
    mixed = torch.einsum("oc,chw->ohw", torch.tensor(_OPSIN, dtype=torch.float64, device="cuda"),
                         linear) + _OPSIN_BIAS
    gamma = mixed ** (1.0 / 3.0) - _OPSIN_BIAS ** (1.0 / 3.0)
    opsin = torch.stack([(gamma[0] - gamma[1]) / 2, (gamma[0] + gamma[1]) / 2, gamma[2]])
    opsin = torch.nn.functional.pad(opsin[None], (0, pw - w, 0, ph - h), mode="replicate")[0]
    return {"linear": _pad_columns(linear), "opsin": opsin} | {
        k: None for k in ("stats", "quant", "strategy_mask", "pixel_mask", "pre", "y_to_x",
                          "y_to_b", "cells", "error")}
