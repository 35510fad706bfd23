"""Section writers against a Python restatement of the streams, at the sizes
where their paths change: ANS batches of 128 tokens, reverse maps in shared
memory or in the code's own memory, maps that are no ANS code;
prefix chunks of 2048 tokens and codes too large for shared memory."""

import ctypes
import threading

import numpy as np
import pytest
import torch

from gjxl_b200 import _lib
from gjxl_b200.entropy import (ANS, PREFIX, EntropyCode, _sections, count_sections,
                               write_sections)
from tests.gpu_util import host

pytestmark = pytest.mark.gpu


def hybrid(v: int) -> tuple[int, int, int]:
    """(symbol, extra bits, count) under {4, 2, 0}."""
    if v < 16:
        return v, 0, 0
    n = v.bit_length() - 1
    return 16 + ((n - 4) << 2) + ((v - (1 << n)) >> (n - 2)), v & ((1 << (n - 2)) - 1), n - 2


def make_tokens(seed: int, n: int, contexts: int):
    rng = np.random.default_rng(seed)
    ctx = rng.integers(0, contexts, n).astype(np.uint16)
    values = (rng.geometric(0.2 + 0.7 * (ctx % 7) / 7.0) - 1).astype(np.uint32)
    large = rng.random(n) < 0.01
    values[large] = rng.integers(0, 1 << 20, int(large.sum()))
    return values, ctx


def make_tables(mode: int, seed: int, contexts: int, clusters: int) -> dict:
    rng = np.random.default_rng(seed)
    t = {"mode": mode, "context_count": contexts, "cluster_count": clusters,
         "context_map": (np.arange(contexts) % clusters).astype(np.uint8),
         "configs": np.tile(np.array([[4, 2, 0]], np.uint8), (clusters, 1))}
    if mode == ANS:
        freq = np.ones((clusters, 128), np.int64)
        for c in range(clusters):  # every frequency from 1 up to most of the table
            room = 4096 - 128
            for s in rng.permutation(16):
                f = int(rng.integers(0, room + 1)) if s else 0
                freq[c, s] += f
                room -= f
            freq[c, 0] += room
        padded = np.zeros((clusters, 256), np.int64)
        padded[:, :128] = freq
        starts = np.cumsum(padded, 1) - padded
        return t | {"frequencies": padded.astype(np.uint16),
                    "reverse_offsets": starts.astype(np.uint16),
                    "reverse_map": np.stack([rng.permutation(4096) for _ in range(clusters)])
                    .astype(np.uint16)}
    depths = rng.integers(1, 16, (clusters, 128)).astype(np.uint8)
    bits = (rng.integers(0, 1 << 15, (clusters, 128)) & ((1 << depths.astype(int)) - 1))
    degenerate = np.full(clusters, 128, np.uint16)
    return t | {"depths": depths, "bits": bits.astype(np.uint16), "degenerate": degenerate}


def ans_stream(t: dict, values, ctx) -> tuple[int, int]:
    """(bits, count): the final state, then the chunks in reverse push order."""
    state, stream, count = 0x130000, 0, 0
    for v, c in zip(values[::-1].tolist(), ctx[::-1].tolist()):
        cluster = t["context_map"][c]
        symbol, extra, n = hybrid(v)
        f = int(t["frequencies"][cluster, symbol])
        stream, count = (stream << n) | extra, count + n
        if (state >> 20) >= f:
            stream, count, state = (stream << 16) | (state & 0xFFFF), count + 16, state >> 16
        slot = t["reverse_map"][cluster, int(t["reverse_offsets"][cluster, symbol]) + state % f]
        state = (state // f << 12) + int(slot)
    return (stream << 32) | state, count + 32


def prefix_stream(t: dict, values, ctx) -> tuple[int, int]:
    parts, count = [], 0
    for v, c in zip(values.tolist(), ctx.tolist()):
        cluster = t["context_map"][c]
        symbol, extra, n = hybrid(v)
        d = int(t["depths"][cluster, symbol])
        parts.append(format((extra << d) | int(t["bits"][cluster, symbol]), f"0{d + n}b"))
        count += d + n
    return (int("".join(parts[::-1]), 2) if parts else 0), count


def check(t: dict, values, ctx, offsets):
    code = EntropyCode(t)
    got = write_sections(code, torch.from_numpy(offsets.astype(np.int32)).cuda(),
                         values=torch.from_numpy(values.view(np.int32)).cuda(),
                         contexts=torch.from_numpy(ctx.view(np.int16)).cuda())
    assert int(host(got["error"])[0]) == 0
    bits, packed = host(got["bit_counts"]), host(got["packed"]).tobytes()
    at = 0
    for s in range(offsets.size - 1):
        lo, hi = int(offsets[s]), int(offsets[s + 1])
        stream, count = (ans_stream if t["mode"] == ANS else prefix_stream)(
            t, values[lo:hi], ctx[lo:hi])
        assert int(bits[s]) == count, f"section {s}: bit count"
        size = (count + 7) // 8
        assert packed[at:at + size] == stream.to_bytes(size, "little"), f"section {s}"
        at += size
    assert host(got["byte_offsets"])[-1] == at
    counted = count_sections([code], torch.from_numpy(offsets.astype(np.int32)).cuda(),
                             values=torch.from_numpy(values.view(np.int32)).cuda(),
                             contexts=torch.from_numpy(ctx.view(np.int16)).cuda())
    assert int(host(counted["error"])[0]) == 0
    assert np.array_equal(host(counted["bit_counts"])[:, 0], bits)


SIZES = [0, 1, 2, 127, 128, 129, 255, 257, 1000, 3]


# 1 and 3 clusters: all maps staged; 30 and 90: some in the code only.
@pytest.mark.parametrize("clusters", [1, 3, 30, 90])
def test_ans_sections(cuda, clusters):
    offsets = np.concatenate([[0], np.cumsum(SIZES + [700] * 3)])
    values, ctx = make_tokens(clusters, int(offsets[-1]), 200)
    check(make_tables(ANS, 5 + clusters, 200, clusters), values, ctx, offsets)


def test_ans_context_map_beyond_shared_memory(cuda):
    offsets = np.array([0, 400, 1000])
    values, ctx = make_tokens(3, 1000, 6000)
    check(make_tables(ANS, 9, 6000, 20), values, ctx, offsets)


def test_ans_map_entry_outside_table_is_reported(cuda):
    """A used reverse-map entry past the 4096-entry table: error bit 2; an
    unused one changes nothing."""
    values, ctx = make_tokens(4, 500, 4)
    t = make_tables(ANS, 11, 4, 4)
    used = set()
    state = 0x130000
    for v, c in zip(values[::-1].tolist(), ctx[::-1].tolist()):
        cluster = int(t["context_map"][c])
        f = int(t["frequencies"][cluster, hybrid(v)[0]])
        if (state >> 20) >= f:
            state >>= 16
        at = int(t["reverse_offsets"][cluster, hybrid(v)[0]]) + state % f
        used.add((cluster, at))
        state = (state // f << 12) + int(t["reverse_map"][cluster, at])
    spare = next((0, i) for i in range(4096) if (0, i) not in used)
    t["reverse_map"][spare] = 5000
    check(t, values, ctx, np.array([0, 500]))
    t["reverse_map"][next(iter(used))] = 5000
    got = write_sections(EntropyCode(t), torch.tensor([0, 500], dtype=torch.int32).cuda(),
                         values=torch.from_numpy(values.view(np.int32)).cuda(),
                         contexts=torch.from_numpy(ctx.view(np.int16)).cuda())
    assert int(host(got["error"])[0]) & 4


# 250 clusters of 129 words exceed the staged size.
@pytest.mark.parametrize("clusters", [1, 40, 250])
def test_prefix_sections(cuda, clusters):
    offsets = np.concatenate([[0], np.cumsum([0, 1, 2047, 2048, 2049, 4100, 7])])
    values, ctx = make_tokens(50 + clusters, int(offsets[-1]), 300)
    check(make_tables(PREFIX, 60 + clusters, 300, clusters), values, ctx, offsets)


def small_offsets(seed: int, sections: int, most: int, first: list[int]) -> np.ndarray:
    sizes = np.random.default_rng(seed).integers(0, most + 1, sections)
    sizes[:len(first)] = first
    return np.concatenate([[0], np.cumsum(sizes)])


# The kernels for small sections, with a few that are not: fewer than 64 tokens
# a section (ANS); 400 sections of fewer than 1024 (prefix, chunks of 1024).
@pytest.mark.parametrize("clusters", [1, 40])
def test_small_sections(cuda, clusters):
    offsets = small_offsets(1, 150, 90, [0, 1, 128, 129, 400, 257])
    values, ctx = make_tokens(90 + clusters, int(offsets[-1]), 300)
    check(make_tables(ANS, 91 + clusters, 300, clusters), values, ctx, offsets)
    offsets = small_offsets(2, 400, 90, [0, 1, 1023, 1024, 1025, 2500])
    values, ctx = make_tokens(92 + clusters, int(offsets[-1]), 300)
    check(make_tables(PREFIX, 93 + clusters, 300, clusters), values, ctx, offsets)


def test_many_sections(cuda):
    """More sections than eight times the SMs: the small ANS kernel below 512 tokens a
    section, the small prefix kernel below 4096."""
    offsets = small_offsets(3, 1200, 130, [700])
    values, ctx = make_tokens(94, int(offsets[-1]), 300)
    check(make_tables(ANS, 95, 300, 40), values, ctx, offsets)
    check(make_tables(PREFIX, 96, 300, 40), values, ctx, offsets)


def test_ans_map_entry_outside_table_in_a_small_section(cuda):
    values, ctx = make_tokens(99, 50, 1)
    t = make_tables(ANS, 100, 1, 1)
    t["reverse_map"][:] = 65535
    got = write_sections(EntropyCode(t), torch.tensor([0, 50], dtype=torch.int32).cuda(),
                         values=torch.from_numpy(values.view(np.int32)).cuda(),
                         contexts=torch.from_numpy(ctx.view(np.int16)).cuda())
    assert int(host(got["error"])[0]) & 4


def test_ans_reverse_map_off_16_bytes(cuda):
    """A map that no 16-byte load may read: looked through and used in place."""
    offsets = np.array([0, 400, 1000])
    values, ctx = make_tokens(97, 1000, 30)
    t = make_tables(ANS, 98, 30, 3)
    expected = [ans_stream(t, values[a:b], ctx[a:b]) for a, b in ((0, 400), (400, 1000))]
    code = EntropyCode(t)
    shifted = torch.empty(3 * 4096 + 1, dtype=torch.int16, device="cuda")[1:]
    shifted.copy_(code._keep["reverse_map"].reshape(-1))
    code._keep["reverse_map"] = shifted
    got = write_sections(code, torch.from_numpy(offsets.astype(np.int32)).cuda(),
                         values=torch.from_numpy(values.view(np.int32)).cuda(),
                         contexts=torch.from_numpy(ctx.view(np.int16)).cuda())
    assert int(host(got["error"])[0]) == 0
    assert host(got["bit_counts"]).tolist() == [count for _, count in expected]
    data = host(got["packed"]).tobytes()
    size = (expected[0][1] + 7) // 8
    assert data[:size] == expected[0][0].to_bytes(size, "little")


@pytest.mark.parametrize("mode", [ANS, PREFIX])
def test_threads_with_codes_of_different_sizes(cuda, mode):
    """Two host threads, each with its own stream and code: neither call's
    shared-memory size may limit the other's launch."""
    work = []
    for clusters in (3, 150 if mode == PREFIX else 25):
        offsets = torch.tensor([0, 300, 1000], dtype=torch.int32).cuda()
        values, ctx = make_tokens(70 + clusters, 1000, 300)
        work.append((EntropyCode(make_tables(mode, 80 + clusters, 300, clusters)), offsets,
                     torch.from_numpy(values.view(np.int32)).cuda(),
                     torch.from_numpy(ctx.view(np.int16)).cuda()))
    want = [write_sections(code, o, values=v, contexts=c, tokens=1000)["packed"]
            for code, o, v, c in work]
    torch.cuda.synchronize()
    start, failed = threading.Barrier(2), []

    def run(k: int) -> None:
        code, o, v, c = work[k]
        stream = torch.cuda.Stream()
        try:
            with torch.cuda.stream(stream):
                # Most of the time inside the library, where threads run at once.
                struct, sections = code.struct(), _sections(o, v, c)
                bits = torch.zeros(2, dtype=torch.int64, device="cuda")
                error = torch.zeros(1, dtype=torch.int32, device="cuda")
                count = _lib.load().gjxl_b200_entropy_count_sections
                call = (ctypes.addressof(struct), 1, ctypes.addressof(sections), bits.data_ptr(),
                        error.data_ptr(), stream.cuda_stream)
                start.wait()
                for _ in range(20000):
                    assert count(*call) == 0, "launch failed"
                got = write_sections(code, o, values=v, contexts=c, tokens=1000)
                assert torch.equal(got["packed"], want[k])
                assert torch.equal(got["bit_counts"], bits) and int(error) == 0
        except Exception as exception:
            failed.append(exception)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed[0]
