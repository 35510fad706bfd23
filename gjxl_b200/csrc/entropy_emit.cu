// Entropy-coded sections on the device: every section's token stream written
// with a prebuilt ANS or prefix code, bit for bit as the reference's CPU
// writers write it, and the exact token-bit counts its rate search compares.
//
// ANS (src/codestream/ans.cpp:1700-1770, AnsReverseBits in
// src/codestream/ans_reverse_bits_internal.h): the tokens are encoded last to
// first from the state 0x13 << 16; each token pushes its hybrid-uint extra
// bits, then, when (state >> 20) >= frequency, the low 16 state bits, and the
// state becomes (state / f << 12) + reverse_map[offset + state % f]. The
// stream is the final 32-bit state followed by the pushed chunks in reverse
// push order. Two sections per CTA, four warps each: two producer warps turn
// batches of tokens into encoder records (hybrid-uint extra bits, frequency,
// exact division factor, reverse-map offset), one thread runs the state
// recurrence, which is serial by the format, over the previous batch, and an
// emitter warp places the bits of the batch before that from the top of the
// section's slot downwards; the CTA then shifts the finished stream to the
// slot's first bit. Bound: the latency of one recurrence step times the
// largest section's tokens.
//
// Prefix (src/codestream/entropy.cpp:1173,2294): every token is its code
// bits followed by its extra bits, in token order; the CTA scans the token
// lengths and ORs the tokens into a shared-memory window of whole words.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "host_util.h"

namespace gjxl_b200 {
namespace {

constexpr uint32_t kAnsLogTable = 12;                 // 4096-entry tables
constexpr uint32_t kAnsTable = 1u << kAnsLogTable;
constexpr uint32_t kAnsInitialState = 0x13u << 16;    // signature << 16
constexpr uint32_t kAnsSymbols = 256;
constexpr uint32_t kPrefixSymbols = 128;
constexpr uint32_t kAnsTokenBits = 47;     // <= 31 extra bits + one 16-bit chunk
constexpr uint32_t kPrefixTokenBits = 46;  // <= 15 code bits + 31 extra bits
constexpr int kMaxCodes = 8;

// Two sections per CTA, each with four warps: one thread running the
// recurrence, two warps building encoder records and a warp placing the bits;
// both sections share the CTA's staged reverse maps.
constexpr int kAnsPairs = 2;
constexpr int kSectionThreads = 128;
constexpr int kAnsThreads = kSectionThreads * kAnsPairs;
constexpr uint32_t kAnsContexts = 4096;  // largest context map kept in shared memory
constexpr uint32_t kMaxHotClusters = 32;
constexpr int kAnsBatch = 128;    // tokens per record batch
constexpr int kPrefixPerThread = 4;
constexpr int kPrefixThreads = 512;
constexpr int kPrefixSmallThreads = 256;  // for small sections

struct Code {
  int mode;
  uint32_t context_count, cluster_count;
  const uint8_t* context_map;
  const uint8_t* uint_configs;
  const uint8_t* prefix_depths;
  const uint16_t* prefix_bits;
  const uint16_t* prefix_degenerate;
  const uint16_t* frequencies;
  const uint16_t* reverse_offsets;
  const uint16_t* reverse_map;
};

struct Tokens {
  const uint2* pairs;
  const uint32_t* values;
  const uint16_t* contexts;
  const uint32_t* offsets;
  uint32_t count;
  uint32_t capacity;  // tokens in the arrays
};

struct EmitParams {
  Code code;
  Tokens tokens;
  uint64_t* slots;        // write mode: section slots; count mode: unused
  size_t slot_capacity;   // words
  uint64_t* bit_counts;   // [section * stride + column]
  uint32_t stride, column;
  uint32_t hot_clusters;  // ANS: reverse maps staged in shared memory
  uint32_t* error;
};

__host__ __device__ __forceinline__ uint32_t TokenBits(int mode) {
  return mode == GJXL_B200_ENTROPY_ANS ? kAnsTokenBits : kPrefixTokenBits;
}

// First word of section s's slot: ceil(B * offset / 64) + 2 s.
__host__ __device__ __forceinline__ uint64_t SlotStart(uint64_t offset, uint64_t s, uint32_t b) {
  return (b * offset + 63) / 64 + 2 * s;
}

__device__ __forceinline__ void FetchToken(const Tokens& t, uint32_t i, uint32_t* context,
                                           uint32_t* value) {
  if (t.pairs != nullptr) {
    const uint2 p = t.pairs[i];
    *context = p.x;
    *value = p.y;
  } else {
    *context = t.contexts[i];
    *value = t.values[i];
  }
}

struct HybridToken {
  uint32_t symbol, extra, count;
};

// JPEG XL's hybrid-uint split of `value` under {split_exponent, msb, lsb}:
// values below 2^split are their own symbol; larger ones keep their
// exponent, `msb` bits below the leading one and the lowest `lsb` bits in
// the symbol, the rest as raw extra bits (EncodeHybridUintValidated,
// src/codestream/entropy_internal.h:31).
__device__ __forceinline__ HybridToken EncodeHybrid(uint32_t value, uint32_t split,
                                                    uint32_t msb, uint32_t lsb) {
  HybridToken h;
  if (value < (1u << split)) {
    h.symbol = value;
    h.extra = 0;
    h.count = 0;
    return h;
  }
  const uint32_t exponent = 31u - static_cast<uint32_t>(__clz(value));
  const uint32_t mantissa = value - (1u << exponent);
  h.symbol = (1u << split) + ((exponent - split) << (msb + lsb)) +
             ((mantissa >> (exponent - msb)) << lsb) + (mantissa & ((1u << lsb) - 1u));
  h.count = exponent - msb - lsb;
  h.extra = static_cast<uint32_t>((value >> lsb) & ((1ull << h.count) - 1ull));
  return h;
}

// The cluster and hybrid-uint token of one stream token under `code`;
// false for a context outside the map, a cluster outside the code or an
// invalid configuration (the reference's InvalidArgument).
__device__ __forceinline__ bool ClusterToken(const Code& code, uint32_t context, uint32_t value,
                                             uint32_t* cluster, HybridToken* h) {
  if (context >= code.context_count) return false;
  *cluster = code.context_map[context];
  if (*cluster >= code.cluster_count) return false;
  const uint8_t* config = code.uint_configs + 3 * *cluster;
  const uint32_t split = config[0], msb = config[1], lsb = config[2];
  if (split > 15 || msb > split || lsb > split - msb) return false;
  *h = EncodeHybrid(value, split, msb, lsb);
  return true;
}

// One cluster's configuration in a word: split, msb, lsb, and whether they
// are valid.
__device__ __forceinline__ uint32_t PackedConfig(const Code& code, uint32_t cluster) {
  const uint8_t* config = code.uint_configs + 3 * cluster;
  const uint32_t split = config[0], msb = config[1], lsb = config[2];
  const bool valid = split <= 15 && msb <= split && lsb <= split - msb;
  return split | msb << 8 | lsb << 16 | (valid ? 1u << 24 : 0u);
}

// ORs `value` (up to 64 bits) into little-endian bits at `at` of shared
// words, in 32-bit halves: 64-bit shared atomics retry while neighbours change
// the same word.
__device__ __forceinline__ void OrBits(unsigned long long* window, uint64_t at, uint64_t value) {
  uint32_t* words = reinterpret_cast<uint32_t*>(window) + (at >> 5);
  const int shift = static_cast<int>(at & 31);
  const uint32_t low = static_cast<uint32_t>(value << shift);
  const uint64_t rest = value >> (32 - shift);
  const uint32_t middle = static_cast<uint32_t>(rest), high = static_cast<uint32_t>(rest >> 32);
  if (low != 0) atomicOr(words, low);
  if (middle != 0) atomicOr(words + 1, middle);
  if (high != 0) atomicOr(words + 2, high);
}

// Section bounds with the checks every kernel makes: false (and the error
// bit) for decreasing offsets, tokens past the arrays' capacity or a slot
// beyond the buffer.
__device__ __forceinline__ bool SectionBounds(const EmitParams& p, uint32_t s, bool write,
                                              uint32_t* begin, uint32_t* end,
                                              uint64_t* slot_begin, uint64_t* slot_end,
                                              bool report) {
  *begin = p.tokens.offsets[s];
  *end = p.tokens.offsets[s + 1];
  const uint32_t b = TokenBits(p.code.mode);
  *slot_begin = SlotStart(*begin, s, b);
  *slot_end = SlotStart(*end, s + 1, b);
  const bool ok = *end >= *begin && *end <= p.tokens.capacity &&
                  (!write || *slot_end <= p.slot_capacity);
  if (!ok && report) {
    RaiseError(p.error, kErrorRange);
    p.bit_counts[static_cast<size_t>(s) * p.stride + p.column] = 0;
  }
  return ok;
}

// ---------------------------------------------------------------- ANS ----

// Exact division of a state below f * 2^20 by a frequency f in 1..4096 with
// one 32 x 32-bit multiply-add: state / f = ((state * factor + addend) >> 32)
// >> shift, where shift = floor(log2 f) and factor is 2^(32 + shift) / f
// rounded up (addend 0) or down (addend = factor, the product of state + 1).
// Rounded up by e / f the quotient is exact while state * e < 2^(32 + shift),
// rounded down by e / f while (state + 1) * e <= 2^(32 + shift); as the two
// e add up to f <= 4096, one of them always is. Powers of two round down
// from 2^32 to 2^32 - 1, where (state + 1) (2^32 - 1) >> 32 is the state.
struct AnsDivisor {
  uint32_t factor, shift, add;
};

__host__ __device__ __forceinline__ AnsDivisor MakeAnsDivisor(uint32_t f) {
  AnsDivisor d;
  d.shift = 0;
#ifdef __CUDA_ARCH__
  d.shift = 31u - static_cast<uint32_t>(__clz(static_cast<int>(f)));
#else
  while ((2u << d.shift) <= f) ++d.shift;
#endif
  if ((f & (f - 1)) == 0) {
    d.factor = 0xFFFFFFFFu;
    d.add = 1;
    return d;
  }
  // 2^(32 + shift) / f in two 16-bit steps of 32-bit divisions.
  const uint32_t n1 = 1u << (16 + d.shift), q1 = n1 / f;
  const uint32_t n2 = (n1 - q1 * f) << 16, q2 = n2 / f;
  const uint32_t down = (q1 << 16) + q2;
  const uint64_t above = f - (n2 - q2 * f);  // e rounded up
  const bool up = above * ((static_cast<uint64_t>(f) << 20) - 1) < 1ull << (32 + d.shift);
  d.factor = up ? down + 1 : down;
  d.add = up ? 0 : 1;
  return d;
}

// Encoder record of one token for the recurrence: {division factor,
// frequency, byte offset of the symbol's reverse-map entries, division shift
// | kAnsAdd | kAnsStaged}, and for the emitter {extra bits, extra-bit count}.
// The offset of a staged cluster is into the CTA's copies, else into the
// code's maps.
constexpr uint32_t kAnsAdd = 1u << 30, kAnsStaged = 1u << 31;

// slot_of: the copy that holds a cluster's map.
constexpr uint8_t kSlotNone = 0xFF;

struct AnsMaps {
  const uint8_t* contexts;      // the code's context map, or its staged copy
  const uint32_t* configs;      // per cluster {split, msb, lsb, valid}
  const uint8_t* slot_of;       // per cluster
  const uint16_t* staged_maps;  // the copies
  bool staged;                  // the first copy holds a map (or zeros)
};

__device__ __forceinline__ void AnsRecord(const Code& code, const AnsMaps& maps, uint32_t context,
                                          uint32_t value, uint4* record, uint2* extra,
                                          bool* bad) {
  uint32_t cluster = code.cluster_count;
  if (context < code.context_count) cluster = maps.contexts[context];
  const uint32_t config = cluster < code.cluster_count ? maps.configs[cluster] : 0u;
  HybridToken h = {kAnsSymbols, 0, 0};
  if (config >> 24) {
    h = EncodeHybrid(value, config & 0xFFu, (config >> 8) & 0xFFu, (config >> 16) & 0xFFu);
  }
  if (h.symbol < kAnsSymbols) {
    const uint32_t k = cluster * kAnsSymbols + h.symbol;
    const uint32_t f = code.frequencies[k];
    const uint32_t offset = code.reverse_offsets[k];
    if (f != 0 && offset + f <= kAnsTable) {
      const AnsDivisor d = MakeAnsDivisor(f);
      const uint32_t slot = maps.slot_of[cluster];
      const uint32_t map = slot != kSlotNone ? slot : cluster;
      *record = make_uint4(d.factor, f, 2 * (map * kAnsTable + offset),
                           d.shift | (d.add ? kAnsAdd : 0u) |
                             (slot != kSlotNone ? kAnsStaged : 0u));
      *extra = make_uint2(h.extra, h.count);
      return;
    }
  }
  *bad = true;
  // A harmless stand-in: frequency 4096 in the first map.
  *record = make_uint4(0xFFFFFFFFu, kAnsTable, 0u,
                       kAnsLogTable | kAnsAdd | (maps.staged ? kAnsStaged : 0u));
  *extra = make_uint2(0u, 0u);
}

// Named barriers 1 and 2: the four warps of one section.
__device__ __forceinline__ void SectionBarrier(int section) {
  if (section == 0) {
    asm volatile("bar.sync 1, 128;" ::: "memory");
  } else {
    asm volatile("bar.sync 2, 128;" ::: "memory");
  }
}

constexpr int kAnsWindow = (kAnsTokenBits * kAnsBatch + 63) / 64 + 2;

// Per-section pipeline buffers: batch k's records are filled in phase k - 1,
// consumed by the recurrence in phase k and emitted in phase k + 1.
struct AnsStage {
  uint4 records[3][kAnsBatch];
  uint2 extra[3][kAnsBatch];
  uint32_t chunks[3][kAnsBatch];  // 0x10000 | low state bits when renormalised
  unsigned long long window[kAnsWindow];
  uint32_t bad_token;
  uint32_t final_state;
  uint64_t stream_start, stream_bits;
};

// The emitter warp places one batch's bits below `*top` (the stream is
// built from its end): token i's bits, its renormalisation chunk and then
// its extra bits, start at top - L + (bits of tokens before i in the
// batch). Whole words go to the slot; the lowest, partial one is carried.
template <bool kCount>
__device__ __forceinline__ void EmitBatch(AnsStage& st, int buffer, int count, int lane,
                                          uint64_t* slots, uint64_t* top, uint64_t* carry,
                                          bool flush, uint32_t final_state) {
  uint64_t value[4];
  uint32_t length[4];
  uint32_t mine = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = 4 * lane + k;
    value[k] = 0;
    length[k] = 0;
    if (flush) {
      if (lane == 0 && k == 0) {
        value[0] = final_state;
        length[0] = 32;
      }
    } else if (i < count) {
      const uint32_t chunk = st.chunks[buffer][i];
      const uint2 e = st.extra[buffer][i];
      const uint32_t renorm = chunk >> 16;
      value[k] = (chunk & 0xFFFFu) | (static_cast<uint64_t>(e.x) << (renorm ? 16 : 0));
      length[k] = (renorm ? 16u : 0u) + e.y;
    }
    mine += length[k];
  }
  uint32_t inclusive = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, inclusive, d);
    if (lane >= d) inclusive += v;
  }
  const uint32_t total = __shfl_sync(0xffffffffu, inclusive, 31);
  if (kCount || (total == 0 && !flush)) {
    *top -= total;
    return;
  }
  const uint64_t base = *top - total;
  const uint64_t low_word = base >> 6;
  const int highest = static_cast<int>(((*top - 1) >> 6) - low_word);
  for (int j = lane; j <= highest; j += 32) {
    st.window[j] = j == highest ? *carry : 0ull;
  }
  __syncwarp();
  uint64_t at = base + (inclusive - mine);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (length[k] != 0) {
      OrBits(st.window, at - 64 * low_word, value[k]);
      at += length[k];
    }
  }
  __syncwarp();
  const int first = (flush || (base & 63) == 0) ? 0 : 1;
  for (int j = first + lane; j <= highest; j += 32) slots[low_word + j] = st.window[j];
  *carry = (base & 63) != 0 ? st.window[0] : 0ull;
  *top = base;
  __syncwarp();
}

// One step of the recurrence for the state q * 4096 + m, m being the last
// token's table slot; returns the token's renormalisation chunk.
//
// The chain from one map lookup to the next is a multiply-add for the
// quotient, its shift, a multiply-add for the address and the load. All else
// depends on the previous quotient only: whether the state is renormalised
// (state >> 20 = q >> 8), the state without m (renormalised, m drops out:
// state >> 16 = q >> 4) and its product; `step` holds it for this token and,
// computed while the lookup is under way, for the next. In a loop of plain
// shared loads a step takes 52 cycles; with a second, predicated load from
// elsewhere 108, with a branch to one 105, as one generic load 86. In the kernel,
// beside the records' loads and the chunks' stores, 78 (70,000 tokens, all maps
// staged), and about 410 for a token that leaves the loop.
struct AnsStep {
  uint64_t partial;      // (the state without m) * factor + addend
  uint32_t factor;       // multiplies m: 0 when the state is renormalised
  uint32_t scale;        // multiplies m in the address: 0 or 2
  uint32_t offset;       // the address without m and the quotient
  uint32_t frequency2;   // 2 * frequency
  uint32_t control;
  uint32_t chunk_mask;   // 0x1FFFF when the low 16 state bits are pushed
};

__device__ __forceinline__ AnsStep PrepareAnsStep(uint32_t q, const uint4& record) {
  AnsStep step;
  const bool renorm = (q >> 8) >= record.y;
  const uint32_t rest = renorm ? q >> 4 : q << kAnsLogTable;
  step.partial = static_cast<uint64_t>(rest) * record.x + ((record.w & kAnsAdd) ? record.x : 0u);
  step.factor = renorm ? 0u : record.x;
  step.scale = renorm ? 0u : 2u;
  step.offset = 2 * rest + record.z;
  step.frequency2 = 2 * record.y;
  step.control = record.w;
  step.chunk_mask = renorm ? 0x1FFFFu : 0u;
  return step;
}

// kStaged: the token's map is one of the CTA's copies, the first of which is
// at shared address base.
template <bool kStaged>
__device__ __forceinline__ uint32_t TakeAnsStep(AnsStep& step, const uint4& next_record,
                                                const uint16_t* code_maps, uint32_t base,
                                                uint32_t& q, uint32_t& m) {
  const uint32_t low = (q << kAnsLogTable) + m;
  const uint32_t chunk_mask = step.chunk_mask;
  const uint64_t product = static_cast<uint64_t>(m) * step.factor + step.partial;
  const uint32_t offset = m * step.scale + step.offset + (kStaged ? base : 0u);
  q = static_cast<uint32_t>(product >> 32) >> (step.control & 15u);
  const uint32_t at = offset - q * step.frequency2;
  if constexpr (kStaged) {
    asm volatile("{\n.reg .u16 h;\nld.shared.u16 h, [%1];\ncvt.u32.u16 %0, h;\n}"
                 : "=r"(m)
                 : "r"(at));
  } else {
    m = __ldg(reinterpret_cast<const uint16_t*>(
      reinterpret_cast<const unsigned char*>(code_maps) + at));
  }
  step = PrepareAnsStep(q, next_record);
  return (low & chunk_mask & 0xFFFFu) | (chunk_mask & 0x10000u);
}

// One section's four warps (role 0 recurrence, 1 and 2 records, 3 bits).
// kSmall: no map is staged or known to be a code's; an entry past the table
// enters the recurrence cut to the table's size, and is reported at the end.
template <bool kCount, bool kSmall>
__device__ __forceinline__ void AnsSection(const EmitParams& p, AnsStage& st, const AnsMaps& where,
                                           bool checked, uint32_t s, int section, int role,
                                           int lane, int st_thread, uint32_t begin, uint32_t end,
                                           uint64_t slot_begin, uint64_t slot_end) {
  const Code& code = p.code;
  const uint32_t n = end - begin;
  const uint32_t batches = (n + kAnsBatch - 1) / kAnsBatch;
  // Batch k (processing order) holds tokens [begin + (batches - 1 - k) *
  // kAnsBatch, ...): the last batch first.
  const auto batch_first = [&](uint32_t k) { return begin + (batches - 1 - k) * kAnsBatch; };
  const auto batch_count = [&](uint32_t k) {
    return static_cast<int>(min(static_cast<uint32_t>(kAnsBatch), end - batch_first(k)));
  };
  // A record warp takes half of every batch; its tokens of the next batch are
  // loaded before this one's records are made.
  constexpr int kHalf = kAnsBatch / 2, kPerLane = kHalf / 32;
  uint32_t contexts[kPerLane], values[kPerLane];
  const auto fetch = [&](uint32_t k) {
    const uint32_t first = batch_first(k);
    const int count = batch_count(k);
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
      const int i = (role - 1) * kHalf + j * 32 + lane;
      if (i < count) FetchToken(p.tokens, first + i, &contexts[j], &values[j]);
    }
  };
  const auto fill = [&](uint32_t k) {
    const int count = batch_count(k);
    const int buffer = k % 3;
    bool bad = false;
    uint32_t context[kPerLane], value[kPerLane];
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
      context[j] = contexts[j];
      value[j] = values[j];
    }
    if (k + 1 < batches) fetch(k + 1);
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
      const int i = (role - 1) * kHalf + j * 32 + lane;
      if (i < count) {
        AnsRecord(code, where, context[j], value[j], &st.records[buffer][i],
                  &st.extra[buffer][i], &bad);
      }
    }
    if (bad) st.bad_token = 1;
  };

  // The state is q * 4096 + m, with m the last token's table slot.
  uint32_t q = kAnsInitialState >> kAnsLogTable, m = kAnsInitialState & (kAnsTable - 1);
  uint32_t map_bits = 0;
  uint64_t top = slot_end * 64, carry = 0;
  const uint32_t base =
    kSmall ? 0 : static_cast<uint32_t>(__cvta_generic_to_shared(where.staged_maps));
  const bool records = role == 1 || role == 2;
  if (records && batches > 0) {
    fetch(0);
    fill(0);
  }
  SectionBarrier(section);
  for (uint32_t k = 0; k <= batches; ++k) {
    if (records) {
      if (k + 1 < batches) fill(k + 1);
    } else if (role == 0) {
      if (k < batches && lane == 0) {
        const int buffer = k % 3;
        const uint4* records = st.records[buffer];
        uint32_t* chunks = st.chunks[buffer];
        const int count = batch_count(k);
        if constexpr (kSmall) {
          AnsStep step = PrepareAnsStep(q, records[count - 1]);
          uint4 next = records[max(count - 2, 0)];
          for (int i = count - 1; i >= 0; --i) {
            const uint4 following = records[max(i - 2, 0)];
            chunks[i] = TakeAnsStep<false>(step, next, code.reverse_map, base, q, m);
            map_bits |= m;
            m &= kAnsTable - 1;
            next = following;
          }
        } else if (!checked) {
          // Runs of tokens whose maps are here, by plain shared loads; a token
          // between them leaves the run's loop (a choice inside the loop costs
          // every token 35 cycles, leaving it costs those that do).
          AnsStep step = PrepareAnsStep(q, records[count - 1]);
          uint4 next = records[max(count - 2, 0)];
          int i = count - 1;
          while (i >= 0) {
            for (; i >= 0 && static_cast<int32_t>(step.control) < 0; --i) {
              const uint4 following = records[max(i - 2, 0)];
              chunks[i] = TakeAnsStep<true>(step, next, code.reverse_map, base, q, m);
              next = following;
            }
            if (i < 0) break;
            const uint4 following = records[max(i - 2, 0)];
            chunks[i] = TakeAnsStep<false>(step, next, code.reverse_map, base, q, m);
            next = following;
            --i;
          }
        } else {
          uint32_t state = (q << kAnsLogTable) + m;
          uint4 next = records[count - 1];
          for (int i = count - 1; i >= 0; --i) {
            const uint4 r = next;
            next = records[max(i - 1, 0)];
            const bool renorm = (state >> (32 - kAnsLogTable)) >= r.y;
            chunks[i] = renorm ? 0x10000u | (state & 0xFFFFu) : 0u;
            state = renorm ? state >> 16 : state;
            const uint32_t quotient = state / r.y;
            const uint32_t slot = __ldg(code.reverse_map + r.z / 2 + (state - quotient * r.y));
            map_bits |= slot;
            state = (quotient << kAnsLogTable) + slot;
          }
          q = state >> kAnsLogTable;
          m = state & (kAnsTable - 1);
        }
      }
    } else if (k >= 1) {
      EmitBatch<kCount>(st, (k - 1) % 3, batch_count(k - 1), lane, p.slots, &top, &carry,
                        false, 0u);
    }
    SectionBarrier(section);
  }
  if (role == 0 && lane == 0) {
    st.final_state = (q << kAnsLogTable) + m;
    if (st.bad_token != 0 || (map_bits >> kAnsLogTable) != 0) RaiseError(p.error, kErrorRange);
  }
  SectionBarrier(section);
  if (role == 3) {
    // The final state opens the stream: its 32 bits go below everything.
    EmitBatch<kCount>(st, 0, 0, lane, p.slots, &top, &carry, true, st.final_state);
    if (lane == 0) {
      if (kCount) {
        p.bit_counts[static_cast<size_t>(s) * p.stride + p.column] = slot_end * 64 - top;
      } else {
        st.stream_start = top - slot_begin * 64;
        st.stream_bits = slot_end * 64 - top;
        p.bit_counts[static_cast<size_t>(s) * p.stride + p.column] = st.stream_bits;
      }
    }
  }
  if (kCount) return;
  SectionBarrier(section);
  // Shift the stream down to the slot's first bit, 128 words at a time; every
  // word is read (at or above its destination) before any is written.
  uint64_t* slot = p.slots + slot_begin;
  const uint64_t slot_words = slot_end - slot_begin;
  const uint64_t start = st.stream_start;
  const uint64_t words = (st.stream_bits + 63) / 64;
  for (uint64_t k0 = 0; k0 < words; k0 += kSectionThreads) {
    const uint64_t k = k0 + st_thread;
    uint64_t v = 0;
    if (k < words) {
      const uint64_t source = start + 64 * k;
      const uint64_t sw = source >> 6;
      const int shift = static_cast<int>(source & 63);
      v = slot[sw] >> shift;
      if (shift != 0 && sw + 1 < slot_words) v |= slot[sw + 1] << (64 - shift);
    }
    SectionBarrier(section);
    if (k < words) slot[k] = v;
    SectionBarrier(section);
  }
}

// Whether a lane's share of a reverse map has an entry past the table. A warp
// takes a map, all its loads under way at once: with the CTA on one map after
// another, sections of 200 tokens spent 10 of 86 us here. Not inlined: inside the
// kernel it lengthened the counting recurrence by 2% (48 sections of 31 K tokens:
// 5285 us against 5078).
__device__ __noinline__ bool MapLeavesTable(const uint16_t* map, bool aligned, int lane) {
  uint32_t bits = 0;
  if (aligned) {
#pragma unroll
    for (uint32_t i = 0; i < kAnsTable / 8; i += 32) {
      const uint4 v = reinterpret_cast<const uint4*>(map)[i + lane];
      bits |= (v.x | v.y | v.z | v.w) & 0xF000F000u;
    }
  } else {
#pragma unroll 16
    for (uint32_t i = lane; i < kAnsTable; i += 32) bits |= map[i] & 0xF000u;
  }
  return bits != 0;
}

template <bool kCount>
__global__ void __launch_bounds__(kAnsThreads) AnsSectionKernel(const __grid_constant__ EmitParams p) {
  static_assert(kAnsPairs == 2, "one named barrier per section");
  __shared__ AnsStage stage[kAnsPairs];
  __shared__ uint32_t cluster_tokens[256];
  __shared__ uint8_t slot_of[256];
  __shared__ uint8_t slot_cluster[kMaxHotClusters];
  __shared__ uint32_t configs[256];
  __shared__ uint8_t contexts[kAnsContexts];
  extern __shared__ uint4 hot_storage[];  // hot_clusters reverse maps
  const Code& code = p.code;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Four warps per section: role 0 recurrence, 1 and 2 records, 3 bits; the
  // two recurrences on different schedulers (warp % 4).
  const int section = warp / 4, role = (warp + 2 * section) % 4;
  const int st_thread = threadIdx.x - kSectionThreads * section;
  AnsStage& st = stage[section];
  const uint32_t s = blockIdx.x * kAnsPairs + section;
  uint32_t begin = 0, end = 0;
  uint64_t slot_begin = 0, slot_end = 0;
  const bool active = s < p.tokens.count && SectionBounds(p, s, !kCount, &begin, &end,
                                                         &slot_begin, &slot_end,
                                                         st_thread == 0);

  // The CTA's most used clusters (by token count over its sections) get
  // their reverse maps copied into shared memory, so that most lookups of
  // the serial recurrence are shared-memory loads.
  for (int c = threadIdx.x; c < 256; c += kAnsThreads) {
    cluster_tokens[c] = 0;
    slot_of[c] = kSlotNone;
  }
  if (threadIdx.x < kMaxHotClusters) slot_cluster[threadIdx.x] = kSlotNone;
  for (uint32_t c = threadIdx.x; c < code.cluster_count; c += kAnsThreads) {
    configs[c] = PackedConfig(code, c);
  }
  const bool stage_contexts = code.context_count <= kAnsContexts;
  for (uint32_t c = threadIdx.x; stage_contexts && c < code.context_count; c += kAnsThreads) {
    contexts[c] = code.context_map[c];
  }
  if (st_thread == 0) st.bad_token = 0;
  const uint32_t hot = min(p.hot_clusters, code.cluster_count);
  __syncthreads();
  if (active) {
    for (uint32_t t = begin + st_thread; t < end; t += kSectionThreads) {
      uint32_t context, value;
      FetchToken(p.tokens, t, &context, &value);
      if (context < code.context_count) {
        const uint32_t cluster = code.context_map[context];
        if (cluster < code.cluster_count) atomicAdd(&cluster_tokens[cluster], 1u);
      }
    }
  }
  __syncthreads();
  for (uint32_t c = threadIdx.x; hot > 0 && c < code.cluster_count; c += kAnsThreads) {
    const uint32_t mine = cluster_tokens[c];
    if (mine == 0) continue;
    uint32_t rank = 0;
    for (uint32_t o = 0; o < code.cluster_count; ++o) {
      const uint32_t other = cluster_tokens[o];
      rank += other > mine || (other == mine && o < c);
    }
    if (rank < hot) {
      slot_of[c] = static_cast<uint8_t>(rank);
      slot_cluster[rank] = static_cast<uint8_t>(c);
    }
  }
  __syncthreads();
  // The maps in use are copied or looked through: one with an entry past the
  // table is no ANS code, and its tokens take the checked recurrence, which
  // reports the entry where it is used.
  bool outside = false;
  constexpr uint32_t kVectors = kAnsTable * 2 / 16;  // uint4 per map
  const uint4* maps = reinterpret_cast<const uint4*>(code.reverse_map);
  const auto out_of_table = [](const uint4& v) {
    return ((v.x | v.y | v.z | v.w) & 0xF000F000u) != 0;
  };
  for (uint32_t i = threadIdx.x; i < hot * kVectors; i += kAnsThreads) {
    const uint32_t cluster = slot_cluster[i / kVectors];
    uint4 v = make_uint4(0, 0, 0, 0);
    if (cluster != kSlotNone) v = maps[cluster * kVectors + i % kVectors];
    outside |= out_of_table(v);
    hot_storage[i] = v;
  }
  const bool aligned = reinterpret_cast<uintptr_t>(maps) % 16 == 0;
  for (uint32_t c = warp; c < code.cluster_count; c += kAnsThreads / 32) {
    // Without copies, the first map stands in for a bad token's.
    const bool needed = cluster_tokens[c] != 0 || (c == 0 && hot == 0);
    if (!needed || slot_of[c] != kSlotNone) continue;
    outside |= MapLeavesTable(code.reverse_map + c * kAnsTable, aligned, lane);
  }
  const bool checked = __syncthreads_or(outside) != 0;
  if (checked) {
    for (int c = threadIdx.x; c < 256; c += kAnsThreads) slot_of[c] = kSlotNone;
  }
  __syncthreads();
  AnsMaps where;
  where.slot_of = slot_of;
  where.configs = configs;
  where.contexts = stage_contexts ? contexts : code.context_map;
  where.staged_maps = reinterpret_cast<const uint16_t*>(hot_storage);
  where.staged = hot > 0 && !checked;
  if (active) {
    AnsSection<kCount, false>(p, st, where, checked, s, section, role, lane, st_thread, begin,
                              end, slot_begin, slot_end);
  }
}

// The same for small sections: nothing is staged but the clusters'
// configurations. The kernel above counts each CTA's clusters, copies maps and
// looks the others through before the first token, 8 KB a map, which a few
// hundred tokens don't repay; and its copies leave room for four CTAs per SM.
template <bool kCount>
__global__ void __launch_bounds__(kAnsThreads, 5)
AnsSmallKernel(const __grid_constant__ EmitParams p) {
  __shared__ AnsStage stage[kAnsPairs];
  __shared__ uint32_t configs[256];
  __shared__ __align__(4) uint8_t slot_of[256];
  const Code& code = p.code;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int section = warp / 4, role = (warp + 2 * section) % 4;
  const int st_thread = threadIdx.x - kSectionThreads * section;
  AnsStage& st = stage[section];
  const uint32_t s = blockIdx.x * kAnsPairs + section;
  uint32_t begin = 0, end = 0;
  uint64_t slot_begin = 0, slot_end = 0;
  const bool active = s < p.tokens.count && SectionBounds(p, s, !kCount, &begin, &end,
                                                         &slot_begin, &slot_end,
                                                         st_thread == 0);
  for (uint32_t c = threadIdx.x; c < code.cluster_count; c += kAnsThreads) {
    configs[c] = PackedConfig(code, c);
    slot_of[c] = kSlotNone;
  }
  if (st_thread == 0) st.bad_token = 0;
  __syncthreads();
  AnsMaps where;
  where.slot_of = slot_of;
  where.configs = configs;
  where.contexts = code.context_map;
  where.staged_maps = nullptr;
  where.staged = false;
  if (active) {
    AnsSection<kCount, true>(p, st, where, false, s, section, role, lane, st_thread, begin, end,
                             slot_begin, slot_end);
  }
}

// ------------------------------------------------------------- prefix ----

// A prefix code's tables as one CTA keeps them in shared memory: the context
// map, one word per cluster {split, msb, lsb, valid} and one per symbol
// {code bits, depth << 16, present << 24}; a degenerate symbol has depth 0.
struct PrefixTables {
  const uint32_t* symbols;
  const uint32_t* configs;
  const uint8_t* contexts;
};

constexpr size_t kPrefixStagedBytes = 96 * 1024;  // two CTAs per SM

__host__ __device__ __forceinline__ size_t PrefixTableBytes(uint32_t contexts,
                                                            uint32_t clusters) {
  return static_cast<size_t>(clusters) * (kPrefixSymbols + 1) * 4 + contexts;
}

__device__ __forceinline__ PrefixTables StagePrefixTables(const Code& code, uint32_t* memory) {
  uint32_t* configs = memory + code.cluster_count * kPrefixSymbols;
  uint8_t* contexts = reinterpret_cast<uint8_t*>(configs + code.cluster_count);
#pragma unroll 4
  for (uint32_t i = threadIdx.x; i < code.cluster_count * kPrefixSymbols; i += kPrefixThreads) {
    const uint32_t depth = code.prefix_depths[i];
    const bool degenerate = code.prefix_degenerate[i / kPrefixSymbols] == i % kPrefixSymbols;
    memory[i] = code.prefix_bits[i] | (degenerate ? 0u : depth << 16) |
                (depth != 0 ? 1u << 24 : 0u);
  }
  for (uint32_t i = threadIdx.x; i < code.cluster_count; i += kPrefixThreads) {
    configs[i] = PackedConfig(code, i);
  }
#pragma unroll 4
  for (uint32_t i = threadIdx.x; i < code.context_count; i += kPrefixThreads) {
    contexts[i] = code.context_map[i];
  }
  return {memory, configs, contexts};
}

// One token's bits and their number; false for a token the code lacks.
__device__ __forceinline__ bool PrefixToken(const Code& code, const PrefixTables& tables,
                                            uint32_t context, uint32_t value, uint64_t* data,
                                            uint32_t* length) {
  if (tables.symbols != nullptr) {
    if (context >= code.context_count) return false;
    const uint32_t cluster = tables.contexts[context];
    if (cluster >= code.cluster_count) return false;
    const uint32_t config = tables.configs[cluster];
    if (!(config >> 24)) return false;
    const HybridToken h =
      EncodeHybrid(value, config & 0xFFu, (config >> 8) & 0xFFu, (config >> 16) & 0xFFu);
    if (h.symbol >= kPrefixSymbols) return false;
    const uint32_t entry = tables.symbols[cluster * kPrefixSymbols + h.symbol];
    if (!(entry >> 24)) return false;
    const uint32_t depth = (entry >> 16) & 0xFFu;
    *data = (entry & 0xFFFFu) | (static_cast<uint64_t>(h.extra) << depth);
    *length = depth + h.count;
    return true;
  }
  uint32_t cluster;
  HybridToken h;
  if (!ClusterToken(code, context, value, &cluster, &h) || h.symbol >= kPrefixSymbols ||
      code.prefix_depths[cluster * kPrefixSymbols + h.symbol] == 0) {
    return false;
  }
  const uint32_t depth = code.prefix_degenerate[cluster] == h.symbol
                           ? 0u
                           : code.prefix_depths[cluster * kPrefixSymbols + h.symbol];
  *data = code.prefix_bits[cluster * kPrefixSymbols + h.symbol] |
          (static_cast<uint64_t>(h.extra) << depth);
  *length = depth + h.count;
  return true;
}

// Bound: latency (a chunk is a token load, three dependent table lookups, a
// scan and a window flush, one CTA per section). The tables sit in shared
// memory where they fit kPrefixStagedBytes, and the next chunk's tokens are
// loaded while this one is placed. With 256 threads and the lookups in global
// memory, 192 sections of 31 K tokens took 353 us.
template <bool kCount, bool kSmall>
__global__ void __launch_bounds__(kSmall ? kPrefixSmallThreads : kPrefixThreads,
                                  kSmall ? (kCount ? 8 : 6) : 2)
PrefixSectionKernel(const __grid_constant__ EmitParams p, bool staged) {
  constexpr int kThreads = kSmall ? kPrefixSmallThreads : kPrefixThreads;
  constexpr int kChunk = kThreads * kPrefixPerThread;
  // Words a chunk can touch: its bits plus the partial word it starts in.
  constexpr int kWindow = (kPrefixTokenBits * kChunk + 63) / 64 + 2;
  extern __shared__ uint32_t prefix_tables[];
  __shared__ unsigned long long window[kWindow];
  __shared__ uint32_t warp_bits[2][kThreads / 32];
  __shared__ uint32_t bad_token;
  uint32_t begin, end;
  uint64_t slot_begin, slot_end;
  if (!SectionBounds(p, blockIdx.x, !kCount, &begin, &end, &slot_begin, &slot_end,
                     threadIdx.x == 0)) {
    return;
  }
  const Code& code = p.code;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t* slot = p.slots + slot_begin;
  uint32_t context[kPrefixPerThread], value[kPrefixPerThread];
  const auto fetch = [&](uint32_t first) {
#pragma unroll
    for (int k = 0; k < kPrefixPerThread; ++k) {
      const uint32_t t = first + threadIdx.x * kPrefixPerThread + k;
      if (t < end) FetchToken(p.tokens, t, &context[k], &value[k]);
    }
  };
  if constexpr (!kSmall) fetch(begin);
  PrefixTables tables = {nullptr, nullptr, nullptr};
  if (!kSmall && staged) tables = StagePrefixTables(code, prefix_tables);
  if (threadIdx.x == 0) bad_token = 0;
  // window[0] holds the partial word a chunk starts in; the rest is zero.
  for (int i = threadIdx.x; i < kWindow; i += kThreads) window[i] = 0;
  __syncthreads();
  uint64_t position = 0;  // bits written so far
  int parity = 0;
  for (uint32_t first = begin; first < end; first += kChunk, parity ^= 1) {
    uint64_t data[kPrefixPerThread];
    uint32_t length[kPrefixPerThread];
    uint32_t mine = 0;
    bool bad = false;
    if constexpr (kSmall) fetch(first);
#pragma unroll
    for (int k = 0; k < kPrefixPerThread; ++k) {
      const uint32_t t = first + threadIdx.x * kPrefixPerThread + k;
      data[k] = 0;
      length[k] = 0;
      if (t < end && !PrefixToken(code, tables, context[k], value[k], &data[k], &length[k])) {
        bad = true;
      }
      mine += length[k];
    }
    if (bad) bad_token = 1;
    if (!kSmall && end - first > kChunk) fetch(first + kChunk);
    // Exclusive scan of the threads' bit counts.
    uint32_t inclusive = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, inclusive, d);
      if (lane >= d) inclusive += v;
    }
    if (lane == 31) warp_bits[parity][warp] = inclusive;
    __syncthreads();
    uint32_t before = inclusive - mine, chunk_bits = 0;
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) {
      const uint32_t v = warp_bits[parity][i];
      if (i < warp) before += v;
      chunk_bits += v;
    }
    if (!kCount) {
      const uint64_t w0 = position >> 6;
      uint64_t at = (position & 63) + before;
#pragma unroll
      for (int k = 0; k < kPrefixPerThread; ++k) {
        if (length[k] != 0) {
          OrBits(window, at, data[k]);
          at += length[k];
        }
      }
      __syncthreads();
      // Whole words finished go out; the one in progress moves to the front.
      const uint64_t end_bit = position + chunk_bits;
      const int full = static_cast<int>((end_bit >> 6) - w0);
      unsigned long long partial = 0;
      if (threadIdx.x == 0) partial = window[full];
      for (int i = threadIdx.x; i < full; i += kThreads) {
        slot[w0 + i] = window[i];
        window[i] = 0;
      }
      if (threadIdx.x == 0) {
        window[full] = 0;
        window[0] = partial;
      }
      __syncthreads();
    }
    position += chunk_bits;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (!kCount && (position & 63) != 0) slot[position >> 6] = window[0];
    if (bad_token != 0) RaiseError(p.error, kErrorRange);
    p.bit_counts[static_cast<size_t>(blockIdx.x) * p.stride + p.column] = position;
  }
}

// ------------------------------------------------------------ packing ----

// byte_offsets[s] = sum over earlier sections of ceil(bits / 8); one CTA.
__global__ void __launch_bounds__(1024) SectionByteOffsetsKernel(const uint64_t* bit_counts,
                                                                 uint32_t count,
                                                                 uint64_t* byte_offsets) {
  __shared__ uint64_t warp_sums[32];
  __shared__ uint64_t carry;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint32_t first = 0; first < count; first += 1024) {
    const uint32_t s = first + threadIdx.x;
    const uint64_t mine = s < count ? (bit_counts[s] + 7) / 8 : 0;
    uint64_t inclusive = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint64_t v = __shfl_up_sync(0xffffffffu, inclusive, d);
      if (lane >= d) inclusive += v;
    }
    if (lane == 31) warp_sums[warp] = inclusive;
    __syncthreads();
    uint64_t before = carry + inclusive - mine, total = 0;
    for (int i = 0; i < 32; ++i) {
      if (i < warp) before += warp_sums[i];
      total += warp_sums[i];
    }
    if (s < count) byte_offsets[s] = before;
    __syncthreads();
    if (threadIdx.x == 0) carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) byte_offsets[count] = carry;
}

// CTAs per section, and the tokens per section that take one only (5000
// sections of 100 tokens: 4 CTAs each cost 8 us of 51).
constexpr unsigned kPackSplit = 4;
constexpr uint32_t kPackOne = 1024;

__global__ void __launch_bounds__(256) PackSectionsKernel(const uint64_t* slots,
                                                          size_t slot_capacity,
                                                          const uint32_t* offsets, int mode,
                                                          const uint64_t* bit_counts,
                                                          const uint64_t* byte_offsets,
                                                          uint8_t* packed, size_t capacity,
                                                          uint32_t* error) {
  const uint32_t s = blockIdx.x;
  const uint64_t bytes = (bit_counts[s] + 7) / 8;
  const uint64_t at = byte_offsets[s];
  const uint64_t first = SlotStart(offsets[s], s, TokenBits(mode));
  if (at + bytes > capacity || first * 8 + bytes > slot_capacity * 8) {
    if (threadIdx.x == 0) RaiseError(error, kErrorRange);
    return;
  }
  // Whole 8-byte words of the destination, each from the two slot words that
  // hold its bytes; single bytes at the section's ends. blockIdx.y shares the
  // words out. Copying byte by byte took 43 us for 5 MB.
  const uint8_t* source = reinterpret_cast<const uint8_t*>(slots + first);
  uint8_t* out = packed + at;
  const uint64_t head =
    min(bytes, static_cast<uint64_t>(-reinterpret_cast<uintptr_t>(out) & 7u));
  const uint64_t words = (bytes - head) / 8;
  const uint64_t tail = head + 8 * words;
  const int shift = 8 * static_cast<int>(head);
  const uint64_t step = static_cast<uint64_t>(gridDim.y) * blockDim.x;
  uint64_t* out_words = reinterpret_cast<uint64_t*>(out + head);
  for (uint64_t i = static_cast<uint64_t>(blockIdx.y) * blockDim.x + threadIdx.x; i < words;
       i += step) {
    uint64_t v = slots[first + i] >> shift;
    if (shift != 0) v |= slots[first + i + 1] << (64 - shift);
    out_words[i] = v;
  }
  if (blockIdx.y == 0) {
    if (threadIdx.x < head) out[threadIdx.x] = source[threadIdx.x];
    if (tail + threadIdx.x < bytes) out[tail + threadIdx.x] = source[tail + threadIdx.x];
  }
}

// ---------------------------------------------------------------- host ----

bool ValidCode(const gjxl_b200_entropy_code* c) {
  if (c == nullptr || c->context_count == 0 || c->context_count > 65536 ||
      c->cluster_count == 0 || c->cluster_count > 256 || c->context_map == nullptr ||
      c->uint_configs == nullptr) {
    return false;
  }
  if (c->mode == GJXL_B200_ENTROPY_PREFIX) {
    return c->prefix_depths != nullptr && c->prefix_bits != nullptr &&
           c->prefix_degenerate != nullptr;
  }
  if (c->mode == GJXL_B200_ENTROPY_ANS) {
    return c->ans_frequencies != nullptr && c->ans_reverse_offsets != nullptr &&
           c->ans_reverse_map != nullptr;
  }
  return false;
}

bool ValidTokens(const gjxl_b200_token_sections* t) {
  if (t == nullptr || t->offsets == nullptr || t->count == 0) return false;
  if (t->pairs != nullptr) {
    return t->values == nullptr && t->contexts == nullptr &&
           reinterpret_cast<uintptr_t>(t->pairs) % 8 == 0;
  }
  return t->values != nullptr && t->contexts != nullptr;
}

Code DeviceCode(const gjxl_b200_entropy_code& c) {
  Code d;
  d.mode = c.mode;
  d.context_count = c.context_count;
  d.cluster_count = c.cluster_count;
  d.context_map = c.context_map;
  d.uint_configs = c.uint_configs;
  d.prefix_depths = c.prefix_depths;
  d.prefix_bits = c.prefix_bits;
  d.prefix_degenerate = c.prefix_degenerate;
  d.frequencies = c.ans_frequencies;
  d.reverse_offsets = c.ans_reverse_offsets;
  d.reverse_map = c.ans_reverse_map;
  return d;
}

Tokens DeviceTokens(const gjxl_b200_token_sections& t) {
  Tokens d;
  d.pairs = reinterpret_cast<const uint2*>(t.pairs);
  d.values = t.values;
  d.contexts = t.contexts;
  d.offsets = t.offsets;
  d.count = t.count;
  d.capacity = t.capacity;
  return d;
}

struct DeviceLimits {
  int sms = 0;
  int smem_per_sm = 0;
  int smem_per_block = 0;
};

DeviceLimits Limits() {
  DeviceLimits l;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess ||
      cudaDeviceGetAttribute(&l.sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
      cudaDeviceGetAttribute(&l.smem_per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor,
                             device) != cudaSuccess ||
      cudaDeviceGetAttribute(&l.smem_per_block, cudaDevAttrMaxSharedMemoryPerBlockOptin,
                             device) != cudaSuccess) {
    cudaGetLastError();
    return DeviceLimits{};
  }
  return l;
}

const DeviceLimits& CachedLimits() {
  static const DeviceLimits limits = Limits();
  return limits;
}

// Reverse maps that fit in `bytes` of shared memory beside the ANS kernel's
// static arrays.
int MapsWithin(int bytes) {
  constexpr int kStatic = kAnsPairs * static_cast<int>(sizeof(AnsStage)) + 2 * 256 * 4 + 256 +
                          static_cast<int>(kAnsContexts) +
                          kMaxHotClusters + 64;
  return std::max(0, std::min((bytes - kStatic) / static_cast<int>(kAnsTable * 2),
                              static_cast<int>(kMaxHotClusters)));
}

// Reverse maps staged per CTA: as many as fit in the shared memory one CTA
// may take while all sections still run in one wave (up to four CTAs per
// SM), at most the code's clusters. Maps must be 16-byte aligned.
uint32_t HotClusters(const EmitParams& p) {
  if (reinterpret_cast<uintptr_t>(p.code.reverse_map) % 16 != 0) return 0;
  const DeviceLimits& limits = CachedLimits();
  if (limits.sms <= 0 || limits.smem_per_sm <= 0) return 0;
  const int ctas = static_cast<int>((p.tokens.count + kAnsPairs - 1) / kAnsPairs);
  const int per_sm = std::min(4, std::max(1, (ctas + limits.sms - 1) / limits.sms));
  const int maps = MapsWithin(std::min(limits.smem_per_block, limits.smem_per_sm / per_sm - 1024));
  return std::min(static_cast<uint32_t>(maps), p.code.cluster_count);
}

// Whether the sections are too small to repay what the full kernels stage for
// each of them, by the tokens per section that the arrays hold. Sections x
// tokens, us a call with packing (and counting only), full against small:
//   ANS     300 x 20: 27 (19) / 23 (15)      5000 x 100: 172 (148) / 123 (99)
//           600 x 100: 50 (43) / 57 (48)     2000 x 500: 303 (294) / 248 (235)
//           300 x 200: 76 (70) / 99 (90)     1000 x 1000: 428 (424) / 409 (402)
//   prefix  48 x 500: 14.5 (6.5) / 14.7 (6.4)    5000 x 100: 93 (58) / 43 (15)
//           300 x 500: 16.6 (9.2) / 14.7 (6.5)   2000 x 2000: 60 (35) / 54 (27)
//           500 x 2000: 25 (14.5) / 29 (14.5)    2000 x 5000: 100 (58) / 109 (59)
// The small ANS kernel takes more CTAs an SM, so that it gains where the
// sections fill the chip several times; below, only tokens that are fewer than
// the full kernel's preparation. Prefix sections cost a staging each, which a
// chip full of them pays once per turn: the more turns, the larger a section
// has to be.
bool SmallAnsSections(const Tokens& t) {
  const uint32_t tokens = t.capacity / t.count;
  return tokens < 64 || (tokens < 512 && t.count / 8 > static_cast<uint32_t>(CachedLimits().sms));
}

bool SmallPrefixSections(const Tokens& t) {
  const uint64_t sms = std::max(1, CachedLimits().sms);
  return t.capacity / t.count < std::min<uint64_t>(4096, 512 * (t.count / sms));
}

// Both writers raise their kernel's shared-memory limit to the most that any
// call asks for, not to this call's need: the limit belongs to the kernel, and
// calls from several host threads share it.
template <bool kCount>
void LaunchAns(EmitParams p, cudaStream_t stream) {
  const unsigned ctas = (p.tokens.count + kAnsPairs - 1) / kAnsPairs;
  if (SmallAnsSections(p.tokens)) {
    AnsSmallKernel<kCount><<<ctas, kAnsThreads, 0, stream>>>(p);
    return;
  }
  p.hot_clusters = HotClusters(p);
  const int most = MapsWithin(CachedLimits().smem_per_block) * static_cast<int>(kAnsTable * 2);
  if (p.hot_clusters > 0 &&
      cudaFuncSetAttribute(AnsSectionKernel<kCount>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           most) != cudaSuccess) {
    cudaGetLastError();
    p.hot_clusters = 0;
  }
  AnsSectionKernel<kCount>
    <<<ctas, kAnsThreads, p.hot_clusters * kAnsTable * 2, stream>>>(p);
}

template <bool kCount>
void LaunchSections(const EmitParams& p, cudaStream_t stream) {
  if (p.code.mode == GJXL_B200_ENTROPY_ANS) {
    LaunchAns<kCount>(p, stream);
  } else {
    if (SmallPrefixSections(p.tokens)) {
      PrefixSectionKernel<kCount, true>
        <<<p.tokens.count, kPrefixSmallThreads, 0, stream>>>(p, false);
      return;
    }
    // The tables are staged where two CTAs of them fit an SM; a larger code is
    // looked up in global memory.
    const size_t bytes = PrefixTableBytes(p.code.context_count, p.code.cluster_count);
    bool staged = bytes <= kPrefixStagedBytes;
    if (staged && cudaFuncSetAttribute(PrefixSectionKernel<kCount, false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(kPrefixStagedBytes)) != cudaSuccess) {
      cudaGetLastError();
      staged = false;
    }
    PrefixSectionKernel<kCount, false>
      <<<p.tokens.count, kPrefixThreads, staged ? bytes : 0, stream>>>(p, staged);
  }
}

}  // namespace
}  // namespace gjxl_b200

using namespace gjxl_b200;

extern "C" size_t gjxl_b200_entropy_slot_words(int mode, size_t tokens, size_t sections) {
  if (mode != GJXL_B200_ENTROPY_ANS && mode != GJXL_B200_ENTROPY_PREFIX) return 0;
  return SlotStart(tokens, sections, TokenBits(mode));
}

extern "C" int gjxl_b200_entropy_write_sections(const gjxl_b200_entropy_code* code,
                                                const gjxl_b200_token_sections* sections,
                                                uint64_t* slot_words, size_t slot_word_capacity,
                                                uint64_t* bit_counts, uint8_t* packed,
                                                size_t packed_capacity, uint64_t* byte_offsets,
                                                uint32_t* device_error, void* stream) {
  ClearLastError();
  if (!ValidCode(code) || !ValidTokens(sections) || slot_words == nullptr ||
      bit_counts == nullptr || slot_word_capacity == 0 ||
      (packed != nullptr && (byte_offsets == nullptr || packed_capacity == 0))) {
    return SetError(GJXL_B200_INVALID_ARGUMENT, "entropy_write_sections: invalid arguments");
  }
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  EmitParams p;
  p.code = DeviceCode(*code);
  p.tokens = DeviceTokens(*sections);
  p.slots = slot_words;
  p.slot_capacity = slot_word_capacity;
  p.bit_counts = bit_counts;
  p.stride = 1;
  p.column = 0;
  p.hot_clusters = 0;
  p.error = device_error;
  LaunchSections<false>(p, s);
  int status = CheckLaunch("entropy sections");
  if (status != GJXL_B200_OK || packed == nullptr) return status;
  SectionByteOffsetsKernel<<<1, 1024, 0, s>>>(bit_counts, sections->count, byte_offsets);
  const unsigned split = sections->capacity / sections->count < kPackOne ? 1 : kPackSplit;
  PackSectionsKernel<<<dim3(sections->count, split), 256, 0, s>>>(
    slot_words, slot_word_capacity, sections->offsets, code->mode, bit_counts, byte_offsets, packed,
    packed_capacity, device_error);
  return CheckLaunch("entropy section packing");
}

extern "C" int gjxl_b200_entropy_count_sections(const gjxl_b200_entropy_code* codes,
                                                uint32_t code_count,
                                                const gjxl_b200_token_sections* sections,
                                                uint64_t* bit_counts, uint32_t* device_error,
                                                void* stream) {
  ClearLastError();
  bool ok = codes != nullptr && code_count >= 1 && code_count <= kMaxCodes &&
            ValidTokens(sections) && bit_counts != nullptr;
  for (uint32_t c = 0; ok && c < code_count; ++c) ok = ValidCode(&codes[c]);
  if (!ok) return SetError(GJXL_B200_INVALID_ARGUMENT, "entropy_count_sections: invalid arguments");
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  for (uint32_t c = 0; c < code_count; ++c) {
    EmitParams p;
    p.code = DeviceCode(codes[c]);
    p.tokens = DeviceTokens(*sections);
    p.slots = nullptr;
    p.slot_capacity = 0;
    p.bit_counts = bit_counts;
    p.stride = code_count;
    p.column = c;
    p.hot_clusters = 0;
    p.error = device_error;
    LaunchSections<true>(p, s);
    const int status = CheckLaunch("entropy section counts");
    if (status != GJXL_B200_OK) return status;
  }
  return GJXL_B200_OK;
}
