// Paged KV cache fill / gather / row moves. Pure byte movement: bit-exact by construction.
//
//   fill   : new K/V rows [T, H, D]  ->  K [NB, H, D/x, B, x], V [NB, H, D, B] at slot_mapping[t]
//   gather : the inverse
//   move   : dest[dest_idx[i]] = row of slot src_slots[i] (K or V)
//   rows   : dest[dest_idx[i]] = src[src_idx[i]] over plain rows
//
// Runs of tokens whose slots are consecutive inside one physical block (prefill) share sectors of the V tiles and
// are written together; a lone decode token degenerates to the scattered element writes the layout forces.
// Block size 16 (the engine's): fills, rotary and moves take windows of 16 tokens (fill_window_kernel,
// move_runs_kernel). Other block sizes, and every gather, take a warp per (run, head): K as 16-byte chunks, V
// transposed through shared memory so that a full block is written with 16-byte stores (kv_run_kernel).
//
// Reference counterparts: reshape_and_cache_kernel / gather_cached_kv_kernel
// (3rdparty/vllm/csrc/cache_kernels.cu:142-182, 229-344) and the Triton movers
// (parrot/engine/builtin/kernels/tokens_moving.py:25-64, 104-160, 222-268).
#include "common.cuh"

namespace pb {
namespace {

constexpr int kFillWarps = 4;

__device__ __forceinline__ long long load_slot(const void* slots, int is64, long long t) {
  return is64 ? reinterpret_cast<const long long*>(slots)[t]
              : (long long)reinterpret_cast<const int*>(slots)[t];
}

// Kernels launched with programmatic serialization begin while the kernel before them still writes: what
// they read (rows, cache cells, cos/sin) is only settled after pdl_wait(). Their loads must therefore be
// ordinary ones; the read-only path (__ldg, or const __restrict__ parameters, which the compiler may turn into
// it) asks for data that nobody writes during the whole life of the kernel. Hence no __restrict__ in those
// kernels, and loads that are to be in flight together are written as load16() into registers first.
__device__ __forceinline__ uint4 load16(const void* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

template <int E> struct ElemOf;
template <> struct ElemOf<2> { using type = uint16_t; };
template <> struct ElemOf<4> { using type = uint32_t; };
template <typename T> __device__ __forceinline__ T load_elem(const void* p);
template <> __device__ __forceinline__ uint16_t load_elem<uint16_t>(const void* p) {
  uint16_t v;
  asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p));
  return v;
}
template <> __device__ __forceinline__ uint32_t load_elem<uint32_t>(const void* p) {
  uint32_t v;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// Runs of a list of slots: lane l of the warp holds entry first - 1 + l (its slot, or a negative number
// outside the list). A run is a maximal stretch of entries with consecutive slots inside one block of 16;
// bit l of `cont` says that entry l continues the run of the entry before it. A run that starts in lanes
// 1..16 ends in lane 31 at the latest.
__device__ __forceinline__ unsigned run_continues(long long slot) {
  const long long before = __shfl_up_sync(0xffffffffu, slot, 1);
  const bool cont = (threadIdx.x & 31) > 0 && slot > 0 && before >= 0 && slot == before + 1 && (slot & 15) != 0;
  return __ballot_sync(0xffffffffu, cont);
}
__device__ __forceinline__ int run_length(unsigned cont, int lane_of_first) {
  const unsigned rest = lane_of_first < 31 ? cont >> (lane_of_first + 1) : 0u;
  return __ffs(~rest);  // 1 + trailing ones (bit 31 of `rest` is never set)
}

// FILL == true : scatter rows into the cache.   FILL == false : gather rows out of the cache.
template <int E, bool FILL>
__global__ void __launch_bounds__(kFillWarps * 32) kv_run_kernel(
    uint8_t* key, uint8_t* value, uint8_t* kcache,
    uint8_t* vcache, const void* slots, const int is64,
    const long long T, const int H, const int D, const int B, const long long key_stride,
    const long long value_stride, const long long kbs, const long long khs,
    const long long num_blocks, int* status) {
  using elem_t = typename ElemOf<E>::type;
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long t = blockIdx.x;
  // Launched with programmatic stream serialization, so the CTAs are resident while the kernel
  // before this one drains: wait for it before reading anything, then let the next kernel (an
  // attention kernel or the planner) set itself up; those wait before they read the cache.
  pdl_wait();
  pdl_trigger();
  // the three slot reads do not depend on each other: issue them together
  const long long slot = load_slot(slots, is64, t);
  const long long prev = (t > 0) ? load_slot(slots, is64, t - 1) : -2;
  const long long next = (lane > 0 && lane < B && t + lane < T) ? load_slot(slots, is64, t + lane) : -3;
  if (slot < 0) return;
  const long long blk = slot / B;
  const int off0 = (int)(slot - blk * B);
  if (blk >= num_blocks) {
    if (threadIdx.x == 0 && status) atomicMax(status, kStatusBadIndex);
    return;
  }
  const bool leader = (t == 0) || (prev + 1 != slot) || (off0 == 0);
  if (!leader) return;
  // run length: tokens t+i with slot+i, staying inside the block
  bool ok = (lane == 0);
  if (lane > 0 && lane < B && off0 + lane < B && t + lane < T) ok = (next == slot + lane);
  const unsigned mask = __ballot_sync(0xffffffffu, ok);
  const int n = __ffs(~mask) - 1;  // trailing ones; mask bit 0 is always set, n in 1..B (32 -> ~mask==0)
  const int run = (~mask == 0u) ? 32 : n;

  constexpr int kVec = 16 / E;
  const int nch = D / kVec;  // 16-byte chunks per (token, head) row
  uint8_t* tile = smem + (size_t)warp * B * D * E;

  for (int h = blockIdx.y * kFillWarps + warp; h < H; h += gridDim.y * kFillWarps) {
    uint8_t* kt = kcache + ((size_t)blk * kbs + (size_t)h * khs) * E;
    uint8_t* vt = vcache + ((size_t)blk * kbs + (size_t)h * khs) * E;
    // ---- K: 16-byte chunk (token i, chunk c) <-> tile[(c*B + off0+i)] ----
    // (four chunks per lane are read before the first is written: a run of a whole block is 8 chunks
    // per lane, and one dependent load-store pair per trip to memory made the copy latency-bound)
    for (int base = 0; base < run * nch; base += 4 * 32) {
      uint4 tmp[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int idx = base + u * 32 + lane;
        if (idx < run * nch) {
          const int i = idx / nch, c = idx - i * nch;
          const uint4* row = reinterpret_cast<const uint4*>(key + ((size_t)(t + i) * key_stride + (size_t)h * D) * E) + c;
          const uint4* cell = reinterpret_cast<const uint4*>(kt) + (size_t)c * B + off0 + i;
          tmp[u] = load16(FILL ? row : cell);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int idx = base + u * 32 + lane;
        if (idx < run * nch) {
          const int i = idx / nch, c = idx - i * nch;
          uint4* row = reinterpret_cast<uint4*>(key + ((size_t)(t + i) * key_stride + (size_t)h * D) * E) + c;
          uint4* cell = reinterpret_cast<uint4*>(kt) + (size_t)c * B + off0 + i;
          if (FILL) *cell = tmp[u]; else *row = tmp[u];
        }
      }
    }
    // ---- V: element (token i, d) <-> tile[d*B + off0+i], transposed through shared memory ----
    if (FILL) {
      for (int base = 0; base < run * nch; base += 4 * 32) {  // four loads in flight per lane, as for K
        uint4 tmp[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int idx = base + u * 32 + lane;
          if (idx < run * nch) {
            const int i = idx / nch, c = idx - i * nch;
            tmp[u] = load16(value + ((size_t)(t + i) * value_stride + (size_t)h * D + c * kVec) * E);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int idx = base + u * 32 + lane;
          if (idx < run * nch) reinterpret_cast<uint4*>(tile)[idx] = tmp[u];  // idx == i * nch + c
        }
      }
      __syncwarp();
      const elem_t* ts = reinterpret_cast<const elem_t*>(tile);
      for (int dd = lane; dd < D; dd += 32) {
        elem_t* dst = reinterpret_cast<elem_t*>(vt) + (size_t)dd * B + off0;
        if (run == B) {  // a full block (off0 == 0): 16-byte stores
          for (int v = 0; v < B / kVec; ++v) {
            elem_t tmp[kVec];
#pragma unroll
            for (int j = 0; j < kVec; ++j) tmp[j] = ts[(size_t)(v * kVec + j) * D + dd];
            reinterpret_cast<uint4*>(dst)[v] = *reinterpret_cast<const uint4*>(tmp);
          }
        } else {
          for (int i = 0; i < run; ++i) dst[i] = ts[(size_t)i * D + dd];
        }
      }
      __syncwarp();
    } else {
      elem_t* ts = reinterpret_cast<elem_t*>(tile);
      for (int dd = lane; dd < D; dd += 32) {
        const elem_t* src = reinterpret_cast<const elem_t*>(vt) + (size_t)dd * B + off0;
        if (run == B) {
          for (int v = 0; v < B / kVec; ++v) {
            const uint4 u = reinterpret_cast<const uint4*>(src)[v];
            const elem_t* tmp = reinterpret_cast<const elem_t*>(&u);
#pragma unroll
            for (int j = 0; j < kVec; ++j) ts[(size_t)(v * kVec + j) * D + dd] = tmp[j];
          }
        } else {
          for (int i = 0; i < run; ++i) ts[(size_t)i * D + dd] = src[i];
        }
      }
      __syncwarp();
      for (int idx = lane; idx < run * nch; idx += 32) {
        const int i = idx / nch, c = idx - i * nch;
        uint4* row = reinterpret_cast<uint4*>(value + ((size_t)(t + i) * value_stride + (size_t)h * D) * E) + c;
        *row = reinterpret_cast<const uint4*>(tile)[i * nch + c];
      }
      __syncwarp();
    }
  }
}

// ---- NeoX rotary embedding fused with the KV fill ----
// q and k rows are rotated at their token's position (first rot_dim elements of every head:
// x = d < rot_dim/2 pairs with y = d + rot_dim/2; out_x = x cos - y sin, out_y = y cos + x sin,
// cos/sin from cos_sin_cache[pos] = [cos(rot_dim/2) | sin(rot_dim/2)]); q is rewritten in place,
// the rotated k goes straight into its cache cell (and back into `key` only if asked), v is
// scattered as in the plain fill. One pass over q, k and v instead of rotary (read+write q, k)
// followed by the fill (read k, v again). Products are formed in fp32 and rounded once.
//
// Reference counterparts: rotary_embedding_neox_kernel (3rdparty/vllm/csrc/pos_encoding_kernels.cu:7-60;
// called from parrot/engine/builtin/models/llama.py:123-129 through kernels/vllm/rotary_embed.py:10-25)
// followed by reshape_and_cache_kernel (3rdparty/vllm/csrc/cache_kernels.cu:142-182).
template <typename T> struct BitsOf { using type = uint16_t; };
template <> struct BitsOf<float> { using type = uint32_t; };

template <typename T>
__device__ __forceinline__ uint4 pack16(const float* f) {
  constexpr int kVec = ElemTraits<T>::kVec;
  uint4 out;
  T* o = reinterpret_cast<T*>(&out);
#pragma unroll
  for (int j = 0; j < kVec; ++j) o[j] = from_float<T>(f[j]);
  return out;
}

// Rotates the chunk pair (cx, cy = cx + half) of one head row; cs points at the token's cos/sin row.
template <typename T>
__device__ __forceinline__ void rotate_pair(const uint4& x, const uint4& y, const uint8_t* cs, int cx, int half_chunks,
                                            uint4& ox, uint4& oy) {
  constexpr int kVec = ElemTraits<T>::kVec;
  float fx[kVec], fy[kVec], fc[kVec], fs[kVec], rx[kVec], ry[kVec];
  unpack16<T>(x, fx);
  unpack16<T>(y, fy);
  unpack16<T>(load16(cs + cx * 16), fc);
  unpack16<T>(load16(cs + (half_chunks + cx) * 16), fs);
#pragma unroll
  for (int j = 0; j < kVec; ++j) {
    rx[j] = fx[j] * fc[j] - fy[j] * fs[j];
    ry[j] = fy[j] * fc[j] + fx[j] * fs[j];
  }
  ox = pack16<T>(rx);
  oy = pack16<T>(ry);
}

template <typename T>
__global__ void __launch_bounds__(kFillWarps * 32) rotary_fill_kernel(
    uint8_t* query, uint8_t* key, const uint8_t* value,
    uint8_t* kcache, uint8_t* vcache, const void* slots, const int is64,
    const long long* positions, const uint8_t* cos_sin, const int rot_dim,
    const long long max_pos, const long long T_tok, const int Hq, const int H, const int D, const int B,
    const long long q_stride, const long long key_stride, const long long value_stride, const long long kbs,
    const long long khs, const long long num_blocks, const int write_key_back) {
  constexpr int E = (int)sizeof(T);
  constexpr int kVec = 16 / E;
  using elem_t = typename BitsOf<T>::type;
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long t = blockIdx.x;
  pdl_wait();
  pdl_trigger();
  const int nch = D / kVec;             // 16-byte chunks per head row
  const int half = rot_dim / kVec / 2;  // chunks in each half of the rotated part
  const int units = nch - half;         // chunk pairs of the rotated part + pass-through chunks
  auto cs_row = [&](long long tok) {
    long long pos = positions[tok];
    pos = pos < 0 ? 0 : (pos >= max_pos ? max_pos - 1 : pos);  // clamped: never read outside the table
    return cos_sin + (size_t)pos * rot_dim * E;
  };

  // ---- q of this token, in place (every token, whether or not it leads a run of slots) ----
  {
    const uint8_t* cs = cs_row(t);
    for (int h = blockIdx.y * kFillWarps + warp; h < Hq; h += gridDim.y * kFillWarps) {
      uint4* row = reinterpret_cast<uint4*>(query + ((size_t)t * q_stride + (size_t)h * D) * E);
      for (int u = lane; u < half; u += 32) {
        uint4 ox, oy;
        rotate_pair<T>(load16(row + u), load16(row + u + half), cs, u, half, ox, oy);
        row[u] = ox;
        row[u + half] = oy;
      }
    }
  }

  if (kcache == nullptr) {
    // rotation only (the reference's rotary_embedding_neox): k of this token in place, no cache
    const uint8_t* cs = cs_row(t);
    for (int h = blockIdx.y * kFillWarps + warp; h < H; h += gridDim.y * kFillWarps) {
      uint4* row = reinterpret_cast<uint4*>(key + ((size_t)t * key_stride + (size_t)h * D) * E);
      for (int u = lane; u < half; u += 32) {
        uint4 ox, oy;
        rotate_pair<T>(load16(row + u), load16(row + u + half), cs, u, half, ox, oy);
        row[u] = ox;
        row[u + half] = oy;
      }
    }
    return;
  }

  // ---- k and v: the warp of a run's first token moves the whole run (as in the plain fill) ----
  const long long slot = load_slot(slots, is64, t);
  const long long prev = (t > 0) ? load_slot(slots, is64, t - 1) : -2;
  const long long next = (lane > 0 && lane < B && t + lane < T_tok) ? load_slot(slots, is64, t + lane) : -3;
  if (slot < 0) return;
  const long long blk = slot / B;
  const int off0 = (int)(slot - blk * B);
  if (blk >= num_blocks) return;
  const bool leader = (t == 0) || (prev + 1 != slot) || (off0 == 0);
  if (!leader) return;
  bool ok = (lane == 0);
  if (lane > 0 && lane < B && off0 + lane < B && t + lane < T_tok) ok = (next == slot + lane);
  const unsigned mask = __ballot_sync(0xffffffffu, ok);
  const int n = __ffs(~mask) - 1;
  const int run = (~mask == 0u) ? 32 : n;
  uint8_t* tile = smem + (size_t)warp * B * D * E;

  for (int h = blockIdx.y * kFillWarps + warp; h < H; h += gridDim.y * kFillWarps) {
    uint8_t* kt = kcache + ((size_t)blk * kbs + (size_t)h * khs) * E;
    uint8_t* vt = vcache + ((size_t)blk * kbs + (size_t)h * khs) * E;
    // K: chunk pair (token i, cx, cx + half) rotated, or pass-through chunk c >= 2 * half
    for (int idx = lane; idx < run * units; idx += 32) {
      const int i = idx / units, u = idx - i * units;
      uint4* row = reinterpret_cast<uint4*>(key + ((size_t)(t + i) * key_stride + (size_t)h * D) * E);
      uint4* cell = reinterpret_cast<uint4*>(kt) + off0 + i;
      if (u < half) {
        uint4 ox, oy;
        rotate_pair<T>(load16(row + u), load16(row + u + half), cs_row(t + i), u, half, ox, oy);
        cell[(size_t)u * B] = ox;
        cell[(size_t)(u + half) * B] = oy;
        if (write_key_back) { row[u] = ox; row[u + half] = oy; }
      } else {
        const int c = u + half;
        cell[(size_t)c * B] = load16(row + c);
      }
    }
    // V: transposed through shared memory, full blocks written with 16-byte stores
    for (int idx = lane; idx < run * nch; idx += 32) {
      const int i = idx / nch, c = idx - i * nch;
      reinterpret_cast<uint4*>(tile)[i * nch + c] = load16(value + ((size_t)(t + i) * value_stride + (size_t)h * D + c * kVec) * E);
    }
    __syncwarp();
    const elem_t* ts = reinterpret_cast<const elem_t*>(tile);
    for (int dd = lane; dd < D; dd += 32) {
      elem_t* dst = reinterpret_cast<elem_t*>(vt) + (size_t)dd * B + off0;
      if (run == B) {
        for (int v = 0; v < B / kVec; ++v) {
          elem_t tmp[kVec];
#pragma unroll
          for (int j = 0; j < kVec; ++j) tmp[j] = ts[(size_t)(v * kVec + j) * D + dd];
          reinterpret_cast<uint4*>(dst)[v] = *reinterpret_cast<const uint4*>(tmp);
        }
      } else {
        for (int i = 0; i < run; ++i) dst[i] = ts[(size_t)i * D + dd];
      }
    }
    __syncwarp();
  }
}

// KV fill at block size 16, with (ROT) or without NeoX rotation of q and k: a CTA takes 16 consecutive
// tokens and kWinHeads heads; every thread owns one (token, chunk) and walks the heads, so that the loads of
// all of them are in flight together and the cos/sin values are read once for them. q and k need no more
// than the token's own slot: neighbouring lanes are neighbouring tokens, whose cells of a block are
// neighbours too. V goes from rows to tiles [d][16 tokens]. The runs of consecutive slots that START among the
// CTA's tokens are written by it up to their end, so that a full block's sectors are written whole. Two forms:
//   long runs (prefill): two tokens of a run share a 4-byte word, so a thread reads the same chunk of both, and
//     eight lanes write one whole 32-byte row of the tile; nothing goes through shared memory. (fp32: a thread per
//     token and chunk; eight lanes are 32 bytes of a tile row.)
//   short ones (decode tokens): a warp per (token, head) with its lanes along d. Every element is a sector of its
//     own then, and the lanes of a store fall into eight 128-byte lines. (With a thread per token and chunk they fall
//     into 32, and the store unit of an SM takes a line at a time: 1024 lone tokens x 32 heads, fp16, 83 us against 49;
//     with the warp per run of the other block sizes 49.)
// Which form: by the mean length of a window's runs. Runs of five, 2000 tokens x 32 heads: fp16 37 us by runs, 53
// by elements, fp32 55 and 87; runs of three: fp16 76 and 73, fp32 85 and 114.
// What bounds it is memory. 10 842 tokens (16 prefills, 240 decodes) x 32 heads, fp16: rotary and fill
// 165 -> 114 us (4.7 TB/s of 534 MB) against a CTA per token of which fifteen of sixteen left at once; the plain
// fill of 8767 prefill tokens about 65 -> 52 us.
constexpr int kMeanRun16 = 4, kMeanRun32 = 3;  // by runs from this mean length on: 16-bit types, fp32

// Heads per CTA: one in small batches, so that the stores spread over the chip (1024 lone tokens x 32 heads 53 us with
// two heads, 49 with one); then 4 with rotation (2: 125 us for the 10 842 tokens above, 4: 118) and 2 without (4: 430 us
// with the attention behind it, 2: 426). Small is, in (window, head) pairs per SM: 16 without rotation (8192 tokens x 32
// heads in whole blocks, 111 per SM: 49 us with two, 57 with one; 2048 x 8, 7 per SM: the same) and 6 with it, where
// the heads share cos and sin (2048 tokens x 8 heads in whole blocks, 7 per SM: 6.8 us with four, 8.0 with one; 256 lone
// tokens x 32 heads, 3.5 per SM: 15.2 and 10.8).
constexpr int win_heads(bool rot, bool small) { return small ? 1 : rot ? 4 : 2; }
// The smallest batches have CTAs of their own for (q,) K and V, whose trips to memory then run beside each other, as
// long as every CTA finds an SM to itself: 64 lone tokens x 8 heads with rotation 4.8 us together, 3.7 apart; with 32
// heads, two CTAs an SM, the plain fill takes 4.5 together and 5.5 apart.
struct WinShape {
  bool small;
  unsigned roles;
};
static WinShape win_shape(long long tokens, int heads, bool rot) {
  const long long pairs = (tokens + 15) / 16 * heads;
  const int sms = sm_count(), roles = rot ? 3 : 2;
  return WinShape{pairs <= (rot ? 6 : 16) * sms, pairs * roles <= sms ? (unsigned)roles : 1u};
}

template <typename T, bool ROT, bool SMALL>
__global__ void __launch_bounds__(128) fill_window_kernel(
    uint8_t* query, uint8_t* key, const uint8_t* value,
    uint8_t* kcache, uint8_t* vcache, const void* slots, const int is64,
    const long long* positions, const uint8_t* cos_sin, const int rot_dim,
    const long long max_pos, const long long T_tok, const int Hq, const int H, const int D,
    const long long q_stride, const long long key_stride, const long long value_stride, const long long kbs,
    const long long khs, const long long num_blocks, const int write_key_back) {
  constexpr int B = 16;
  constexpr int kWinHeads = win_heads(ROT, SMALL);
  constexpr int E = (int)sizeof(T);
  constexpr int kVec = 16 / E;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long first = (long long)blockIdx.x * 16;
  const int h0 = blockIdx.y * kWinHeads;
  // the smallest batches have CTAs of their own for q, K and V (blockIdx.z)
  const bool all = !SMALL || gridDim.z == 1;
  const bool do_q = ROT && (all || blockIdx.z == 0), do_k = all || blockIdx.z == (ROT ? 1 : 0), do_v = all || blockIdx.z == (ROT ? 2 : 1);
  // resident while the kernel before this one drains: wait for it before reading anything, then let the
  // next kernel set itself up (it waits before it reads the cache)
  pdl_wait();
  pdl_trigger();
  const int nch = D / kVec;                       // 16-byte chunks per (token, head) row
  const int half = ROT ? rot_dim / kVec / 2 : 0;  // chunks in each half of the rotated part
  auto cs_row = [&](long long tok) {
    long long pos = positions[tok];
    pos = pos < 0 ? 0 : (pos >= max_pos ? max_pos - 1 : pos);  // clamped: never read outside the table
    return cos_sin + (size_t)pos * rot_dim * E;
  };
  // rotates the chunk pair u of one token's rows of this CTA's heads: dst_x / dst_y(head) say where to
  auto rotate_rows = [&](const uint8_t* row0, int heads, const uint8_t* cs, int u, auto&& store) {
    uint4 x[kWinHeads], y[kWinHeads];
#pragma unroll
    for (int k = 0; k < kWinHeads; ++k) {
      if (h0 + k < heads) {
        const uint4* row = reinterpret_cast<const uint4*>(row0 + (size_t)(h0 + k) * D * E);
        x[k] = load16(row + u);
        y[k] = load16(row + u + half);
      }
    }
    float fc[kVec], fs[kVec];
    unpack16<T>(load16(cs + u * 16), fc);
    unpack16<T>(load16(cs + (half + u) * 16), fs);
#pragma unroll
    for (int k = 0; k < kWinHeads; ++k) {
      if (h0 + k < heads) {
        float fx[kVec], fy[kVec], rx[kVec], ry[kVec];
        unpack16<T>(x[k], fx);
        unpack16<T>(y[k], fy);
#pragma unroll
        for (int j = 0; j < kVec; ++j) {
          rx[j] = fx[j] * fc[j] - fy[j] * fs[j];
          ry[j] = fy[j] * fc[j] + fx[j] * fs[j];
        }
        store(h0 + k, pack16<T>(rx), pack16<T>(ry));
      }
    }
  };

  // lane l: the slot of token first - 1 + l (negative: none, or outside the cache); asked for before q is worked on
  const long long my = first - 1 + lane;
  long long slot = (kcache != nullptr && my >= 0 && my < T_tok) ? load_slot(slots, is64, my) : -1;
  if (slot >= num_blocks * B) slot = -1;

  if (do_q) {  // q in place; with no cache k too (eight lanes: 128 contiguous bytes of a row)
    const long long tok = first + warp * 4 + (lane >> 3);
    if (tok < T_tok) {
      const uint8_t* cs = cs_row(tok);
      for (int u = lane & 7; u < half; u += 8) {
        uint8_t* qrow = query + (size_t)tok * q_stride * E;
        rotate_rows(qrow, Hq, cs, u, [&](int h, const uint4& ox, const uint4& oy) {
          uint4* row = reinterpret_cast<uint4*>(qrow + (size_t)h * D * E);
          row[u] = ox;
          row[u + half] = oy;
        });
        if (kcache == nullptr) {
          uint8_t* krow = key + (size_t)tok * key_stride * E;
          rotate_rows(krow, H, cs, u, [&](int h, const uint4& ox, const uint4& oy) {
            uint4* row = reinterpret_cast<uint4*>(krow + (size_t)h * D * E);
            row[u] = ox;
            row[u + half] = oy;
          });
        }
      }
    }
  }
  if (h0 >= H || kcache == nullptr || !(do_k || do_v)) return;

  // ---- K: token `i` of the window, chunks g, g + 8, ... ----
  const int i = (lane & 7) + 8 * (warp & 1), g = (lane >> 3) + 4 * (warp >> 1);
  const long long s_i = __shfl_sync(0xffffffffu, slot, i + 1);
  if (do_k && s_i >= 0) {
    uint8_t* krow = key + (size_t)(first + i) * key_stride * E;
    uint4* cell0 = reinterpret_cast<uint4*>(kcache + (size_t)(s_i / B) * kbs * E) + (s_i & (B - 1));
    auto cell = [&](int h) { return reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(cell0) + (size_t)h * khs * E); };
    if (ROT) {
      const uint8_t* cs = cs_row(first + i);
      for (int u = g; u < half; u += 8)
        rotate_rows(krow, H, cs, u, [&](int h, const uint4& ox, const uint4& oy) {
          cell(h)[(size_t)u * B] = ox;
          cell(h)[(size_t)(u + half) * B] = oy;
          if (write_key_back) {
            uint4* row = reinterpret_cast<uint4*>(krow + (size_t)h * D * E);
            row[u] = ox;
            row[u + half] = oy;
          }
        });
    }
    constexpr int kChunks = SMALL ? 4 : 2;  // chunks per head in flight
    for (int c0 = 2 * half + g; c0 < nch; c0 += 8 * kChunks) {
      uint4 v[kChunks][kWinHeads];
#pragma unroll
      for (int u = 0; u < kChunks; ++u)
#pragma unroll
        for (int k = 0; k < kWinHeads; ++k)
          if (c0 + 8 * u < nch && h0 + k < H) v[u][k] = load16(krow + (size_t)(h0 + k) * D * E + (c0 + 8 * u) * 16);
#pragma unroll
      for (int u = 0; u < kChunks; ++u)
#pragma unroll
        for (int k = 0; k < kWinHeads; ++k)
          if (c0 + 8 * u < nch && h0 + k < H) cell(h0 + k)[(size_t)(c0 + 8 * u) * B] = v[u][k];
    }
  }

  // ---- V: the runs that start among tokens first .. first + 15 (lanes 1 .. 16) ----
  const unsigned cont = run_continues(slot);
  const unsigned starts = ~cont & __ballot_sync(0xffffffffu, slot >= 0) & 0x1fffeu;
  if (starts == 0 || !do_v) return;
  // lanes [lo, hi) hold the tokens of those runs
  const int last = 31 - __clz(starts), lo = __ffs(starts) - 1, hi = last + run_length(cont, last);
  const bool by_runs = hi - lo >= (E == 2 ? kMeanRun16 : kMeanRun32) * __popc(starts);
  if (E == 2 && by_runs) {
    for (unsigned left = starts; left; left &= left - 1) {
      const int at = __ffs(left) - 1, run = run_length(cont, at);
      const long long s0 = __shfl_sync(0xffffffffu, slot, at);
      const int off = (int)(s0 & (B - 1));
      const int pair = lane & 7;  // positions 2 pair, 2 pair + 1 of the block
      const int ia = 2 * pair - off, ib = ia + 1;
      const bool in_a = ia >= 0 && ia < run, in_b = ib >= 0 && ib < run;
      if (!in_a && !in_b) continue;
      const uint8_t* rows = value + (size_t)(first - 1 + at + (in_a ? ia : ib)) * value_stride * E;
      const size_t next = (in_a && in_b) ? (size_t)value_stride * E : 0;
      uint8_t* tile = vcache + ((size_t)(s0 / B) * kbs + (size_t)h0 * khs) * E + pair * 4;
      for (int c = (lane >> 3) + 4 * warp; c < nch; c += 16) {
        uint4 a[kWinHeads], b[kWinHeads];
#pragma unroll
        for (int k = 0; k < kWinHeads; ++k) {
          if (h0 + k < H) {
            const uint8_t* p = rows + (size_t)(h0 + k) * D * E + c * 16;
            a[k] = load16(p);
            b[k] = load16(p + next);
          }
        }
#pragma unroll
        for (int k = 0; k < kWinHeads; ++k) {
          if (h0 + k < H) {
            uint8_t* out = tile + (size_t)k * khs * E + c * kVec * 32;
            const uint32_t av[4] = {a[k].x, a[k].y, a[k].z, a[k].w}, bv[4] = {b[k].x, b[k].y, b[k].z, b[k].w};
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const uint32_t w = __byte_perm(av[j >> 1], bv[j >> 1], (j & 1) ? 0x7632 : 0x5410);
              if (in_a && in_b) *reinterpret_cast<uint32_t*>(out + j * 32) = w;
              else *reinterpret_cast<uint16_t*>(out + j * 32 + (in_a ? 0 : 2)) = (uint16_t)(in_a ? w : w >> 16);
            }
          }
        }
      }
    }
    return;
  }
  using elem_t = typename ElemOf<E>::type;
  if (E == 4 && by_runs) {  // eight lanes are eight tokens: 32 contiguous bytes of a tile row
    for (int base = lo; base < hi; base += 16) {
      const int l = base + i;
      const long long s = __shfl_sync(0xffffffffu, slot, min(l, 31));
      if (l >= hi || s < 0) continue;
      const uint8_t* row = value + (size_t)(first - 1 + l) * value_stride * E;
      uint8_t* tile = vcache + ((size_t)(s / B) * kbs + (size_t)h0 * khs) * E + (s & (B - 1)) * E;
      for (int c = g; c < nch; c += 8) {
        uint4 v[kWinHeads];
#pragma unroll
        for (int k = 0; k < kWinHeads; ++k)
          if (h0 + k < H) v[k] = load16(row + (size_t)(h0 + k) * D * E + c * 16);
#pragma unroll
        for (int k = 0; k < kWinHeads; ++k) {
          if (h0 + k < H) {
            const elem_t* e = reinterpret_cast<const elem_t*>(&v[k]);
            uint8_t* out = tile + (size_t)k * khs * E + (size_t)c * 16 * B;
#pragma unroll
            for (int j = 0; j < kVec; ++j) *reinterpret_cast<elem_t*>(out + j * B * E) = e[j];
          }
        }
      }
    }
    return;
  }
  // a warp per (token, head), four of them at a time: all their loads in flight
  constexpr int kBatch = 4, kSteps = 4;  // kSteps x 32 elements of a row
  const int n_pairs = (hi - lo) * kWinHeads;
  for (int p0 = warp; p0 < n_pairs; p0 += 4 * kBatch) {
    const uint8_t* row[kBatch];
    uint8_t* tile[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int p = min(p0 + 4 * u, n_pairs - 1);
      const int l = lo + p / kWinHeads, h = h0 + p % kWinHeads;
      const long long s = __shfl_sync(0xffffffffu, slot, l);
      row[u] = (p0 + 4 * u < n_pairs && s >= 0 && h < H) ? value + ((size_t)(first - 1 + l) * value_stride + (size_t)h * D) * E : nullptr;
      tile[u] = vcache + ((size_t)(s / B) * kbs + (size_t)h * khs + (s & (B - 1))) * E;
    }
    for (int d0 = lane; d0 < D; d0 += kSteps * 32) {
      elem_t e[kBatch][kSteps];
#pragma unroll
      for (int u = 0; u < kBatch; ++u)
#pragma unroll
        for (int r = 0; r < kSteps; ++r)
          if (row[u] && d0 + r * 32 < D) e[u][r] = load_elem<elem_t>(row[u] + (d0 + r * 32) * E);
#pragma unroll
      for (int u = 0; u < kBatch; ++u)
#pragma unroll
        for (int r = 0; r < kSteps; ++r)
          if (row[u] && d0 + r * 32 < D) *reinterpret_cast<elem_t*>(tile[u] + (size_t)(d0 + r * 32) * B * E) = e[u][r];
    }
  }
}

// dest[dest_idx[i]] = cache row at slot src_slots[i], block size 16: a CTA takes 16 entries of the list and a few
// heads. What bounds it is memory.
//   K: a warp per head, a pair of lanes per entry: 16-byte chunks, two neighbouring ones of a token per
//     instruction, so that reads and writes are whole sectors (consecutive slots: neighbouring cells).
//   V: a tile's 32-byte rows hold 16 tokens, so a warp per (token, head) fetches a tile sixteen times (from L2)
//     in two-byte loads. The runs of consecutive slots that start among the entries are read once, a warp per (run,
//     head), with 16-byte loads, and turned in shared memory. Short runs (scattered slots): a warp per (token, head)
//     after all, four of them at a time, because a whole tile for a few tokens is work in vain (2000 tokens x 32
//     heads, runs of eleven: fp16 11.8 us, by elements 16; of five 16 and 20, fp32 35 and 52; of three 22 and 19).
// K and V of 8090 tokens x 32 heads x 128 in whole blocks (fp16, 265 MB read and written): 127 -> 57 us, 4.6 TB/s.
// 1024 scattered tokens x 32 heads: K 5.8 us, V 13.6 (a warp per run for all of them: 18 and 34; a warp per (token,
// head): 8.8 and 13.1). In fp32 V takes 70, and 33 with a warp per (token, head) each in a CTA of their own.
constexpr int kMeanRunMove = 4;  // V moves by runs from this mean length on

template <int E, bool IS_V>
__global__ void __launch_bounds__(128) move_runs_kernel(
    const uint8_t* cache, uint8_t* dest, const long long* src_slots,
    const long long* dest_idx, const long long n, const int H, const int heads_per_cta, const int D,
    const long long dest_stride, const long long kbs, const long long khs, const long long num_blocks,
    const long long dest_rows, int* status) {
  constexpr int B = 16;
  constexpr int kVec = 16 / E;
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long first = (long long)blockIdx.x * 16;
  const int h0 = blockIdx.y * heads_per_cta, nh = min(heads_per_cta, H - h0);
  pdl_wait();
  pdl_trigger();
  const long long my = first - 1 + lane;
  const bool in_list = my >= 0 && my < n;
  long long slot = in_list ? src_slots[my] : -1;
  long long di = in_list ? dest_idx[my] : -1;
  if (in_list && (slot < 0 || slot >= num_blocks * B || di < 0 || di >= dest_rows)) {
    if (status) atomicMax(status, kStatusBadIndex);
    if (slot < 0 || slot >= num_blocks * B) slot = -1;
    di = -1;  // this entry is skipped
  }
  if (!IS_V) {
    const int nch = D / kVec;
    const long long s = __shfl_sync(0xffffffffu, slot, 1 + (lane >> 1)), to = __shfl_sync(0xffffffffu, di, 1 + (lane >> 1));
    if (s < 0 || to < 0) return;
    for (int h = h0 + warp; h < h0 + nh; h += 4) {
      const uint4* cell = reinterpret_cast<const uint4*>(cache + ((size_t)(s >> 4) * kbs + (size_t)h * khs) * E) + (s & 15);
      uint4* row = reinterpret_cast<uint4*>(dest + ((size_t)to * dest_stride + (size_t)h * D) * E);
      for (int base = lane & 1; base < nch; base += 16) {
        uint4 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (base + 2 * u < nch) v[u] = load16(cell + (size_t)(base + 2 * u) * B);
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (base + 2 * u < nch) row[base + 2 * u] = v[u];
      }
    }
    return;
  }
  const unsigned cont = run_continues(slot);
  const unsigned starts = ~cont & __ballot_sync(0xffffffffu, slot >= 0) & 0x1fffeu;  // entries first .. first + 15
  if (starts == 0) return;
  const int n_runs = __popc(starts);
  using elem_t = typename ElemOf<E>::type;
  // lanes [lo, hi) hold the entries of those runs
  const int last = 31 - __clz(starts), lo = __ffs(starts) - 1, hi = last + run_length(cont, last);
  if (hi - lo < kMeanRunMove * n_runs) {
    constexpr int kBatch = 4, kSteps = 4;  // kSteps x 32 elements of a row
    const int n_pairs = (hi - lo) * nh;
    for (int p0 = warp; p0 < n_pairs; p0 += 4 * kBatch) {
      const uint8_t* src[kBatch];
      uint8_t* row[kBatch];
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const int q = min(p0 + 4 * u, n_pairs - 1), l = lo + q / nh, h = h0 + q % nh;
        const long long s = __shfl_sync(0xffffffffu, slot, l), to = __shfl_sync(0xffffffffu, di, l);
        src[u] = (p0 + 4 * u < n_pairs && s >= 0 && to >= 0) ? cache + ((size_t)(s >> 4) * kbs + (size_t)h * khs + (s & 15)) * E : nullptr;
        row[u] = dest + ((size_t)to * dest_stride + (size_t)h * D) * E;
      }
      for (int d0 = lane; d0 < D; d0 += kSteps * 32) {
        elem_t e[kBatch][kSteps];
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
#pragma unroll
          for (int r = 0; r < kSteps; ++r)
            if (src[u] && d0 + r * 32 < D) e[u][r] = load_elem<elem_t>(src[u] + (size_t)(d0 + r * 32) * B * E);
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
#pragma unroll
          for (int r = 0; r < kSteps; ++r)
            if (src[u] && d0 + r * 32 < D) reinterpret_cast<elem_t*>(row[u])[d0 + r * 32] = e[u][r];
      }
    }
    return;
  }
  const int words = D * E / 4, pitch = words + 2;  // (two words of padding spread the columns over the banks)
  uint32_t* tile = reinterpret_cast<uint32_t*>(smem) + (size_t)warp * B * pitch;
  for (int task = warp; task < n_runs * nh; task += 4) {
    const int r = task / nh, h = h0 + (task - r * nh);
    const int at = __fns(starts, 0, r + 1);
    const int run = run_length(cont, at);
    const long long s0 = __shfl_sync(0xffffffffu, slot, at);
    const int off = (int)(s0 & 15);
    const uint8_t* src = cache + ((size_t)(s0 >> 4) * kbs + (size_t)h * khs) * E;
    // 16-byte chunk: kVec tokens of one d; chunks without a token of the run are left out
    if (E == 2) {  // rows d, d + 1 and eight tokens: words (token, d pair)
      const int half = lane & 1;
      if (half * 8 < off + run && half * 8 + 8 > off) {
#pragma unroll 4
        for (int p = lane >> 1; p < D / 2; p += 16) {
          const uint4 a = load16(src + (size_t)p * 64 + half * 16);
          const uint4 b = load16(src + (size_t)p * 64 + 32 + half * 16);
          const uint32_t av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            tile[(half * 8 + 2 * j) * pitch + p] = __byte_perm(av[j], bv[j], 0x5410);
            tile[(half * 8 + 2 * j + 1) * pitch + p] = __byte_perm(av[j], bv[j], 0x7632);
          }
        }
      }
    } else {
      const int quarter = lane & 3;
      if (quarter * 4 < off + run && quarter * 4 + 4 > off) {
#pragma unroll 4
        for (int d = lane >> 2; d < D; d += 8) {
          const uint4 a = load16(src + (size_t)d * 64 + quarter * 16);
          tile[(quarter * 4 + 0) * pitch + d] = a.x;
          tile[(quarter * 4 + 1) * pitch + d] = a.y;
          tile[(quarter * 4 + 2) * pitch + d] = a.z;
          tile[(quarter * 4 + 3) * pitch + d] = a.w;
        }
      }
    }
    __syncwarp();
    for (int i = 0; i < run; ++i) {
      const long long to = __shfl_sync(0xffffffffu, di, at + i);
      if (to < 0) continue;
      uint2* row = reinterpret_cast<uint2*>(dest + ((size_t)to * dest_stride + (size_t)h * D) * E);
      const uint2* from = reinterpret_cast<const uint2*>(tile + (off + i) * pitch);
      for (int w = lane; w < words / 2; w += 32) row[w] = from[w];
    }
    __syncwarp();
  }
}

// dest[dest_idx[i]] = cache row at slot src_slots[i] for any block size; one warp per (token, head).
template <int E, bool IS_V>
__global__ void __launch_bounds__(128) move_from_cache_kernel(
    const uint8_t* __restrict__ cache, uint8_t* __restrict__ dest, const long long* __restrict__ src_slots,
    const long long* __restrict__ dest_idx, const long long n, const int H, const int D, const int B,
    const long long dest_stride, const long long kbs, const long long khs, const long long num_blocks,
    const long long dest_rows, int* __restrict__ status) {
  using elem_t = typename ElemOf<E>::type;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long gw = (long long)blockIdx.x * 4 + warp;
  if (gw >= n * H) return;
  const long long i = gw / H;
  const int h = (int)(gw - i * H);
  const long long slot = src_slots[i], di = dest_idx[i];
  const long long blk = slot / B;
  const int off = (int)(slot - blk * B);
  if (slot < 0 || blk >= num_blocks || di < 0 || di >= dest_rows) {
    if (lane == 0 && status) atomicMax(status, kStatusBadIndex);
    return;
  }
  constexpr int kVec = 16 / E;
  const uint8_t* tile = cache + ((size_t)blk * kbs + (size_t)h * khs) * E;
  uint8_t* row = dest + ((size_t)di * dest_stride + (size_t)h * D) * E;
  if (IS_V) {
    for (int dd = lane; dd < D; dd += 32)
      reinterpret_cast<elem_t*>(row)[dd] = reinterpret_cast<const elem_t*>(tile)[(size_t)dd * B + off];
  } else {
    for (int c = lane; c < D / kVec; c += 32)
      reinterpret_cast<uint4*>(row)[c] = reinterpret_cast<const uint4*>(tile)[(size_t)c * B + off];
  }
}

// dest[dest_idx[i]] = src[src_idx[i]] over rows of row_bytes bytes; one warp per row.
template <bool VEC16>
__global__ void __launch_bounds__(128) move_rows_kernel(
    const uint8_t* __restrict__ src, uint8_t* __restrict__ dest, const long long* __restrict__ src_idx,
    const long long* __restrict__ dest_idx, const long long n, const long long row_bytes,
    const long long src_stride, const long long dest_stride, const long long src_rows,
    const long long dest_rows, int* __restrict__ status) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long i = (long long)blockIdx.x * 4 + warp;
  if (i >= n) return;
  const long long si = src_idx[i], di = dest_idx[i];
  if (si < 0 || si >= src_rows || di < 0 || di >= dest_rows) {
    if (lane == 0 && status) atomicMax(status, kStatusBadIndex);
    return;
  }
  const uint8_t* s = src + (size_t)si * src_stride;
  uint8_t* t = dest + (size_t)di * dest_stride;
  if (VEC16) {
    for (long long b = lane; b < row_bytes / 16; b += 32)
      reinterpret_cast<uint4*>(t)[b] = reinterpret_cast<const uint4*>(s)[b];
  } else {
    for (long long b = lane; b < row_bytes; b += 32) t[b] = s[b];
  }
}

thread_local char g_err[256] = "";

}  // namespace

void set_cuda_error(cudaError_t e) {
  const char* s = cudaGetErrorString(e);
  int i = 0;
  for (; s && s[i] && i < 255; ++i) g_err[i] = s[i];
  g_err[i] = 0;
}
const char* last_cuda_error() { return g_err; }

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

static int kv_run_launch(bool fill, void* key, void* value, void* kcache, void* vcache, const void* slots,
                         int is64, long long T, int H, int D, int B, long long ks, long long vs,
                         long long kbs, long long khs, long long num_blocks, int dtype, cudaStream_t s) {
  if (T < 0 || H <= 0 || D <= 0 || num_blocks < 0) return PB_ERR_INVALID_ARG;
  if (T == 0) return PB_OK;
  if (!key || !value || !kcache || !vcache || !slots) return PB_ERR_INVALID_ARG;
  if (dtype != PB_F32 && dtype != PB_F16 && dtype != PB_BF16) return PB_ERR_UNSUPPORTED;
  const int E = (dtype == PB_F32) ? 4 : 2;
  const int vec = 16 / E;
  if (B != 8 && B != 16 && B != 32) return PB_ERR_UNSUPPORTED;
  if (D % vec != 0 || D > 256) return PB_ERR_UNSUPPORTED;
  if (!aligned16(key) || !aligned16(value) || !aligned16(kcache) || !aligned16(vcache)) return PB_ERR_INVALID_ARG;
  if (ks % vec || vs % vec || kbs % vec || khs % vec) return PB_ERR_INVALID_ARG;
  if (T > 0x7fffffffll) return PB_ERR_INVALID_ARG;
  if (fill && B == 16) {  // the engine's block size; the others take the warp per (run, head) below
    const WinShape shape = win_shape(T, H, false);
    const bool small = shape.small;
    const int per = win_heads(false, small);
    const dim3 grid((unsigned)((T + 15) / 16), (unsigned)((H + per - 1) / per), shape.roles);
    const long long* no_pos = nullptr;
    const uint8_t* no_table = nullptr;
    auto launch = [&](auto kfn) {
      return launch_kernel(kfn, grid, dim3(128), 0, s, true, (uint8_t*)nullptr, (uint8_t*)key, (const uint8_t*)value, (uint8_t*)kcache,
                           (uint8_t*)vcache, slots, is64, no_pos, no_table, 0, 0ll, T, 0, H, D, 0ll, ks, vs, kbs, khs, num_blocks, 0);
    };
    const cudaError_t err = E == 2 ? (small ? launch(fill_window_kernel<__half, false, true>) : launch(fill_window_kernel<__half, false, false>))
                                   : (small ? launch(fill_window_kernel<float, false, true>) : launch(fill_window_kernel<float, false, false>));
    if (err != cudaSuccess) { set_cuda_error(err); return PB_ERR_LAUNCH; }
    return PB_OK;
  }
  const size_t smem = (size_t)kFillWarps * B * D * E;
  // few tokens (decode): spread the heads over more CTAs; many tokens (prefill): at most four CTAs per token
  unsigned hgroups = (unsigned)((H + kFillWarps - 1) / kFillWarps);
  if (T >= 2048 && hgroups > 4) hgroups = 4;
  cudaError_t e = cudaSuccess;
#define PB_KV_RUN(EE, FF)                                                                              \
  do {                                                                                                 \
    auto kfn = kv_run_kernel<EE, FF>;                                                                  \
    if (smem > 48 * 1024) e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    if (e == cudaSuccess) {                                                                            \
      e = launch_kernel(kfn, dim3((unsigned)T, hgroups), dim3(kFillWarps * 32), smem, s, FF,                       \
                        (uint8_t*)key, (uint8_t*)value, (uint8_t*)kcache, (uint8_t*)vcache, slots, is64, T, H, D, B, \
                        ks, vs, kbs, khs, num_blocks, (int*)nullptr);                                  \
    }                                                                                                  \
  } while (0)
  if (E == 2) { if (fill) PB_KV_RUN(2, true); else PB_KV_RUN(2, false); }
  else { if (fill) PB_KV_RUN(4, true); else PB_KV_RUN(4, false); }
#undef PB_KV_RUN
  if (e != cudaSuccess) { set_cuda_error(e); return PB_ERR_LAUNCH; }
  return PB_OK;
}

template <typename T>
static cudaError_t rotary_fill_launch_t(void* q, void* k, const void* v, void* kc, void* vc, const void* slots, int is64,
                                        const int64_t* positions, const void* cos_sin, int rot_dim, long long max_pos,
                                        long long T_tok, int Hq, int H, int D, int B, long long qs, long long ks,
                                        long long vs, long long kbs, long long khs, long long num_blocks, int write_back,
                                        cudaStream_t s) {
  if (B == 16) {  // the engine's block size (and rotation without a cache)
    const int heads = Hq > H ? Hq : H;
    const WinShape shape = win_shape(T_tok, heads, true);
    const bool small = shape.small;
    const int per = win_heads(true, small);
    const dim3 win((unsigned)((T_tok + 15) / 16), (unsigned)((heads + per - 1) / per), kc ? shape.roles : 1u);
    auto kfn = small ? fill_window_kernel<T, true, true> : fill_window_kernel<T, true, false>;
    return launch_kernel(kfn, win, dim3(128), 0, s, true, (uint8_t*)q, (uint8_t*)k, (const uint8_t*)v, (uint8_t*)kc, (uint8_t*)vc,
                         slots, is64, (const long long*)positions, (const uint8_t*)cos_sin, rot_dim, max_pos, T_tok, Hq, H, D, qs, ks,
                         vs, kbs, khs, num_blocks, write_back);
  }
  const size_t smem = (size_t)kFillWarps * B * D * sizeof(T);
  auto kfn = rotary_fill_kernel<T>;
  cudaError_t e = cudaSuccess;
  if (smem > 48 * 1024) e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int hmax = Hq > H ? Hq : H;
  unsigned hgroups = (unsigned)((hmax + kFillWarps - 1) / kFillWarps);
  if (T_tok >= 2048 && hgroups > 4) hgroups = 4;  // many tokens: four CTAs per token measured best (1, 2, 4, 8 tried)
  return launch_kernel(kfn, dim3((unsigned)T_tok, hgroups), dim3(kFillWarps * 32), smem, s, true,
                       (uint8_t*)q, (uint8_t*)k, (const uint8_t*)v, (uint8_t*)kc, (uint8_t*)vc, slots, is64,
                       (const long long*)positions, (const uint8_t*)cos_sin, rot_dim, max_pos, T_tok, Hq, H, D, B, qs, ks,
                       vs, kbs, khs, num_blocks, write_back);
}

}  // namespace pb

extern "C" {

int pb_reshape_and_cache(const void* key, const void* value, void* key_cache, void* value_cache,
                         const void* slot_mapping, int32_t slot_is_i64, int64_t num_tokens,
                         int32_t num_heads, int32_t head_size, int32_t block_size, int64_t key_stride,
                         int64_t value_stride, int64_t kv_block_stride, int64_t kv_head_stride,
                         int64_t num_blocks, int32_t dtype, void* stream) {
  return pb::kv_run_launch(true, const_cast<void*>(key), const_cast<void*>(value), key_cache, value_cache,
                           slot_mapping, slot_is_i64, num_tokens, num_heads, head_size, block_size,
                           key_stride, value_stride, kv_block_stride, kv_head_stride, num_blocks, dtype,
                           static_cast<cudaStream_t>(stream));
}

int pb_rotary_reshape_and_cache(void* query, void* key, const void* value, void* key_cache, void* value_cache,
                                const void* slot_mapping, int32_t slot_is_i64, const int64_t* positions,
                                const void* cos_sin_cache, int32_t rot_dim, int64_t max_position, int64_t num_tokens,
                                int32_t num_heads, int32_t num_kv_heads, int32_t head_size, int32_t block_size,
                                int64_t query_stride, int64_t key_stride, int64_t value_stride,
                                int64_t kv_block_stride, int64_t kv_head_stride, int64_t num_blocks,
                                int32_t write_key_back, int32_t dtype, void* stream) {
  if (num_tokens == 0) return PB_OK;
  const bool rotate_only = (key_cache == nullptr);  // q and k rotated in place, nothing cached
  if (!query || !key || !positions || !cos_sin_cache) return PB_ERR_INVALID_ARG;
  if (!rotate_only && (!value || !value_cache || !slot_mapping)) return PB_ERR_INVALID_ARG;
  if (num_tokens < 0 || num_tokens > 0x7fffffffll || num_heads <= 0 || num_kv_heads <= 0 || max_position <= 0)
    return PB_ERR_INVALID_ARG;
  if (dtype != PB_F32 && dtype != PB_F16 && dtype != PB_BF16) return PB_ERR_UNSUPPORTED;
  const int E = (dtype == PB_F32) ? 4 : 2;
  const int vec = 16 / E;
  if (block_size != 8 && block_size != 16 && block_size != 32) return PB_ERR_UNSUPPORTED;
  if (head_size % vec != 0 || head_size > 256) return PB_ERR_UNSUPPORTED;
  // both halves of the rotated part must be whole 16-byte chunks
  if (rot_dim <= 0 || rot_dim > head_size || rot_dim % (2 * vec) != 0) return PB_ERR_UNSUPPORTED;
  if (!pb::aligned16(query) || !pb::aligned16(key) || !pb::aligned16(cos_sin_cache)) return PB_ERR_INVALID_ARG;
  if (query_stride % vec || key_stride % vec) return PB_ERR_INVALID_ARG;
  if (!rotate_only) {
    if (!pb::aligned16(value) || !pb::aligned16(key_cache) || !pb::aligned16(value_cache)) return PB_ERR_INVALID_ARG;
    if (value_stride % vec || kv_block_stride % vec || kv_head_stride % vec || num_blocks <= 0) return PB_ERR_INVALID_ARG;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e;
#define PB_ROT(TT)                                                                                              \
  e = pb::rotary_fill_launch_t<TT>(query, key, value, key_cache, value_cache, slot_mapping, slot_is_i64, positions, \
                                   cos_sin_cache, rot_dim, max_position, num_tokens, num_heads, num_kv_heads,   \
                                   head_size, block_size, query_stride, key_stride, value_stride, kv_block_stride, \
                                   kv_head_stride, num_blocks, write_key_back, s)
  if (dtype == PB_F16) PB_ROT(__half);
  else if (dtype == PB_BF16) PB_ROT(__nv_bfloat16);
  else PB_ROT(float);
#undef PB_ROT
  if (e != cudaSuccess) { pb::set_cuda_error(e); return PB_ERR_LAUNCH; }
  return PB_OK;
}

int pb_gather_cached_kv(void* key, void* value, const void* key_cache, const void* value_cache,
                        const void* slot_mapping, int32_t slot_is_i64, int64_t num_tokens,
                        int32_t num_heads, int32_t head_size, int32_t block_size, int64_t key_stride,
                        int64_t value_stride, int64_t kv_block_stride, int64_t kv_head_stride,
                        int64_t num_blocks, int32_t dtype, void* stream) {
  return pb::kv_run_launch(false, key, value, const_cast<void*>(key_cache), const_cast<void*>(value_cache),
                           slot_mapping, slot_is_i64, num_tokens, num_heads, head_size, block_size,
                           key_stride, value_stride, kv_block_stride, kv_head_stride, num_blocks, dtype,
                           static_cast<cudaStream_t>(stream));
}

int pb_move_tokens_from_blocked_cache(const void* cache, void* dest, const int64_t* src_slots,
                                      const int64_t* dest_indices, int64_t num_tokens, int32_t is_value,
                                      int32_t num_heads, int32_t head_size, int32_t block_size,
                                      int64_t dest_stride, int64_t kv_block_stride, int64_t kv_head_stride,
                                      int64_t num_blocks, int64_t dest_rows, int32_t dtype, void* stream) {
  using namespace pb;
  if (num_tokens < 0 || num_heads <= 0 || head_size <= 0) return PB_ERR_INVALID_ARG;
  if (num_tokens == 0) return PB_OK;
  if (!cache || !dest || !src_slots || !dest_indices) return PB_ERR_INVALID_ARG;
  if (dtype != PB_F32 && dtype != PB_F16 && dtype != PB_BF16) return PB_ERR_UNSUPPORTED;
  const int E = (dtype == PB_F32) ? 4 : 2;
  const int vec = 16 / E;
  if (block_size <= 0 || head_size % vec) return PB_ERR_UNSUPPORTED;
  if (!aligned16(cache) || !aligned16(dest) || dest_stride % vec || kv_block_stride % vec ||
      kv_head_stride % vec)
    return PB_ERR_INVALID_ARG;
  // Block size 16, the size of the engine's caches: a CTA per 16 entries (comment of the kernel) and four heads,
  // one per warp (eight: 69 us instead of 57 for K and V of 8090 tokens x 32 heads). A short list is bound by
  // latency, and there a warp per (token, head) is as fast or faster: V up to 8192 pairs (256 tokens x 32 heads in
  // whole blocks 4.5 us against 4.8, 16 tokens 2.4 against 4.7; 2048 x 8 heads 6.4 against 5.1), K up to 4096 (64
  // tokens x 32 heads in fp32 2.8 against 3.7, 256 tokens 4.2 against 3.8). Head sizes beyond 256 and other block
  // sizes take that kernel for everything.
  if (block_size == 16 && head_size <= 256 && num_tokens * num_heads > (is_value ? 8192 : 4096)) {
    const int heads_per_cta = 4;
    const dim3 runs_grid((unsigned)((num_tokens + 15) / 16), (unsigned)((num_heads + heads_per_cta - 1) / heads_per_cta));
    const size_t smem = is_value ? (size_t)4 * 16 * (head_size * E / 4 + 2) * 4 : 0;
    cudaStream_t on = static_cast<cudaStream_t>(stream);
    cudaError_t err = cudaSuccess;
#define PB_MOVE_RUNS(EE, VV)                                                                                          \
  do {                                                                                                                \
    auto kfn = move_runs_kernel<EE, VV>;                                                                              \
    if (smem > 48 * 1024) err = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);    \
    if (err == cudaSuccess)                                                                                           \
      err = launch_kernel(kfn, runs_grid, dim3(128), smem, on, true,  (const uint8_t*)cache, (uint8_t*)dest,          \
                          (const long long*)src_slots, (const long long*)dest_indices, num_tokens, num_heads,         \
                          heads_per_cta, head_size, dest_stride, kv_block_stride, kv_head_stride, num_blocks,         \
                          dest_rows, (int*)nullptr);                                                                  \
  } while (0)
    if (E == 2) { if (is_value) PB_MOVE_RUNS(2, true); else PB_MOVE_RUNS(2, false); }
    else { if (is_value) PB_MOVE_RUNS(4, true); else PB_MOVE_RUNS(4, false); }
#undef PB_MOVE_RUNS
    if (err != cudaSuccess) { set_cuda_error(err); return PB_ERR_LAUNCH; }
    return PB_OK;
  }
  const long long warps = (long long)num_tokens * num_heads;
  const unsigned grid = (unsigned)((warps + 3) / 4);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
#define PB_MOVE(EE, VV)                                                                               \
  move_from_cache_kernel<EE, VV><<<grid, 128, 0, s>>>(                                                \
      (const uint8_t*)cache, (uint8_t*)dest, (const long long*)src_slots, (const long long*)dest_indices, \
      num_tokens, num_heads, head_size, block_size, dest_stride, kv_block_stride, kv_head_stride,     \
      num_blocks, dest_rows, nullptr)
  if (E == 2) { if (is_value) PB_MOVE(2, true); else PB_MOVE(2, false); }
  else { if (is_value) PB_MOVE(4, true); else PB_MOVE(4, false); }
#undef PB_MOVE
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_cuda_error(e); return PB_ERR_LAUNCH; }
  return PB_OK;
}

int pb_discontinuous_move_tokens(const void* src, void* dest, const int64_t* src_indices,
                                 const int64_t* dest_indices, int64_t num_tokens, int64_t row_bytes,
                                 int64_t src_stride_bytes, int64_t dest_stride_bytes, int64_t src_rows,
                                 int64_t dest_rows, void* stream) {
  using namespace pb;
  if (num_tokens < 0 || row_bytes < 0) return PB_ERR_INVALID_ARG;
  if (num_tokens == 0 || row_bytes == 0) return PB_OK;
  if (!src || !dest || !src_indices || !dest_indices) return PB_ERR_INVALID_ARG;
  const bool vec = aligned16(src) && aligned16(dest) && row_bytes % 16 == 0 && src_stride_bytes % 16 == 0 &&
                   dest_stride_bytes % 16 == 0;
  const unsigned grid = (unsigned)((num_tokens + 3) / 4);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (vec)
    move_rows_kernel<true><<<grid, 128, 0, s>>>((const uint8_t*)src, (uint8_t*)dest, (const long long*)src_indices,
                                                (const long long*)dest_indices, num_tokens, row_bytes,
                                                src_stride_bytes, dest_stride_bytes, src_rows, dest_rows, nullptr);
  else
    move_rows_kernel<false><<<grid, 128, 0, s>>>((const uint8_t*)src, (uint8_t*)dest, (const long long*)src_indices,
                                                 (const long long*)dest_indices, num_tokens, row_bytes,
                                                 src_stride_bytes, dest_stride_bytes, src_rows, dest_rows, nullptr);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_cuda_error(e); return PB_ERR_LAUNCH; }
  return PB_OK;
}

}  // extern "C"
