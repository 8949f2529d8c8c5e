// Log-sum-exp merge of the partial results of one (row, head): prefix chunks, suffix chunks and,
// in LOAD mode, the caller's earlier partial held in out / qk_max / exp_sum.
//
// Algebra (base-2 domain): partial i carries (acc_i, m_i, l_i) with acc_i un-normalised;
// M = max m_i, w_i = 2^(m_i - M), out = sum w_i acc_i / sum w_i l_i. Associative, so the order
// of the partials does not matter.
//
// Reference counterparts: _reduce_kernel (parrot/engine/builtin/kernels/shared_flash_decoding.py:137-199)
// and the in-place merge tail of single_query_cached_kv_post_attention_kernel
// (csrc/attention/attention_post_kernels.cu:321-340).
#include "common.cuh"

namespace pb {
namespace {

constexpr int kMergeWarps = 4;
constexpr int kPairLanes = 16;                 // lanes that share one (row, head)
constexpr int kPairsPerWarp = 32 / kPairLanes;  // two (row, head) pairs per warp: twice the loads in flight
constexpr int kPairs = kMergeWarps * kPairsPerWarp;  // heads a CTA works on at once
constexpr int kMaxHeadsPerCta = kMergeWarps * 32;    // one thread each finds a head's partials
constexpr int kManyRows = 1024;                      // prefill rows from which a CTA walks up to kMaxHeadsPerCta heads of a row

// dense_cta_of_tile without a 64-bit division (a routine of some hundred instructions, and every (row, head) asks
// twice): the quotient is at most kMaxSMs, so an estimate in fp32 is off by one at most, and the remainder says so.
__device__ __forceinline__ int cta_of_tile(long long g, long long total, int ctas) {
  const int c = dense_active_ctas(total, ctas);
  const long long num = (g + 1) * c + total - 1;
  int q = (int)__fdividef((float)num, (float)total);
  const long long rest = num - q * total;
  q += rest >= total ? 1 : rest < 0 ? -1 : 0;
  return q - 1;
}

// Partials of one (row, head): [prefix][causal segment][suffix][outer prefix]; a dense stage leaves one partial per
// CTA that touched the (row tile, head), the single-query kernel one per chunk (suffix: info.nsc).
struct PartCounts {
  int prefix, segment, outer;
  bool direct;  // finished by the dense kernel (its only partial, held whole by one CTA): nothing to merge
};
__device__ __forceinline__ PartCounts count_parts(const AttnDev& d, const RowInfo& info, long long total, int dctas, int head) {
  auto dense_parts = [&](int dn) {
    const int nt = d.dn_items[dn].nt, fixed = d.dn_items[dn].fixed;
    const long long g0 = (long long)d.dn_items[dn].tile_base + (long long)head * (fixed + nt) + fixed;
    return cta_of_tile(g0 + nt - 1, total, dctas) - cta_of_tile(g0, total, dctas) + 1;
  };
  PartCounts p;
  p.prefix = (info.dn >= 0) ? dense_parts(info.dn) : info.np_sq;
  p.segment = (info.seg_dn >= 0) ? dense_parts(info.seg_dn) : info.nc_sq;
  p.outer = (info.odn >= 0) ? dense_parts(info.odn) : info.onp_sq;
  const int only = (info.dn >= 0 && p.prefix == 1 && p.segment == 0)       ? info.dn
                   : (info.seg_dn >= 0 && p.segment == 1 && p.prefix == 0) ? info.seg_dn
                                                                           : -1;
  p.direct = only >= 0 && info.nsc == 0 && p.outer == 0 && dense_direct_ok(d, d.dn_items[only]);
  return p;
}

// A call whose kernels recorded a fault (a wait that ran out, an index outside the cache, a list
// that did not fit) has results that cannot be trusted: every output row becomes NaN, so that the
// fault cannot pass unnoticed into the sampler even if nobody reads the status word.
__device__ __forceinline__ bool call_failed(const AttnDev& d) { return __ldcg(&d.hdr[kHdrStatus]) != kStatusOk; }

// Merges the partials of (row, head); the kPairLanes lanes of a (row, head) call it together, both halves of a warp
// in lockstep (active == false: a half without work).
template <typename T, int D>
__device__ __forceinline__ void merge_one(const AttnDev& d, const int row, const int head, const long long idx, const bool active,
                                          const int nsc, const PartCounts& parts, const bool poison) {
  const int sub = (threadIdx.x & 31) % kPairLanes;  // position inside the pair's lane group
  const int np = parts.prefix, nc = parts.segment;
  const int n = (active && !parts.direct) ? np + nc + nsc + parts.outer : 0;
  int n_warp = n;  // the two pairs of a warp walk their partials in lockstep
#pragma unroll
  for (int o = kPairLanes; o < 32; o <<= 1) n_warp = max(n_warp, __shfl_xor_sync(0xffffffffu, n_warp, o));
  constexpr int kVecs = D / 4;                                     // float4 per partial row
  constexpr int kPer = (kVecs + kPairLanes - 1) / kPairLanes;      // float4 per lane
  auto part_of = [&](int j) {  // partial ranges of a row: [prefix][segment][suffix][outer prefix]
    if (j < np) return j;
    if (j < np + nc) return d.pparts + (j - np);
    if (j < np + nc + nsc) return d.pparts + d.cparts + (j - np - nc);
    return d.pparts + d.cparts + d.sparts + (j - np - nc - nsc);
  };

  const bool load_prev = (d.stats_mode & PB_STATS_LOAD) != 0;
  float m_prev = -INFINITY, l_prev = 0.f;
  if (load_prev && active) {
    m_prev = d.qk_max[idx];
    l_prev = d.exp_sum[idx];
    if (!(l_prev > 0.f)) { l_prev = 0.f; m_prev = -INFINITY; }
  }

  // pass 1: global maximum (lane j of the pair reads the statistics of partial j; with at most
  // kPairLanes partials, the usual case, they stay in registers and are not read again)
  float M = m_prev;
  float2 ml0 = make_float2(-INFINITY, 0.f);
  if (sub < n) ml0 = d.ml[partial_slot(d, row, part_of(sub), head)];
  M = fmaxf(M, ml0.x);
  for (int j = sub + kPairLanes; j < n; j += kPairLanes) M = fmaxf(M, d.ml[partial_slot(d, row, part_of(j), head)].x);
#pragma unroll
  for (int o = kPairLanes / 2; o >= 1; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
  // The next kernel in the stream may become resident: every kernel of this library that is launched early
  // waits for this grid's completion before it writes anything to global memory (the planner counts first).
  pdl_trigger();

  float4 o4[kPer];
#pragma unroll
  for (int k = 0; k < kPer; ++k) o4[k] = make_float4(0.f, 0.f, 0.f, 0.f);
  float L = 0.f;
  const bool any = M > -INFINITY;

  for (int jb = 0; jb < n_warp; jb += kPairLanes) {
    // weights of up to kPairLanes partials at once, then their accumulators with independent loads
    float w_lane = 0.f;
    if (any && jb + sub < n) {
      const float2 ml = (jb == 0) ? ml0 : d.ml[partial_slot(d, row, part_of(jb + sub), head)];
      w_lane = fast_exp2(ml.x - M);
      L = fmaf(ml.y, w_lane, L);
    }
    const int cnt = any ? min(kPairLanes, n - jb) : 0;          // this pair's partials in the round
    const int cnt_warp = min(kPairLanes, n_warp - jb);
    for (int j0 = 0; j0 < cnt_warp; j0 += 4) {
      // four partials per round: all their loads are issued before the first is used
      float4 a[4][kPer];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool live = j0 + u < cnt;
        const float4* ap = reinterpret_cast<const float4*>(
            d.acc + partial_slot(d, row, part_of(jb + (live ? j0 + u : 0)), head) * D);
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
          const int v = sub + kPairLanes * k;
          a[u][k] = (live && v < kVecs) ? __ldcs(ap + v) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float w = __shfl_sync(0xffffffffu, w_lane, (j0 + u) % kPairLanes, kPairLanes);
        if (j0 + u >= cnt) w = 0.f;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
          o4[k].x = fmaf(a[u][k].x, w, o4[k].x); o4[k].y = fmaf(a[u][k].y, w, o4[k].y);
          o4[k].z = fmaf(a[u][k].z, w, o4[k].z); o4[k].w = fmaf(a[u][k].w, w, o4[k].w);
        }
      }
    }
  }
#pragma unroll
  for (int o = kPairLanes / 2; o >= 1; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
  if (!active || (parts.direct && !poison)) return;
  if (l_prev > 0.f) {
    const float w = fast_exp2(m_prev - M) * l_prev;
    L += w;
    const T* op = reinterpret_cast<const T*>(d.out) + (size_t)row * d.out_stride + (size_t)head * D;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int v = sub + kPairLanes * k;
      if (v < kVecs) {
        o4[k].x = fmaf(to_float<T>(op[v * 4 + 0]), w, o4[k].x);
        o4[k].y = fmaf(to_float<T>(op[v * 4 + 1]), w, o4[k].y);
        o4[k].z = fmaf(to_float<T>(op[v * 4 + 2]), w, o4[k].z);
        o4[k].w = fmaf(to_float<T>(op[v * 4 + 3]), w, o4[k].w);
      }
    }
  }
  const float inv = poison ? __int_as_float(0x7fc00000) : (L > 0.f) ? 1.f / L : 0.f;
  T* op = reinterpret_cast<T*>(d.out) + (size_t)row * d.out_stride + (size_t)head * D;
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int v = sub + kPairLanes * k;
    if (v < kVecs) {
      op[v * 4 + 0] = from_float<T>(o4[k].x * inv);
      op[v * 4 + 1] = from_float<T>(o4[k].y * inv);
      op[v * 4 + 2] = from_float<T>(o4[k].z * inv);
      op[v * 4 + 3] = from_float<T>(o4[k].w * inv);
    }
  }
  if ((d.stats_mode & PB_STATS_SAVE) && sub == 0) {
    d.qk_max[idx] = M;
    d.exp_sum[idx] = L;
  }
}

// Decode batches and small ones: (row, head) pairs packed over the rows, eight to a CTA; the lanes of a pair find
// its partials for themselves. A head count that is no multiple of eight leaves no lane idle (a step of 1024 rows x
// 4 heads over 2048 tokens: 42.4 us with CTAs that end with their row, 41.6 so). Registers decide how many pairs are
// in flight: 72 are seven CTAs an SM (256 rows x 32 heads: 67.0 us a step with 76 registers, six CTAs, 64.5 so; the
// headline step of 64 rows, whose merge fits the chip once, 72.1 and 72.4). What only the walk below needs stays out.
template <typename T, int D>
__global__ void __launch_bounds__(kMergeWarps * 32) merge_kernel(const AttnDev d) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long idx = ((long long)blockIdx.x * kMergeWarps + warp) * kPairsPerWarp + lane / kPairLanes;
  const int H = d.num_heads;
  const bool active = idx < (long long)d.num_rows * H;
  const int row = active ? (int)(idx / H) : 0, head = active ? (int)(idx - (long long)row * H) : 0;
  // The planner's output (row_info, dense items, header) is older than the attention kernels of
  // this call, so it is read while they still run; only then wait for their partials.
  const RowInfo info = d.row_info[row];
  const PartCounts parts = count_parts(d, info, d.hdr[kHdrDnTiles], dense_ctas_of(d), head);
  pdl_wait();  // every partial of the prefix and suffix stages is complete and visible
  if (blockIdx.x == 0 && threadIdx.x == 0) d.hdr[kHdrSqCounter] = 0;  // ready for the next layer call
  merge_one<T, D>(d, row, head, idx, active, info.nsc, parts, call_failed(d));
}

// Batches with many prefill rows: a CTA per row (and 128 heads) walks its heads eight at a time. How many partials
// a head has is worked out by one thread per head; a row that the dense kernel has finished leaves at once. (With a
// CTA per eight pairs, all lanes dividing, a batch of ten thousand prefill rows spent 100 us on finding out that there
// was nothing to do. For few rows the detour through shared memory costs 1.5 us.)
template <typename T, int D>
__global__ void __launch_bounds__(kMergeWarps * 32) merge_rows_kernel(const AttnDev d, const int heads_per_cta) {
  extern __shared__ PartCounts parts_of[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int H = d.num_heads;
  const int per_row = (H + heads_per_cta - 1) / heads_per_cta;  // CTAs of a row, next to each other
  const int row = blockIdx.x / per_row, h_lo = (blockIdx.x - row * per_row) * heads_per_cta, h_hi = min(H, h_lo + heads_per_cta);
  const RowInfo info = d.row_info[row];
  bool open = false;
  if ((int)threadIdx.x < h_hi - h_lo) {
    const PartCounts mine = count_parts(d, info, d.hdr[kHdrDnTiles], dense_ctas_of(d), h_lo + threadIdx.x);
    parts_of[threadIdx.x] = mine;
    open = !mine.direct;
  }
  const bool any_open = __syncthreads_or(open);
  pdl_wait();  // as above
  if (blockIdx.x == 0 && threadIdx.x == 0) d.hdr[kHdrSqCounter] = 0;
  const bool poison = call_failed(d);
  if (!any_open && !poison) return;
  for (int hb = h_lo; hb < h_hi; hb += kPairs) {
    const int head = hb + warp * kPairsPerWarp + lane / kPairLanes;
    const bool active = head < h_hi;
    merge_one<T, D>(d, row, head, (long long)row * H + head, active, info.nsc, parts_of[(active ? head : h_lo) - h_lo], poison);
  }
}

template <typename T, int D>
cudaError_t launch_merge_d(const AttnDev& d, cudaStream_t s) {
  if (d.seg_rows_max >= kManyRows) {  // (only prefill rows are ever finished before; decode rows do not count)
    const int hpc = d.num_heads < kMaxHeadsPerCta ? d.num_heads : kMaxHeadsPerCta;
    const unsigned grid = (unsigned)((long long)d.num_rows * ((d.num_heads + hpc - 1) / hpc));
    return launch_kernel(merge_rows_kernel<T, D>, grid, kMergeWarps * 32, (size_t)hpc * sizeof(PartCounts), s, true, d, hpc);
  }
  const unsigned grid = (unsigned)(((long long)d.num_rows * d.num_heads + kPairs - 1) / kPairs);
  return launch_kernel(merge_kernel<T, D>, grid, kMergeWarps * 32, 0, s, true, d);
}

template <typename T>
cudaError_t launch_merge_t(const AttnDev& d, int head_size, cudaStream_t s) {
  if (d.num_rows == 0) return cudaSuccess;
  switch (head_size) {
    case 64: return launch_merge_d<T, 64>(d, s);
    case 80: return launch_merge_d<T, 80>(d, s);
    case 96: return launch_merge_d<T, 96>(d, s);
    case 112: return launch_merge_d<T, 112>(d, s);
    case 128: return launch_merge_d<T, 128>(d, s);
    case 256: return launch_merge_d<T, 256>(d, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t launch_merge(const AttnDev& d, int dtype, int head_size, cudaStream_t s) {
  if (dtype == PB_F16) return launch_merge_t<__half>(d, head_size, s);
  if (dtype == PB_BF16) return launch_merge_t<__nv_bfloat16>(d, head_size, s);
  if (dtype == PB_F32) return launch_merge_t<float>(d, head_size, s);
  return cudaErrorInvalidValue;
}

}  // namespace pb
