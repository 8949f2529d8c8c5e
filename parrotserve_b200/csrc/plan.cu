// Work-list builder: turns the device-resident lengths of one iteration into the item lists the
// attention kernels walk. One CTA; the lists depend on lengths only, so one plan serves every
// layer of the iteration.
//
// Reference counterpart: the per-iteration metadata of
// xFormersFill_SharedPromptsGenerate.init_iteration_state (parrot/engine/builtin/attn_func.py:461-599)
// stops at block tables and lengths; the split-KV decomposition there is implicit in the Triton
// grid (parrot/engine/builtin/kernels/shared_flash_decoding.py:240-243).
#include "common.cuh"

namespace pb {
namespace {

constexpr int kPlanThreads = 1024;
// Up to this many rows the suffix items are written by all threads, an item each: a thread per row wrote its
// chunks one after the other, each behind the load of the block ids of the one before. With the scans taken
// together: 128 rows of up to 16 chunks 17.0 -> 14.1 us, 64 rows over a prefix 11.8 -> 9.1 us. Beyond it the rows
// alone keep the threads busy (11 393 rows: 160 -> 152 us).
constexpr int kFlatRows = 4096;
constexpr double kDenseTileWeight = 3.5;  // SM time of a dense kv tile relative to streaming it once

// Exclusive scans of N ints per thread over the CTA, all with the same two barriers (N scans one after the
// other were a third of the kernel's time on a small batch): v[k] becomes the exclusive prefix, total[k] the sum.
template <int N>
__device__ __forceinline__ void block_exclusive_scans(int (&v)[N], int (&total)[N], int (*warp_sums)[33]) {
  static_assert(N <= (kPlanThreads >> 5), "one warp per scan");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const int mine = v[k];
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += n;
    }
    if (lane == 31) warp_sums[k][warp] = incl;
    v[k] = incl - mine;
  }
  __syncthreads();
  if (warp < N) {
    const int w = warp_sums[warp][lane];
    int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += n;
    }
    warp_sums[warp][lane] = wi - w;             // exclusive per warp
    if (lane == 31) warp_sums[warp][32] = wi;   // total
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; ++k) {
    total[k] = warp_sums[k][32];
    v[k] += warp_sums[k][warp];
  }
}

// Short chunks carry their block ids inside the item; longer ones point into their table.
// table_kind: 0 suffix_tables, 1 group_tables, 2 seg_tables, 3 outer_tables.
__device__ __forceinline__ SqItem make_sq_item(int row, const int32_t* table, int tbl_off, int table_kind, int nblk,
                                               int ntok, int part) {
  SqItem it;
  it.row = row;
  it.ntok = ntok;
  it.part = part;
  const bool embed = nblk <= kSqEmbedMax;
  it.meta = nblk | (table_kind << 18) | ((embed ? 1 : 0) << 17);
#pragma unroll
  for (int j = 0; j < kSqEmbedMax; ++j) it.bid[j] = (embed && j < nblk) ? table[tbl_off + j] : 0;
  if (!embed) it.bid[0] = tbl_off;
  return it;
}

struct GroupPlan {
  int r0, n_rows, plen, nblk, npc, dense, n_rt, nt;
};

__device__ __forceinline__ GroupPlan plan_of(const AttnDev& d, const int32_t* row_offsets, const int32_t* prefix_lens,
                                             int table_stride, int g, int B, bool dense_ok);
__device__ __forceinline__ GroupPlan group_plan(const AttnDev& d, int g, int B, bool dense_ok) {
  return plan_of(d, d.group_row_offsets, d.group_prefix_lens, d.group_table_stride, g, B, dense_ok);
}
__device__ __forceinline__ GroupPlan outer_plan(const AttnDev& d, int g, int B, bool dense_ok) {
  return plan_of(d, d.outer_row_offsets, d.outer_prefix_lens, d.outer_table_stride, g, B, dense_ok);
}
__device__ __forceinline__ GroupPlan plan_of(const AttnDev& d, const int32_t* row_offsets, const int32_t* prefix_lens,
                                             int table_stride, int g, int B, bool dense_ok) {
  GroupPlan p;
  int r0 = row_offsets[g], r1 = row_offsets[g + 1];
  if (r0 < 0 || r1 > d.num_rows) {  // offsets outside the batch
    r0 = max(r0, 0);
    r1 = min(r1, d.num_rows);
    atomicMax(&d.hdr[kHdrStatus], kStatusBadIndex);
  }
  p.r0 = r0;
  p.n_rows = max(r1 - r0, 0);
  p.plen = max(prefix_lens[g], 0);
  p.nblk = (p.plen + B - 1) / B;
  if (p.nblk > table_stride) {  // length claims more blocks than the table holds
    p.nblk = table_stride;
    p.plen = p.nblk * B;
    atomicMax(&d.hdr[kHdrStatus], kStatusBadIndex);
  }
  p.npc = (p.nblk + d.cp - 1) / d.cp;
  if (p.n_rows == 0) p.npc = 0;
  p.dense = (dense_ok && p.npc > 0 && p.n_rows >= d.dense_min_rows) ? 1 : 0;
  p.n_rt = (p.n_rows + d.dense_row_tile - 1) / d.dense_row_tile;
  p.nt = (p.nblk + kDenseTileBlocks - 1) / kDenseTileBlocks;
  return p;
}

// A causal segment: n new tokens (rows) of one request over kv private context tokens.
struct SegPlan {
  int r0, n, kv, n_rt;
};

__device__ __forceinline__ SegPlan seg_plan(const AttnDev& d, int s, int B) {
  SegPlan p;
  p.r0 = d.seg_row_offsets[s];
  int r1 = d.seg_row_offsets[s + 1];
  if (p.r0 < 0 || r1 > d.num_rows) {  // offsets outside the batch
    p.r0 = max(p.r0, 0);
    r1 = min(r1, d.num_rows);
    atomicMax(&d.hdr[kHdrStatus], kStatusBadIndex);
  }
  p.n = max(r1 - p.r0, 0);
  p.kv = max(d.seg_kv_lens[s], 0);
  if (p.kv < p.n || (p.kv + B - 1) / B > d.seg_table_stride) {  // inconsistent lengths
    atomicMax(&d.hdr[kHdrStatus], kStatusBadIndex);
    p.kv = max(p.n, min(p.kv, d.seg_table_stride * B));
    if ((p.kv + B - 1) / B > d.seg_table_stride) { p.n = 0; p.kv = 0; }
  }
  p.n_rt = (p.n + d.dense_row_tile - 1) / d.dense_row_tile;
  return p;
}
// tokens the last row of row tile rt sees = kv tokens the tile's dense item has to cover
__device__ __forceinline__ int seg_tile_visible(const AttnDev& d, const SegPlan& p, int rt) {
  return p.kv - p.n + min(p.n, (rt + 1) * d.dense_row_tile);
}

// Index i in [0, n) with offs[i] <= r < offs[i + 1] of a CSR offsets array, or -1.
__device__ __forceinline__ int csr_find(const int32_t* offs, int n, int r) {
  if (n <= 0 || r < offs[0] || r >= offs[n]) return -1;
  int lo = 0, hi = n - 1;  // last i with offs[i] <= r
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (offs[mid] <= r) lo = mid; else hi = mid - 1;
  }
  return r < offs[lo + 1] ? lo : -1;
}
// Dense item in [lo, hi) (ascending row0) whose rows contain r, or -1.
__device__ __forceinline__ int item_find(const DnItem* items, int lo, int hi, int r) {
  if (lo >= hi) return -1;
  int a = lo, b = hi - 1;  // last item with row0 <= r
  while (a < b) {
    const int mid = (a + b + 1) >> 1;
    if (items[mid].row0 <= r) a = mid; else b = mid - 1;
  }
  const DnItem it = items[a];
  return (r >= it.row0 && r < it.row0 + it.nrows) ? a : -1;
}

// A prefill request whose rows all lie inside one prefix group that runs on the dense kernel is
// planned TOGETHER with that group: its row tiles become two-piece items (the group's prefix, then
// the request's own context under the causal mask) that accumulate both in one pass and leave one
// partial instead of two. Returns the group, or -1 when the segment keeps items of its own.
__device__ __forceinline__ int seg_joined_group(const AttnDev& d, const SegPlan& sp, int B, bool dense_ok) {
  if (!dense_ok || sp.n <= 0 || d.num_groups <= 0) return -1;
  const int g = csr_find(d.group_row_offsets, d.num_groups, sp.r0);
  if (g < 0) return -1;
  const GroupPlan p = group_plan(d, g, B, dense_ok);
  if (!p.dense || p.npc == 0) return -1;
  return (sp.r0 >= p.r0 && sp.r0 + sp.n <= p.r0 + p.n_rows) ? g : -1;
}
// kv tiles of a segment's row tile rt (its own context only)
__device__ __forceinline__ int seg_tiles(const AttnDev& d, const SegPlan& sp, int rt, int B) {
  return ((seg_tile_visible(d, sp, rt) + B - 1) / B + kDenseTileBlocks - 1) / kDenseTileBlocks;
}
// Walks the rows of a dense group in ascending order: gap(r_lo, r_hi) for every run of rows outside
// joined segments, joined(s, sp) for every joined segment.
template <typename GapFn, typename SegFn>
__device__ __forceinline__ void walk_group_rows(const AttnDev& d, int g, const GroupPlan& p, int B, bool dense_ok,
                                                GapFn gap, SegFn joined) {
  int cursor = p.r0;
  const int r_end = p.r0 + p.n_rows;
  const int NS = d.num_segments;
  if (NS > 0) {
    // first segment whose rows end after the group's first row
    int lo = 0, hi = NS;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (d.seg_row_offsets[mid + 1] <= p.r0) lo = mid + 1; else hi = mid;
    }
    for (int s = lo; s < NS && d.seg_row_offsets[s] < r_end; ++s) {
      const SegPlan sp = seg_plan(d, s, B);
      if (sp.n <= 0 || sp.r0 < cursor || seg_joined_group(d, sp, B, dense_ok) != g) continue;
      if (sp.r0 > cursor) gap(cursor, sp.r0);
      joined(s, sp);
      cursor = sp.r0 + sp.n;
    }
  }
  if (cursor < r_end) gap(cursor, r_end);
}

__global__ void __launch_bounds__(kPlanThreads, 1) plan_kernel(const AttnDev d, const int B, const bool dense_ok) {
  constexpr int kScans = 8;
  __shared__ int warp_sums[kScans][33];
  // first suffix item of every row (kCarries: the row's last item carries its new token), for batches whose
  // suffix items are written by all threads in item order
  constexpr int kCarries = 1 << 30;
  __shared__ int row_first[kFlatRows + 1];
  __shared__ unsigned long long sq_blocks;  // blocks all single-query items stream, per head
  // The kernel before this one may still be at work, and it may own the very memory this call's workspace lies
  // in: a merge of another call on the same scratch, whose partials are where this call's lists go, or the
  // stores of an output whose memory has been handed out again. Until pdl_wait() only lengths and offsets are
  // read and nothing is written outside shared memory; faults found while counting are kept here.
  __shared__ int32_t count_hdr[kHdrStatus + 1];
  AttnDev c = d;
  c.hdr = count_hdr;
  const int tid = threadIdx.x;
  const int S = d.num_rows, G = d.num_groups, NS = d.num_segments;
  const int RT = d.dense_row_tile;  // rows per dense item: 128, or 256 when the dense kernel works on row-tile pairs

  if (tid == 0) { count_hdr[kHdrStatus] = kStatusOk; sq_blocks = 0; }
  __syncthreads();

  // ---- counts: groups (dense items / single-query prefix items) ----
  const int gper = (G + kPlanThreads - 1) / kPlanThreads;
  const int g_lo = min(tid * gper, G), g_hi = min(g_lo + gper, G);
  int my_dng = 0, my_dns = 0, my_sq = 0, my_tiles_g = 0, my_tiles_s = 0;
  long long my_blocks = 0;
  for (int g = g_lo; g < g_hi; ++g) {
    const GroupPlan p = group_plan(c, g, B, dense_ok);
    if (p.dense) {
      walk_group_rows(c, g, p, B, dense_ok,
                      [&](int r_lo, int r_hi) {
                        const int n_rt = (r_hi - r_lo + RT - 1) / RT;
                        my_dng += n_rt;
                        my_tiles_g += n_rt * p.nt;
                      },
                      [&](int, const SegPlan& sp) {
                        my_dng += sp.n_rt;
                        for (int rt = 0; rt < sp.n_rt; ++rt) my_tiles_g += kCausalFixedTiles + p.nt + seg_tiles(c, sp, rt, B);
                      });
    } else {
      my_sq += p.npc * p.n_rows;
      my_blocks += (long long)p.nblk * p.n_rows;
    }
  }
  // ---- counts: causal segments (dense items per row tile / single-query items per row) ----
  const int sper = (NS + kPlanThreads - 1) / kPlanThreads;
  const int s_lo = min(tid * sper, NS), s_hi = min(s_lo + sper, NS);
  for (int s = s_lo; s < s_hi; ++s) {
    const SegPlan p = seg_plan(c, s, B);
    if (seg_joined_group(c, p, B, dense_ok) >= 0) continue;  // counted with its group
    if (dense_ok) {
      my_dns += p.n_rt;
      for (int rt = 0; rt < p.n_rt; ++rt) my_tiles_s += kCausalFixedTiles + seg_tiles(c, p, rt, B);
    } else {
      for (int i = 0; i < p.n; ++i) {
        const int nb = (p.kv - p.n + i + 1 + B - 1) / B;
        my_sq += (nb + d.cs - 1) / d.cs;
        my_blocks += nb;
      }
    }
  }
  // ---- counts: outer prefix groups (dense items per row tile / single-query items per row) ----
  const int NO = d.num_outer_groups;
  const int oper = (NO + kPlanThreads - 1) / kPlanThreads;
  const int o_lo = min(tid * oper, NO), o_hi = min(o_lo + oper, NO);
  int my_dno = 0, my_tiles_o = 0;
  for (int o = o_lo; o < o_hi; ++o) {
    const GroupPlan p = outer_plan(c, o, B, dense_ok);
    if (p.dense) { my_dno += p.n_rt; my_tiles_o += p.n_rt * p.nt; }
    else { my_sq += p.npc * p.n_rows; my_blocks += (long long)p.nblk * p.n_rows; }
  }
  // ---- counts: rows (suffix items) ----
  const int rper = (S + kPlanThreads - 1) / kPlanThreads;
  const int r_lo = min(tid * rper, S), r_hi = min(r_lo + rper, S);
  int my_sqs = 0;
  for (int r = r_lo; r < r_hi; ++r) {
    int len = d.suffix_lens ? max(d.suffix_lens[r], 0) : 0;
    int nblk = (len + B - 1) / B;
    if (nblk > d.suffix_table_stride) nblk = d.suffix_table_stride;
    my_sqs += (nblk + d.cs - 1) / d.cs;
    my_blocks += nblk;
  }
  if (my_blocks) atomicAdd(&sq_blocks, (unsigned long long)my_blocks);
  // Dense items: all group items first (ascending rows), then all segment items (ascending rows),
  // so that a row finds its items by binary search and tile_base grows with the item index.
  int scan[kScans] = {my_dng, my_dns, my_sq, my_tiles_g, my_tiles_s, my_sqs, my_dno, my_tiles_o}, sum[kScans];
  block_exclusive_scans<kScans>(scan, sum, warp_sums);
  const int total_dng = sum[0], total_sq = sum[2], total_tiles_g = sum[3], total_sqs = sum[5];
  const int total_dn_inner = total_dng + sum[1], total_dn = total_dn_inner + sum[6];
  const int total_tiles = total_tiles_g + sum[4] + sum[7];
  int dng_base = scan[0], dns_base = scan[1] + total_dng, sq_base = scan[2], tile_g_base = scan[3];
  int tile_s_base = scan[4] + total_tiles_g, dno_base = scan[6] + total_dn_inner;
  int tile_o_base = scan[7] + total_tiles_g + sum[4];
  const int sqs_base = scan[5];

  const bool overflow = (total_dn > d.cap_dn) || (total_sq + total_sqs > d.cap_sq);
  // From here on the workspace is written: the kernel before this one has to be complete (see count_hdr), and the
  // attention kernels, which wait only for their direct predecessor, find it complete too.
  pdl_wait();
  if (tid == 0) {
    d.hdr[kHdrStatus] = max(count_hdr[kHdrStatus], overflow ? kStatusListOverflow : kStatusOk);
    d.hdr[kHdrSqCounter] = 0;
    d.hdr[kHdrPlannedSlots] = (d.slot_mapping && NS == 0 && !d.head_mapping) ? 1 : 0;
    d.hdr[kHdrNumSq] = overflow ? 0 : total_sq + total_sqs;
    d.hdr[kHdrNumDn] = overflow ? 0 : total_dn;
    d.hdr[kHdrDnTiles] = overflow ? 0 : total_tiles * d.num_heads;
    // Split of the SMs between the dense kernel and the single-query kernel that runs beside it:
    // proportional to their work in units of one 128-token kv tile of one head (64 KiB of KV for
    // the streaming kernel). A dense tile is weighted: giving the dense kernel too many SMs costs
    // little, because its CTAs retire early and the single-query kernel takes their SMs over, while
    // too few make it the long pole.
    // (In positions of the tile order, the fixed ones included, twice as many where items are row-tile pairs: what an
    // (item, head) costs beside its tiles keeps an SM busy too, and a lone row tile costs nearly what a pair does. With
    // the kv tiles of row tiles of 128 rows alone: 64 groups x 16 decode rows and a 512-token prefill 461 us against 417,
    // 4 groups x 250 and a 2000-token one 421 against 382.)
    const double td = kDenseTileWeight * (double)total_tiles * d.num_heads * (RT / 128);
    const double ts = (double)sq_blocks * d.num_heads / kDenseTileBlocks;
    const int sms = d.num_sms;
    int c = sms;
    if (td > 0 && ts > 0) {
      c = (int)(sms * td / (td + ts) + 0.5);
      c = (c >= sms * 4 / 5) ? sms : max(4, c);
    }
    if (d.dense_ctas > 0) c = min(d.dense_ctas, sms);  // the caller's choice
    d.hdr[kHdrDenseCtas] = c;
  }
  if (overflow) {  // no lists: no row has a partial (the merge reads the row infos and writes NaN)
    RowInfo none = {};
    none.group = none.dn = none.seg_dn = none.odn = -1;
    for (int r = tid; r < S; r += kPlanThreads) d.row_info[r] = none;
    return;
  }
  __syncthreads();  // the header's status is in place; faults found below are added to it

  // ---- groups: dense items (whole prefix per row tile) or single-query prefix items per row ----
  for (int g = g_lo; g < g_hi; ++g) {
    const GroupPlan p = group_plan(d, g, B, dense_ok);
    const int r0 = p.r0;
    if (p.npc == 0) continue;
    if (p.dense) {
      walk_group_rows(
          d, g, p, B, dense_ok,
          [&](int r_lo, int r_hi) {  // rows outside joined segments: the prefix alone
            for (int rr = r_lo; rr < r_hi; rr += RT) {
              DnItem it;
              it.row0 = rr;
              it.nrows = min(RT, r_hi - rr);
              it.tbl_off = g * d.group_table_stride;
              it.nblk = p.nblk;
              it.ntok = p.plen;
              it.nt = p.nt;
              it.tile_base = tile_g_base * d.num_heads;
              it.causal_base = 0;
              it.nt1 = it.nblk1 = it.ntok1 = it.tbl2_off = 0;
              it.flags = 0; it.fixed = it.pad[0] = it.pad[1] = 0;
              tile_g_base += it.nt;
              d.dn_items[dng_base++] = it;
            }
          },
          [&](int sidx, const SegPlan& sp) {  // a joined prefill request: prefix, then its own context
            for (int rt = 0; rt < sp.n_rt; ++rt) {
              const int vis = seg_tile_visible(d, sp, rt);
              DnItem it;
              it.row0 = sp.r0 + rt * RT;
              it.nrows = min(RT, sp.n - rt * RT);
              it.tbl_off = g * d.group_table_stride;
              it.nt1 = p.nt;
              it.nblk1 = p.nblk;
              it.ntok1 = p.plen;
              it.tbl2_off = sidx * d.seg_table_stride;
              it.flags = kDnDirect;  // withdrawn below if a row of the tile turns out to have a suffix
              it.fixed = kCausalFixedTiles; it.pad[0] = it.pad[1] = 0;
              it.nblk = (vis + B - 1) / B;
              it.ntok = vis;
              it.nt = p.nt + seg_tiles(d, sp, rt, B);
              it.tile_base = tile_g_base * d.num_heads;
              it.causal_base = sp.kv - sp.n + rt * RT + 1;  // own tokens row 0 of the tile sees
              tile_g_base += it.fixed + it.nt;
              d.dn_items[dng_base++] = it;
            }
          });
    } else {
      for (int i = 0; i < p.n_rows; ++i)
        for (int c = 0; c < p.npc; ++c) {
          const int nb = min(d.cp, p.nblk - c * d.cp);
          d.sq_items[sq_base++] = make_sq_item(r0 + i, d.group_tables, g * d.group_table_stride + c * d.cp, 1, nb,
                                               min(p.plen - c * d.cp * B, nb * B), c);
        }
    }
  }

  // ---- causal segments: one dense item per row tile, covering the kv tokens its last row
  //      sees; without a tensor-core path every row becomes single-query items over its own view ----
  for (int s = s_lo; s < s_hi; ++s) {
    const SegPlan p = seg_plan(d, s, B);
    if (seg_joined_group(d, p, B, dense_ok) >= 0) continue;  // emitted with its group
    if (dense_ok) {
      for (int rt = 0; rt < p.n_rt; ++rt) {
        const int vis = seg_tile_visible(d, p, rt);
        DnItem it;
        it.nt1 = it.nblk1 = it.ntok1 = it.tbl2_off = 0;
        it.flags = kDnDirect;  // withdrawn below if a row of the tile has a prefix or a suffix besides
        it.fixed = kCausalFixedTiles; it.pad[0] = it.pad[1] = 0;
        it.row0 = p.r0 + rt * RT;
        it.nrows = min(RT, p.n - rt * RT);
        it.tbl_off = s * d.seg_table_stride;
        it.nblk = (vis + B - 1) / B;
        it.ntok = vis;
        it.nt = (it.nblk + kDenseTileBlocks - 1) / kDenseTileBlocks;
        it.tile_base = tile_s_base * d.num_heads;
        it.causal_base = p.kv - p.n + rt * RT + 1;  // tokens row 0 of the tile sees
        tile_s_base += it.fixed + it.nt;
        d.dn_items[dns_base++] = it;
      }
    } else {
      for (int i = 0; i < p.n; ++i) {
        const int r = p.r0 + i, vis = p.kv - p.n + i + 1;
        const int nblk = (vis + B - 1) / B, nc = (nblk + d.cs - 1) / d.cs;
        for (int c = 0; c < nc; ++c) {
          const int nb = min(d.cs, nblk - c * d.cs);
          d.sq_items[sq_base++] = make_sq_item(r, d.seg_tables, s * d.seg_table_stride + c * d.cs, 2, nb,
                                               min(vis - c * d.cs * B, nb * B), d.pparts + c);
        }
      }
    }
  }
  // ---- outer prefix groups: like plain groups, in their own item and partial ranges ----
  for (int o = o_lo; o < o_hi; ++o) {
    const GroupPlan p = outer_plan(d, o, B, dense_ok);
    if (p.npc == 0) continue;
    if (p.dense) {
      for (int rr = p.r0; rr < p.r0 + p.n_rows; rr += RT) {
        DnItem it;
        it.row0 = rr;
        it.nrows = min(RT, p.r0 + p.n_rows - rr);
        it.tbl_off = o * d.outer_table_stride;
        it.nblk = p.nblk;
        it.ntok = p.plen;
        it.nt = p.nt;
        it.tile_base = tile_o_base * d.num_heads;
        it.causal_base = 0;
        it.nt1 = it.nblk1 = it.ntok1 = it.tbl2_off = 0;
        it.flags = kDnOuter; it.fixed = it.pad[0] = it.pad[1] = 0;
        tile_o_base += it.nt;
        d.dn_items[dno_base++] = it;
      }
    } else {
      for (int i = 0; i < p.n_rows; ++i)
        for (int c = 0; c < p.npc; ++c) {
          const int nb = min(d.cp, p.nblk - c * d.cp);
          d.sq_items[sq_base++] = make_sq_item(p.r0 + i, d.outer_tables, o * d.outer_table_stride + c * d.cp, 3, nb,
                                               min(p.plen - c * d.cp * B, nb * B), d.pparts + d.cparts + d.sparts + c);
        }
    }
  }
  __syncthreads();  // the dense items are in place; rows look theirs up below

  // ---- rows: row_info (group, segment and dense items of the row) and the suffix items ----
  int w = total_sq + sqs_base;
  for (int r = r_lo; r < r_hi; ++r) {
    int len = d.suffix_lens ? max(d.suffix_lens[r], 0) : 0;
    int nblk = (len + B - 1) / B;
    if (nblk > d.suffix_table_stride) {
      nblk = d.suffix_table_stride;
      len = nblk * B;
      atomicMax(&d.hdr[kHdrStatus], kStatusBadIndex);
    }
    const int nsc = (nblk + d.cs - 1) / d.cs;
    RowInfo info;
    info.group = -1; info.np_sq = 0; info.nsc = nsc; info.dn = -1; info.seg_dn = -1; info.nc_sq = 0;
    info.odn = -1; info.onp_sq = 0;
    if (NO > 0) {
      const int o = csr_find(d.outer_row_offsets, NO, r);
      if (o >= 0) {
        const GroupPlan p = outer_plan(d, o, B, dense_ok);
        if (p.dense) info.odn = item_find(d.dn_items, total_dn_inner, total_dn, r);
        else info.onp_sq = p.npc;
      }
    }
    const int g = csr_find(d.group_row_offsets, G, r);
    if (g >= 0) {
      const GroupPlan p = group_plan(d, g, B, dense_ok);
      info.group = g;
      info.np_sq = p.dense ? 0 : p.npc;
      info.dn = (p.dense && p.npc > 0) ? item_find(d.dn_items, 0, total_dng, r) : -1;
    }
    if (NS > 0) {
      if (dense_ok) {
        info.seg_dn = item_find(d.dn_items, total_dng, total_dn_inner, r);
      } else {
        const int s = csr_find(d.seg_row_offsets, NS, r);
        if (s >= 0) {
          const SegPlan p = seg_plan(d, s, B);
          if (r - p.r0 < p.n) info.nc_sq = (((p.kv - p.n + (r - p.r0) + 1 + B - 1) / B) + d.cs - 1) / d.cs;
        }
      }
    }
    d.row_info[r] = info;
    // this row has other partials and needs the merge: so does its tile
    const bool other = nsc > 0 || info.odn >= 0 || info.onp_sq > 0;
    if (info.dn >= 0 && (other || info.seg_dn >= 0) && (d.dn_items[info.dn].flags & kDnDirect))
      atomicAnd(&d.dn_items[info.dn].flags, ~kDnDirect);
    if (info.seg_dn >= 0 && (other || info.dn >= 0 || info.np_sq > 0) && (d.dn_items[info.seg_dn].flags & kDnDirect))
      atomicAnd(&d.dn_items[info.seg_dn].flags, ~kDnDirect);
    // The row's new token (a pure decode batch whose fill the suffix kernel performs itself): it must be
    // the last token of the row's suffix, so that the item of the last chunk can carry it.
    bool carries_new = false;
    if (d.slot_mapping && NS == 0 && !d.head_mapping) {
      const long long slot = d.slot_is_i64 ? reinterpret_cast<const long long*>(d.slot_mapping)[r]
                                           : (long long)reinterpret_cast<const int*>(d.slot_mapping)[r];
      if (slot >= 0) {
        const long long want = (len > 0 && nsc > 0)
            ? (long long)d.suffix_tables[(size_t)r * d.suffix_table_stride + (len - 1) / B] * B + (len - 1) % B : -1;
        if (slot == want) carries_new = true;
        else atomicMax(&d.hdr[kHdrStatus], kStatusBadIndex);
      }
    }
    if (S <= kFlatRows) {
      row_first[r] = (w - total_sq) | (carries_new ? kCarries : 0);
      w += nsc;
      continue;
    }
    for (int c = 0; c < nsc; ++c) {
      const int nb = min(d.cs, nblk - c * d.cs);
      SqItem it = make_sq_item(r, d.suffix_tables, r * d.suffix_table_stride + c * d.cs, 0, nb,
                               min(len - c * d.cs * B, nb * B), d.pparts + d.cparts + c);
      if (carries_new && c == nsc - 1) it.meta |= 1 << 20;
      d.sq_items[w++] = it;
    }
  }
  if (S <= kFlatRows) {
    if (tid == 0) row_first[S] = total_sqs;
    __syncthreads();
    auto first_of = [&](int r) { return row_first[r] & (kCarries - 1); };
    for (int idx = tid; idx < total_sqs; idx += kPlanThreads) {
      int lo = 0, hi = S - 1;  // last row whose items start at idx or before (rows without items start where the next one does)
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (first_of(mid) <= idx) lo = mid; else hi = mid - 1;
      }
      const int r = lo, c = idx - first_of(r);
      int len = max(d.suffix_lens[r], 0), nblk = (len + B - 1) / B;
      if (nblk > d.suffix_table_stride) { nblk = d.suffix_table_stride; len = nblk * B; }
      const int nb = min(d.cs, nblk - c * d.cs);
      SqItem it = make_sq_item(r, d.suffix_tables, r * d.suffix_table_stride + c * d.cs, 0, nb,
                               min(len - c * d.cs * B, nb * B), d.pparts + d.cparts + c);
      if ((row_first[r] & kCarries) && idx + 1 == first_of(r + 1)) it.meta |= 1 << 20;
      d.sq_items[total_sq + idx] = it;
    }
  }
}

}  // namespace

cudaError_t launch_plan(const AttnDev& d, int block_size, bool dense_supported, cudaStream_t s) {
  return launch_kernel(plan_kernel, 1, kPlanThreads, 0, s, true, d, block_size, dense_supported);
}

}  // namespace pb
