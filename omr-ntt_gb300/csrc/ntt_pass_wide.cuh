// ntt_pass_wide.cuh -- persistent, double-buffered pass of 64-, 128- and
// 256-point lines on 128-byte-wide tiles.
//
// How fast a four-step pass can move its data depends on the width of its
// tile rows: on GB300 a copy in the pattern of a column pass (rows 16 KB
// apart) moves 2 x 64 MB in 43 us with 16-byte rows, 32 us with 32-byte rows,
// 27 us with 64-byte rows and 23 us -- the speed of a contiguous copy -- with
// 128-byte rows.  A 4096-point line fills 64 KB of shared memory with only 16
// bytes of lines per row; a 256-point line allows 128 bytes of lines per row
// in 32 KB.  So this pass takes 128 / word lines (32 for the 32-bit fields, 16
// for Goldilocks) of 256 points per tile, or twice as many (two boxes side by
// side) of 128 or 64 points:
//
//   * column passes: one 2-D TMA box [128 bytes of lines x T rows] per box,
//     landed with the 128-byte swizzle (16-byte chunk ch of row r at chunk
//     ch ^ (r mod 8)), so that with the lane mapping of wide_lane_l /
//     wide_lane_u every access below is conflict-free;
//     row passes: one 1-D bulk copy per line into a padded line-major layout,
//     or (wide_line_boxes) TMA boxes of 32 words of every line;
//   * warp w owns unit w (one or two 16-byte column groups); its lanes run
//     the line transforms as 16 x 16, 16 x 8 or 8 x 8 (first round, twiddle
//     omega_T^(l a), exchange through the warp's own column groups with an XOR
//     swizzle and __syncwarp, second round), then the four-step twiddle
//     (column passes: one operand per output from the domain's [line][k] table
//     where launch_pass gives one, else a base * step^q chain) and the inverse
//     scale;
//   * the results go back as 128-byte rows k = a + R1 b (natural order) and
//     one 2-D TMA store per box writes the tile;
//   * two tile buffers: the next tile lands while this one computes.
// Per tile that is one CTA barrier for column passes (every warp's results
// in the buffer before the store) and two for row passes (the lines are
// re-laid as rows in place).  Waits are bounded as in the other passes.
// Thread 0 waits on the previous kernel of the stream (programmatic
// dependent launch) before the first load.  Goldilocks column
// passes run the warp-specialised form at the end of this file; its row passes
// are faster in three CTAs an SM, which hide each other's barriers (the 2^24
// row pass 73.0 against 80.5 us).
//
// The line transform is the same split as the slab pass (ntt_pass_slab.cuh),
// i.e. the reference's four-step decomposition
// (src/encoders/winterfell_four_step.rs:31-81) within a line.
#pragma once
#include <cuda.h>

#include "ntt_pass_slab.cuh"

namespace omr {

// Line transform T = R1 x L: 16 x 16, 16 x 8 or 8 x 8.
template <int LOGT>
constexpr int wide_r1_log() {
  return LOGT == 6 ? 3 : 4;
}
// A tile is one (256 points) or two 128-byte-wide boxes of T rows; a warp's
// unit is one or two 16-byte column groups of it, so a tile is eight units.
template <int LOGT>
constexpr int wide_boxes() {
  return LOGT == 8 ? 1 : 2;
}
template <class F, int LOGT>
constexpr int wide_cols() {
  return wide_boxes<LOGT>() * 128 / F::WORD;  // lines per tile
}
constexpr int kWideThreads = 256;  // 8 warps: one per unit
// Row passes of 32-bit fields at 64 and 128 points land their lines by TMA in
// [32-word column box][line] rows of 128 bytes (128-byte swizzle): two to four
// loads a tile instead of 64 line copies from one thread.  The others copy
// line by line into padded runs.
template <class F, int LOGT>
constexpr bool wide_line_boxes() {
  return F::WORD == 4 && LOGT < 8;
}
template <class F, int LOGT>
constexpr int wide_line_bytes() {
  // line-major layout, padded so that the lines of a unit sit on other
  // banks: lines 2u + c of the 32-bit fields 8 banks apart (4-byte accesses,
  // a whole warp at a time), Goldilocks lines u 16 banks apart (8-byte
  // accesses, a half-warp of eight l and two u at a time)
  return (1 << LOGT) * F::WORD + (F::WORD == 8 ? 64 : 32);
}
template <class F, int LOGT>
constexpr int wide_buf_bytes() {  // a 1024-byte multiple (128-byte swizzle atoms)
  constexpr int a = (1 << LOGT) * 128 * wide_boxes<LOGT>(),
                b = wide_line_boxes<F, LOGT>() ? 0 : wide_cols<F, LOGT>() * wide_line_bytes<F, LOGT>();
  return ((a > b ? a : b) + 1023) / 1024 * 1024;
}
// In-line twiddles omega_T^(l a): [a - 1][l] for the 32-bit fields, which
// multiply before the exchange, [l - 1][a] for Goldilocks, which does after.
template <class F, int LOGT>
constexpr int wide_tab_entries() {
  constexpr int R1 = 1 << wide_r1_log<LOGT>(), L = (1 << LOGT) / R1;
  return F::ID == GOLDILOCKS ? (L - 1) * R1 : (R1 - 1) * L;
}
template <class F, int LOGT>
constexpr size_t wide_smem_bytes() {
  return 2 * (size_t)wide_buf_bytes<F, LOGT>() + wide_tab_entries<F, LOGT>() * sizeof(typename F::Tw) + 1024;
}
template <class F, int LOGT>
OMR_D void wide_fill_tab(typename F::Tw* tab1, const PassArgs<F>& a, int nt) {
  constexpr int R1 = 1 << wide_r1_log<LOGT>(), L = (1 << LOGT) / R1;
  constexpr int LW = F::ID == GOLDILOCKS ? wide_r1_log<LOGT>() : LOGT - wide_r1_log<LOGT>();  // log2 table width
  static_assert(wide_tab_entries<F, LOGT>() == (F::ID == GOLDILOCKS ? (L - 1) * R1 : (R1 - 1) * L), "whole rows");
  for (int i = threadIdx.x; i < wide_tab_entries<F, LOGT>(); i += nt)
    tab1[i] = round_table<F, LOGT - LW, LW>(a)[(1 << LW) + i];
}

// 128-byte-swizzled row layout: byte of (row r, 16-byte chunk ch, offset o)
template <int LOGT>
OMR_D int wide_sw(int r, int ch, int o) {
  return (ch >> 3) * (128 << LOGT) + r * 128 + (((ch ^ r) & 7) << 4) + o;
}

// Lane -> (l, u, g) of the line transforms.  256 points: l = lane bits 0-2 and
// 4, u = bit 3; shorter lines: l = bits 0-2, u = bit 3, g = bit 4 (the unit's
// column group).  The shared-memory pipe serves 8-byte accesses a half-warp at
// a time, so each half-warp (lanes 0-15, 16-31) holds the eight values of l
// mod 8 -- eight distinct chunk positions of the swizzle, as rows r = l + L m,
// L a + (l ^ a) and a + R1 b all have r mod 8 = l mod 8 (^ a) -- and both
// units u: 16 distinct 8-byte slots, one wavefront per half-warp.  (l = lane
// & 15, u = lane >> 4 put rows r and r + 8 of one unit into the same
// half-warp: a two-way conflict on every access.)
template <int LOGT>
OMR_D int wide_lane_l(int lane) {
  return LOGT == 8 ? ((lane & 7) | ((lane >> 1) & 8)) : (lane & 7);
}
OMR_D int wide_lane_u(int lane) { return (lane >> 3) & 1; }
// the lane's 16-byte column group of unit w
template <int LOGT>
OMR_D int wide_chunk(int w, int lane) {
  return LOGT == 8 ? w : 2 * w + (lane >> 4);
}

// The column unit u (8 bytes) of column group ch, row r.
template <class F, int LOGT, bool ROWS_LAYOUT>
OMR_D typename F::E* wide_word(unsigned char* s, int r, int ch, int u, int c) {
  using E = typename F::E;
  const int line = ch * (16 / F::WORD) + u * slab_vpu<F>() + c;
  if constexpr (ROWS_LAYOUT)
    return reinterpret_cast<E*>(s + wide_sw<LOGT>(r, ch, u * 8 + c * F::WORD));
  else if constexpr (wide_line_boxes<F, LOGT>())
    return reinterpret_cast<E*>(s + (r >> 5) * (wide_cols<F, LOGT>() * 128) + line * 128 +
                                (((r & 31) * 4) ^ ((line & 7) << 4)));
  else
    return reinterpret_cast<E*>(s + line * wide_line_bytes<F, LOGT>() + r * F::WORD);
}
template <class F, int LOGT, bool ROWS_LAYOUT>
OMR_D void wide_load_unit(unsigned char* s, int r, int ch, int u, typename F::E* dst) {
  constexpr int VPU = slab_vpu<F>();
  if constexpr (ROWS_LAYOUT && F::WORD == 4) {
    const uint2 x = *reinterpret_cast<const uint2*>(wide_word<F, LOGT, true>(s, r, ch, u, 0));
    dst[0] = x.x;
    dst[1] = x.y;
  } else {
#pragma unroll
    for (int c = 0; c < VPU; c++) dst[c] = *wide_word<F, LOGT, ROWS_LAYOUT>(s, r, ch, u, c);
  }
}
template <class F, int LOGT, bool ROWS_LAYOUT>
OMR_D void wide_store_unit(unsigned char* s, int r, int ch, int u, const typename F::E* src) {
  constexpr int VPU = slab_vpu<F>();
  if constexpr (ROWS_LAYOUT && F::WORD == 4) {
    *reinterpret_cast<uint2*>(wide_word<F, LOGT, true>(s, r, ch, u, 0)) = make_uint2(src[0], src[1]);
  } else {
#pragma unroll
    for (int c = 0; c < VPU; c++) *wide_word<F, LOGT, ROWS_LAYOUT>(s, r, ch, u, c) = src[c];
  }
}

OMR_D void tma_load_4d(void* dst, const CUtensorMap* map, int x, int y, int z, int w, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar))
      : "memory");
}

template <class F, int LOGT, int MODE>
OMR_D void wide_issue_load(const CUtensorMap* map, const PassArgs<F>& a, uint64_t tile,
                           unsigned char* buf, uint64_t* bar) {
  using E = typename F::E;
  constexpr int T = 1 << LOGT, C = wide_cols<F, LOGT>(), BX = wide_boxes<LOGT>();
  uint32_t g, lm;
  uint64_t lb;
  tile_coords<F, C>(a, tile, g, lm, lb);
  mbar_arrive_expect_tx(bar, (uint32_t)(T * C * F::WORD));
  if constexpr (MODE == MODE_COL) {
#pragma unroll
    for (int b = 0; b < BX; b++)
      tma_load_2d(buf + b * T * 128, map, (int)(g * C) + b * (C / BX), (int)((lb * a.L_m + lm) * (uint64_t)T), bar);
  } else if constexpr (wide_line_boxes<F, LOGT>()) {
#pragma unroll
    for (int j = 0; j < T / 32; j++)
      tma_load_4d(buf + j * C * 128, map, 32 * j, (int)(g * C), (int)lm, (int)lb, bar);
  } else {
    const E* src = a.in + (lb * a.is_b + lm * a.is_m + (uint64_t)(g * C) * a.is_lo);
#pragma unroll 1
    for (int c = 0; c < C; c++)
      bulk_load(buf + c * wide_line_bytes<F, LOGT>(), src + (uint64_t)c * a.is_lo, T * F::WORD, bar);
  }
}

template <class F, int LOGT, int MODE>
OMR_D void wide_issue_store(const CUtensorMap* map, const PassArgs<F>& a, uint64_t tile,
                            const unsigned char* buf) {
  constexpr int T = 1 << LOGT, C = wide_cols<F, LOGT>(), BX = wide_boxes<LOGT>();
  uint32_t g, lm;
  uint64_t lb;
  tile_coords<F, C>(a, tile, g, lm, lb);
#pragma unroll
  for (int b = 0; b < BX; b++) {
    if constexpr (MODE == MODE_COL)
      tma_store_2d(map, (int)(g * C) + b * (C / BX), (int)((lb * a.L_m + lm) * (uint64_t)T), buf + b * T * 128);
    else
      tma_store_2d(map, (int)(g * C + lm * (uint32_t)a.os_m) + b * (C / BX), (int)(lb * (uint64_t)T),
                   buf + b * T * 128);
  }
  bulk_commit();
}

// Unit w's results (wide_lines) to the swizzled rows.
template <class F, int LOGT>
OMR_D void wide_store_rows(unsigned char* s, int w, const typename F::E (&v)[slab_vpu<F>()][1 << wide_r1_log<LOGT>()]) {
  using E = typename F::E;
  constexpr int VPU = slab_vpu<F>(), R1 = 1 << wide_r1_log<LOGT>(), L = (1 << LOGT) / R1;
  const int lane = threadIdx.x & 31;
  const int am = wide_lane_l<LOGT>(lane), u = wide_lane_u(lane), ch = wide_chunk<LOGT>(w, lane);
#pragma unroll
  for (int i = 0; i < R1 / L; i++)
#pragma unroll
    for (int b = 0; b < L; b++) {
      E x[VPU];
#pragma unroll
      for (int c = 0; c < VPU; c++) x[c] = v[c][i * L + b];
      wide_store_unit<F, LOGT, true>(s, am + L * i + R1 * b, ch, u, x);
    }
}

// One warp: the line transforms of unit w.  The results are left in
// registers, v[c][i L + b] = line entry (am + L i) + R1 b (am =
// wide_lane_l(lane)); column passes also write them to the swizzled rows in
// place, row passes re-lay them as rows after a CTA barrier (their lines span
// every unit).
template <class F, int LOGT, int MODE, bool INV, bool TW>
OMR_D void wide_lines(const PassArgs<F>& a, unsigned char* s, const typename F::Tw* tab1, int w,
                      uint32_t llo0, uint32_t lm, typename F::E (&v)[slab_vpu<F>()][1 << wide_r1_log<LOGT>()]) {
  using E = typename F::E;
  constexpr int VPU = slab_vpu<F>(), LR1 = wide_r1_log<LOGT>(), R1 = 1 << LR1, LL = LOGT - LR1, L = 1 << LL;
  constexpr int PER = R1 / L;  // second-round DFTs per line and lane
  constexpr bool ROWS = MODE == MODE_COL;
  const int lane = threadIdx.x & 31;
  const int l = wide_lane_l<LOGT>(lane), u = wide_lane_u(lane), ch = wide_chunk<LOGT>(w, lane);
#pragma unroll
  for (int m = 0; m < R1; m++) {
    E x[VPU];
    wide_load_unit<F, LOGT, ROWS>(s, l + L * m, ch, u, x);
#pragma unroll
    for (int c = 0; c < VPU; c++) v[c][m] = x[c];
  }
  __syncwarp();
#pragma unroll
  for (int c = 0; c < VPU; c++) dft_reg_mul<F, LR1, INV>(v[c]);
  // twiddle omega_T^(l a): Goldilocks multiplies after the exchange, where
  // the products enter the second DFT unreduced
  if constexpr (F::ID != GOLDILOCKS) {
#pragma unroll
    for (int aa = 1; aa < R1; aa++) {
      const typename F::Tw t = tab1[(aa - 1) * L + l];
#pragma unroll
      for (int c = 0; c < VPU; c++) v[c][aa] = F::mul_tw(v[c][aa], t);
    }
  }
#pragma unroll
  for (int aa = 0; aa < R1; aa++) {
    E x[VPU];
#pragma unroll
    for (int c = 0; c < VPU; c++) x[c] = v[c][aa];
    wide_store_unit<F, LOGT, ROWS>(s, L * aa + (l ^ (aa & (L - 1))), ch, u, x);
  }
  __syncwarp();
  const int am = l;
#pragma unroll
  for (int i = 0; i < PER; i++)
#pragma unroll
    for (int ll = 0; ll < L; ll++) {
      E x[VPU];
      wide_load_unit<F, LOGT, ROWS>(s, L * (am + L * i) + (ll ^ am), ch, u, x);
#pragma unroll
      for (int c = 0; c < VPU; c++) v[c][i * L + ll] = x[c];
    }
  __syncwarp();
#pragma unroll
  for (int c = 0; c < VPU; c++)
#pragma unroll
    for (int i = 0; i < PER; i++) {
      const int aa = am + L * i;  // outputs b = 0 .. L - 1 are line entries aa + R1 b
      E y[L];
#pragma unroll
      for (int b = 0; b < L; b++) y[b] = v[c][i * L + b];
      if constexpr (F::ID == GOLDILOCKS)
        dft_reg_tw<F, LL, INV>(y, [&](int ll) { return tab1[(ll - 1) * R1 + aa]; });
      else  // column passes and inverse row passes multiply every result
        dft_reg<F, LL, INV, TW || INV>(y);
      const uint32_t line = llo0 + (uint32_t)(ch * (16 / F::WORD) + u * VPU + c) + lm * a.tw_line_mul_m;
      if (TW && a.tw_tab != nullptr) {
        // twiddle table [line][k]: one operand per output (tw_line_mul_m == 0)
        const typename F::Tw* row = a.tw_tab + ((size_t)line << LOGT) + aa;
#pragma unroll
        for (int b = 0; b < L; b++) y[b] = F::mul_tw(y[b], row[R1 * b]);
      } else if constexpr (TW) {
        const uint32_t ls = line * a.tw_scale;
        const uint32_t e0 = (ls * (uint32_t)aa) & a.tw_mask;
        const uint32_t es = (ls * (uint32_t)R1) & a.tw_mask;
        E t = F::mul_tw(__ldg(&a.tw_lo[e0 & ((1u << kTwLoBits) - 1)]), a.tw_hi[e0 >> kTwLoBits]);
        const E step = F::mul_tw(__ldg(&a.tw_lo[es & ((1u << kTwLoBits) - 1)]), a.tw_hi[es >> kTwLoBits]);
#pragma unroll
        for (int b = 0; b < L; b++) {
          y[b] = mul_m<F>(y[b], t);
          if (b + 1 < L) t = F::mont_mul(t, step);
        }
      }
      if constexpr (INV && !TW) {  // the last pass of an inverse transform
#pragma unroll
        for (int b = 0; b < L; b++) y[b] = F::mul_tw(y[b], a.scale);
      }
#pragma unroll
      for (int b = 0; b < L; b++) {
        if constexpr (MODE != MODE_COL) y[b] = F::canon(y[b]);  // the transform's results
        v[c][i * L + b] = y[b];
      }
    }
  if constexpr (ROWS) wide_store_rows<F, LOGT>(s, w, v);
}

template <class F, int LOGT, int MODE, bool INV, bool TW>
__global__ void __launch_bounds__(kWideThreads, 3)  // shared memory holds three CTAs an SM
    ntt_wide_pass(const __grid_constant__ CUtensorMap in_map,
                  const __grid_constant__ CUtensorMap out_map, const PassArgs<F> a, int* err) {
  using E = typename F::E;
  using Tw = typename F::Tw;
  constexpr int C = wide_cols<F, LOGT>(), VPU = slab_vpu<F>();
  constexpr int BB = wide_buf_bytes<F, LOGT>();
  extern __shared__ __align__(1024) unsigned char wide_smem_raw[];
  __shared__ __align__(8) uint64_t bars[2];
  __shared__ int abort_flag;
  unsigned char* base = wide_smem_raw + ((1024u - (smem_u32(wide_smem_raw) & 1023u)) & 1023u);
  Tw* tab1 = reinterpret_cast<Tw*>(base + 2 * BB);
  const int warp = threadIdx.x >> 5;

  const uint64_t ntiles = a.L_b * (uint64_t)a.L_m * (a.L_lo / C);
  uint64_t tile = blockIdx.x;
  if (threadIdx.x == 0) {
    prefetch_tmap(&in_map);
    prefetch_tmap(&out_map);
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    fence_mbar_init();
    fence_proxy_async();
    abort_flag = 0;
  }
  __syncthreads();
  uint32_t outstanding = 0;  // bit b: a load into buffer b has not been waited for
  if (threadIdx.x == 0) {
    // the previous pass's output is this one's input (and its input may be
    // this one's output): every global access of the pass follows this wait
    grid_dep_wait();
    if (tile < ntiles) {
      wide_issue_load<F, LOGT, MODE>(&in_map, a, tile, base, &bars[0]);
      outstanding |= 1u;
    }
    if (tile + gridDim.x < ntiles) {
      wide_issue_load<F, LOGT, MODE>(&in_map, a, tile + gridDim.x, base + BB, &bars[1]);
      outstanding |= 2u;
    }
  }
  grid_dep_launch();
  wide_fill_tab<F, LOGT>(tab1, a, kWideThreads);
  __syncthreads();

  uint32_t phase = 0;
  for (int it = 0; tile < ntiles; tile += gridDim.x, it++) {
    const int b = it & 1;
    unsigned char* s = base + b * BB;
    if (mbar_wait_bounded(&bars[b], (phase >> b) & 1)) {
      phase ^= 1u << b;
      outstanding &= ~(1u << b);
    } else {
      atomicExch(err, OMR_NTT_ERR_TIMEOUT);
      abort_flag = 1;
    }
    uint32_t g, lm;
    uint64_t lb;
    tile_coords<F, C>(a, tile, g, lm, lb);
    E v[VPU][1 << wide_r1_log<LOGT>()];
    wide_lines<F, LOGT, MODE, INV, TW>(a, s, tab1, warp, g * C, lm, v);
    if constexpr (MODE != MODE_COL) {
      // every warp has read its lines: re-lay the results as swizzled rows
      __syncthreads();
      wide_store_rows<F, LOGT>(s, warp, v);
    }
    fence_proxy_async();  // this thread's writes become visible to the TMA store
    __syncthreads();
    if (abort_flag) break;
    if (threadIdx.x == 0) {
      wide_issue_store<F, LOGT, MODE>(&out_map, a, tile, s);
      if (tile + 2ull * gridDim.x < ntiles) {
        bulk_wait_read_all();  // the store has read the buffer
        fence_proxy_async();
        wide_issue_load<F, LOGT, MODE>(&in_map, a, tile + 2ull * gridDim.x, s, &bars[b]);
        outstanding |= 1u << b;
      }
    }
  }
  if (threadIdx.x == 0) {
    bulk_wait_all();
    for (int bb = 0; bb < 2; bb++)
      if ((outstanding >> bb) & 1) mbar_wait_bounded(&bars[bb], (phase >> bb) & 1);
  }
}

// ---------------------------------------------------------------------------
// The column pass as one warp-specialised CTA per SM.  kWideSlots tile buffers
// cycle through load -> compute -> store: a loader warp issues the TMA loads,
// 24 consumer warps claim units (tile j, column group w) in order from a
// shared counter, so the eight column groups of a tile run on eight warps at
// once and every warp stays busy until the CTA's last unit, and a storer warp
// issues each tile's TMA store and hands the buffer back.  No CTA barrier:
// per buffer slot, `full` completes when the tile has landed, `done` when its
// eight units are written back, `empty` when its store has read it.
//
// Units are claimed in order but finish in any order, so a consumer can be
// more than one use of its slot ahead of the loads (a slow warp holding a
// unit of tile j - kWideSlots keeps that slot from being refilled while
// others run on).  A parity wait alone would then see an old phase as done:
// the producer publishes which tile each slot holds (`slot_tile`) before it
// issues the load, and a consumer waits for its tile to be the slot's before
// it waits on `full`.  `done` is safe without that check, because a unit
// reaches it only after its tile's load, i.e. after every unit of the slot's
// previous tile has passed it.
// 24 consumer warps (72 registers at 832 threads).  For the 32-bit fields
// the form measured slower than the three-CTA pass with 24 consumers at 72
// registers and with 22 at 80, so only Goldilocks launches it.
template <class F>
constexpr int wide_consumers() {
  return 24;
}
template <class F>
constexpr int wide_ws_threads() {
  return 32 * (wide_consumers<F>() + 2);  // + loader and storer warps
}
constexpr int kWideSlots = 6;

template <class F, int LOGT>
constexpr size_t wide_ws_smem_bytes() {
  return kWideSlots * (size_t)wide_buf_bytes<F, LOGT>() + wide_tab_entries<F, LOGT>() * sizeof(typename F::Tw) + 1024;
}

template <class F, int LOGT, bool INV>  // column passes
__global__ void __launch_bounds__(wide_ws_threads<F>(), 1)
    ntt_wide_ws_pass(const __grid_constant__ CUtensorMap in_map,
                     const __grid_constant__ CUtensorMap out_map, const PassArgs<F> a, int* err) {
  using E = typename F::E;
  using Tw = typename F::Tw;
  constexpr int C = wide_cols<F, LOGT>(), VPU = slab_vpu<F>(), S = kWideSlots;
  constexpr int BB = wide_buf_bytes<F, LOGT>();
  extern __shared__ __align__(1024) unsigned char wide_ws_smem_raw[];
  __shared__ __align__(8) uint64_t full[S], done[S], empty[S];
  __shared__ uint32_t unit_next;
  __shared__ volatile uint32_t slot_tile[S];  // j of the load last issued into each slot
  __shared__ volatile int abort_flag;
  unsigned char* base = wide_ws_smem_raw + ((1024u - (smem_u32(wide_ws_smem_raw) & 1023u)) & 1023u);
  Tw* tab1 = reinterpret_cast<Tw*>(base + S * BB);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // this CTA's tiles: blockIdx.x + j * gridDim.x, j < njobs
  const uint64_t ntiles = a.L_b * (uint64_t)a.L_m * (a.L_lo / C);
  const uint32_t njobs =
      ntiles > blockIdx.x ? (uint32_t)((ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x) : 0u;
  auto tile_of = [&](uint32_t j) { return blockIdx.x + (uint64_t)j * gridDim.x; };

  // The loader warp sets up the barriers and sends the first loads before
  // anything else, so the copies overlap the table setup.
  constexpr int NC = wide_consumers<F>();
  const bool loader = warp == NC;
  uint32_t j_load = 0;
  auto issue_next = [&]() -> bool {  // loader warp: tile j_load into its slot
    const int s = (int)(j_load % S);
    int go = 1;
    if (lane == 0) {
      if (j_load >= (uint32_t)S && !mbar_wait_bounded(&empty[s], ((j_load / S) - 1) & 1)) {
        atomicExch(err, OMR_NTT_ERR_TIMEOUT);
        abort_flag = 1;
      }
      go = !abort_flag;
      if (go) {
        slot_tile[s] = j_load;
        wide_issue_load<F, LOGT, MODE_COL>(&in_map, a, tile_of(j_load), base + s * BB, &full[s]);
      }
    }
    go = __shfl_sync(0xffffffffu, go, 0);
    if (!go) return false;
    j_load++;
    return true;
  };
  if (loader) {
    if (lane == 0) {
      for (int s = 0; s < S; s++) {
        mbar_init(&full[s], 1);
        mbar_init(&done[s], 8);
        mbar_init(&empty[s], 1);
        slot_tile[s] = 0xffffffffu;
      }
      fence_mbar_init();
      unit_next = 0;
      abort_flag = 0;
    }
    __syncwarp();
    // the previous pass's output is this one's input (and its input may be
    // this one's output): every global access of the pass follows the
    // loader's wait (the storer writes only tiles that were loaded after it)
    if (lane == 0) {
      prefetch_tmap(&in_map);
      prefetch_tmap(&out_map);
    }
    grid_dep_wait();
    while (j_load < njobs && j_load < (uint32_t)S && issue_next()) {
    }
  }
  grid_dep_launch();
  wide_fill_tab<F, LOGT>(tab1, a, wide_ws_threads<F>());
  __syncthreads();

  if (loader) {
    // slot s takes tile j once the store of tile j - S has read it
    while (j_load < njobs && issue_next()) {
    }
    // every issued load has landed before the CTA exits (all of them have
    // been consumed unless a wait gave up)
    if (lane == 0)
      for (uint32_t k = j_load > (uint32_t)S ? j_load - S : 0u; k < j_load; k++)
        mbar_wait_bounded(&full[k % S], (k / S) & 1);
    return;
  }
  if (warp == NC + 1) {
    // storer: one lane; tiles in order
    if (lane != 0) return;
    for (uint32_t j = 0; j < njobs; j++) {
      const int s = (int)(j % S);
      if (!mbar_wait_bounded(&done[s], (j / S) & 1)) {
        atomicExch(err, OMR_NTT_ERR_TIMEOUT);
        abort_flag = 1;
      }
      if (abort_flag) break;
      wide_issue_store<F, LOGT, MODE_COL>(&out_map, a, tile_of(j), base + s * BB);
      if (j + S < njobs) {
        bulk_wait_read_all();
        mbar_arrive(&empty[s]);
      }
    }
    bulk_wait_all();
    return;
  }

  // consumers
  for (;;) {
    uint32_t u = 0;
    if (lane == 0) u = atomicAdd(&unit_next, 1u);
    u = __shfl_sync(0xffffffffu, u, 0);
    const uint32_t j = u >> 3;
    const int w = (int)(u & 7u);
    if (j >= njobs || abort_flag) break;
    const int s = (int)(j % S);
    const uint32_t par = (j / S) & 1;
    unsigned char* buf = base + s * BB;
    bool mine = false;
    for (unsigned long long i = 0; i < kSpinLimit && !(mine = slot_tile[s] == j); i++) __nanosleep(20);
    if (!mine || !mbar_wait_bounded(&full[s], par)) {
      if (lane == 0) {
        atomicExch(err, OMR_NTT_ERR_TIMEOUT);
        abort_flag = 1;
      }
      break;
    }
    uint32_t g, lm;
    uint64_t lb;
    tile_coords<F, C>(a, tile_of(j), g, lm, lb);
    E v[VPU][1 << wide_r1_log<LOGT>()];
    wide_lines<F, LOGT, MODE_COL, INV, true>(a, buf, tab1, w, g * C, lm, v);
    fence_proxy_async();  // this thread's writes become visible to the TMA store
    __syncwarp();
    if (lane == 0) mbar_arrive(&done[s]);
  }
}

}  // namespace omr
