// ntt_pass_duo.cuh -- pass of 512- and 1024-point lines in two register rounds
// on 64-byte-wide tiles (32-bit fields).
//
// A 1024-point line is 32 x 32 and a 512-point line 32 x 16, so a thread that
// holds 32 words of one line runs the whole line transform with one exchange:
// radix-32 round, twiddle omega_T^(l a), exchange, second round, four-step
// twiddle.  Against the three rounds of the other passes at these lengths that
// is one exchange, one twiddle product and one barrier less per word.
//
// Four adjacent lines (one 16-byte column group) are the work of one thread
// group: 128 threads at 1024 points, 64 at 512.  In a warp eight l (or a)
// times four lines make one shared-memory wavefront of every access below:
//   * rows layout (column passes; the staging of every pass's results): tile
//     rows of 64 bytes with the 64-byte TMA swizzle, in which eight
//     consecutive rows of one 16-byte chunk take the eight 16-byte slots of a
//     128-byte bank line;
//   * line-major layout (row passes until the staging): lines padded by 32
//     bytes, so the four lines of a group lie eight banks apart;
//   * exchange: V[l][a] at row L a + (l ^ (a mod L)), L = T / 32.
//
// Four groups make a tile, a team of threads: the width of its rows (64 bytes)
// sets how fast a column pass can move data (a copy of 2 x 64 MB in that
// pattern takes 43 us with the slab pass's 16-byte rows, 27 us with 64-byte
// rows on GB300).  A 1024-point tile takes 64 KB and 512 threads: two teams in
// one CTA an SM share three buffers, so the tile after the two in work lands
// meanwhile (BabyBear 64 x 2^20: 287-289 us; with one buffer in each of two
// CTAs 356, with 32-byte rows 326, on the slab and TMA passes 433-450).  A
// 512-point tile takes 32 KB and 256 threads, four single-buffered CTAs an SM
// (64 x 2^18: 86 us; TMA pass 104).  Waits are bounded as in the other passes.
//
// The line transform is the reference's four-step decomposition
// (src/encoders/winterfell_four_step.rs:31-81) within a line.
#pragma once
#include <cuda.h>

#include "ntt_pass_wide.cuh"
#include "team_ring.cuh"

namespace omr {

template <class F, int LOGT>
constexpr bool has_duo_pass() {
  return F::WORD == 4 && (LOGT == 9 || LOGT == 10);
}
template <int LOGT>
constexpr int duo_group_threads() {
  return (1 << LOGT) / 8;  // 4 lines, 32 words a thread
}
constexpr int kDuoGroups = 4, kDuoCols = 16, kDuoRowBytes = 64;  // of a tile
template <int LOGT>
constexpr int duo_team_threads() {
  return kDuoGroups * duo_group_threads<LOGT>();
}
template <int LOGT>
constexpr int duo_teams() {
  return LOGT == 10 ? 2 : 1;
}
template <int LOGT>
constexpr int duo_line_bytes() {
  return (4 << LOGT) + 32;
}
template <int LOGT>
constexpr int duo_buf_bytes() {  // the larger of the two layouts
  return (kDuoCols * duo_line_bytes<LOGT>() + 1023) / 1024 * 1024;
}
template <int LOGT>
constexpr int duo_bufs() {
  return duo_teams<LOGT>() == 1 ? 1 : duo_teams<LOGT>() + 1;
}
template <class F, int LOGT>
constexpr size_t duo_smem_bytes() {
  return duo_bufs<LOGT>() * (size_t)duo_buf_bytes<LOGT>() +
         (size_t)31 * ((1 << LOGT) / 32) * sizeof(typename F::Tw) + 1024;
}
// Named barriers: groups synchronise by 128 threads (one group of 1024-point
// lines, two of 512-point lines; barriers 1 .. 8), a team by one of the next.
constexpr int kDuoSyncThreads = 128;
OMR_D int duo_team_barrier(int team) { return 9 + team; }

// Byte of row r in rows layout, chunk ch, in the buffer.  The three terms'
// bits are disjoint and the swizzle repeats every 8 rows, so the byte of row
// r ^ k is the byte of row r, XOR duo_row(k, 0).
OMR_D constexpr uint32_t duo_row(uint32_t r, uint32_t ch) { return r * kDuoRowBytes + ((ch ^ ((r >> 1) & 3u)) << 4); }

// Byte of entry l ^ k of line c of chunk ch (k a compile-time constant).
template <int LOGT, bool ROWS>
OMR_D uint32_t duo_at(uint32_t l, uint32_t k, uint32_t ch, uint32_t c) {
  if constexpr (ROWS)
    return (duo_row(l, ch) + 4 * c) ^ duo_row(k, 0);
  else
    return (4 * ch + c) * duo_line_bytes<LOGT>() + ((4 * l) ^ (4 * k));
}

OMR_D void named_barrier(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// ... that tells all of its threads whether any of them brought `x`
OMR_D bool named_barrier_any(int id, int threads, bool x) {
  uint32_t any;
  asm volatile(
      "{.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %3, 0;\n\t"
      "bar.red.or.pred p, %1, %2, q;\n\t"
      "selp.u32 %0, 1, 0, p;}"
      : "=r"(any)
      : "r"(id), "r"(threads), "r"((uint32_t)x)
      : "memory");
  return any != 0;
}

template <class F, int LOGT, int MODE>
OMR_D void duo_issue_load(const CUtensorMap* map, const PassArgs<F>& a, uint64_t tile, unsigned char* buf,
                          uint64_t* bar) {
  using E = typename F::E;
  constexpr int T = 1 << LOGT, C = kDuoCols;
  uint32_t g, lm;
  uint64_t lb;
  tile_coords<F, C>(a, tile, g, lm, lb);
  mbar_arrive_expect_tx(bar, (uint32_t)(T * C * F::WORD));
  if constexpr (MODE == MODE_COL) {
    const int y0 = (int)((lb * a.L_m + lm) * (uint64_t)T);
#pragma unroll 1
    for (int t = 0; t < T; t += 256) tma_load_2d(buf + t * C * F::WORD, map, (int)(g * C), y0 + t, bar);
  } else {
    const E* src = a.in + (lb * a.is_b + lm * a.is_m + (uint64_t)(g * C) * a.is_lo);
#pragma unroll 1
    for (int c = 0; c < C; c++)
      bulk_load(buf + c * duo_line_bytes<LOGT>(), src + (uint64_t)c * a.is_lo, T * F::WORD, bar);
  }
}

template <class F, int LOGT, int MODE>
OMR_D void duo_issue_store(const CUtensorMap* map, const PassArgs<F>& a, uint64_t tile, const unsigned char* buf) {
  constexpr int T = 1 << LOGT, C = kDuoCols;
  uint32_t g, lm;
  uint64_t lb;
  tile_coords<F, C>(a, tile, g, lm, lb);
  const int x = MODE == MODE_COL ? (int)(g * C) : (int)(g * C + lm * (uint32_t)a.os_m);
  const int y0 = MODE == MODE_COL ? (int)((lb * a.L_m + lm) * (uint64_t)T) : (int)(lb * (uint64_t)T);
#pragma unroll 1
  for (int t = 0; t < T; t += 256) tma_store_2d(map, x, y0 + t, buf + t * C * F::WORD);
  bulk_commit();
}

// The transform of one thread's line: line 4 ch + c of the team's tile.
template <class F, int LOGT, int MODE, bool INV, bool TW>
OMR_D void duo_lines(const PassArgs<F>& a, unsigned char* s, const typename F::Tw* tab, uint32_t llo0, uint32_t lm,
                     int team) {
  using E = typename F::E;
  constexpr int T = 1 << LOGT, R1 = 32, L = T / R1, LOGL = LOGT - 5;
  constexpr int GT = duo_group_threads<LOGT>();
  constexpr bool ROWS = MODE == MODE_COL;
  constexpr int PER = R1 / L;        // second-round DFTs per thread
  constexpr uint32_t RB = ROWS ? kDuoRowBytes : 4;  // bytes per entry step
  constexpr int NT = duo_team_threads<LOGT>();
  const uint32_t ch = threadIdx.x % NT / GT, tid = threadIdx.x % GT;
  const auto group_sync = [&] { named_barrier(1 + (int)(threadIdx.x / kDuoSyncThreads), kDuoSyncThreads); };
  const uint32_t c = tid & 3, l = tid >> 2;  // l < L
  const auto at = [&](uint32_t k) { return duo_at<LOGT, ROWS>(l, k, ch, c); };  // entry l ^ k
  E v[R1];
  {
    const unsigned char* p = s + at(0);
#pragma unroll
    for (int m = 0; m < R1; m++) v[m] = *reinterpret_cast<const E*>(p + L * m * RB);  // entries l + L m
  }
  group_sync();  // the group's reads precede its exchange
  dft_reg_mul<F, 5, INV>(v);
#pragma unroll
  for (int aa = 1; aa < R1; aa++) v[aa] = F::mul_tw(v[aa], tab[(aa - 1) * L + l]);  // omega_T^(l a)
#pragma unroll
  for (int aa = 0; aa < R1; aa++)
    *reinterpret_cast<E*>(s + L * aa * RB + at((uint32_t)(aa & (L - 1)))) = v[aa];
  group_sync();
#pragma unroll
  for (int i = 0; i < PER; i++) {
    const uint32_t am = l + L * i;
    const unsigned char* p = s + L * am * RB;
#pragma unroll
    for (int ll = 0; ll < L; ll++) v[i * L + ll] = *reinterpret_cast<const E*>(p + at((uint32_t)ll));
  }
  // the rows of a row pass's results span every group's lines
  if constexpr (ROWS)
    group_sync();
  else
    named_barrier(duo_team_barrier(team), NT);
#pragma unroll
  for (int i = 0; i < PER; i++) {
    const uint32_t am = l + L * i;  // outputs b < L are line entries am + 32 b
    E w[L];
#pragma unroll
    for (int b = 0; b < L; b++) w[b] = v[i * L + b];
    dft_reg<F, LOGL, INV, TW || INV>(w);
    // (TeddyBear, 16 points: keeps the compiler from mixing the chain below
    // into the DFT and spilling more; 64 x 2^18 122.7 -> 121.3 us)
    if constexpr (TW && !F::SMALL && L == 16) __syncwarp();
    if constexpr (TW) {
      const uint32_t line = llo0 + 4 * ch + c + lm * a.tw_line_mul_m, ls = line * a.tw_scale;
      const uint32_t e0 = (ls * am) & a.tw_mask, es = (ls * (uint32_t)R1) & a.tw_mask;
      E t = F::mul_tw(__ldg(&a.tw_lo[e0 & ((1u << kTwLoBits) - 1)]), a.tw_hi[e0 >> kTwLoBits]);
      const E step = F::mul_tw(__ldg(&a.tw_lo[es & ((1u << kTwLoBits) - 1)]), a.tw_hi[es >> kTwLoBits]);
#pragma unroll
      for (int b = 0; b < L; b++) {
        w[b] = mul_m<F>(w[b], t);
        if (b + 1 < L) t = F::mont_mul(t, step);
      }
    }
    if constexpr (INV && !TW) {  // the last pass of an inverse transform
#pragma unroll
      for (int b = 0; b < L; b++) w[b] = F::mul_tw(w[b], a.scale);
    }
    unsigned char* p = s + duo_row(am, ch) + 4 * c;
#pragma unroll
    for (int b = 0; b < L; b++) *reinterpret_cast<E*>(p + R1 * b * kDuoRowBytes) = w[b];
  }
}

template <class F, int LOGT, int MODE, bool INV, bool TW>
__global__ void __launch_bounds__(duo_teams<LOGT>() * duo_team_threads<LOGT>(),
                                  1024 / (duo_teams<LOGT>() * duo_team_threads<LOGT>()))
    ntt_duo_pass(const __grid_constant__ CUtensorMap in_map, const __grid_constant__ CUtensorMap out_map,
                 const PassArgs<F> a, int* err) {
  using Tw = typename F::Tw;
  constexpr int C = kDuoCols, NT = duo_team_threads<LOGT>(), TEAMS = duo_teams<LOGT>(), L = (1 << LOGT) / 32;
  constexpr int NB = duo_bufs<LOGT>(), BB = duo_buf_bytes<LOGT>();
  extern __shared__ __align__(1024) unsigned char duo_smem_raw[];
  __shared__ __align__(8) uint64_t sent[NB], full[NB];  // the buffer's load issued, landed
  __shared__ uint32_t issued[NB], landed[NB];  // loads of each buffer
  __shared__ volatile int abort_flag;
  unsigned char* base = duo_smem_raw + ((1024u - (smem_u32(duo_smem_raw) & 1023u)) & 1023u);
  Tw* tab = reinterpret_cast<Tw*>(base + NB * BB);

  // this CTA's tiles: blockIdx.x + j gridDim.x, j < njobs; team j mod TEAMS, buffer j mod NB
  const uint64_t ntiles = a.L_b * (uint64_t)a.L_m * (a.L_lo / C);
  const uint32_t njobs =
      ntiles > blockIdx.x ? (uint32_t)((ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x) : 0u;
  const auto issue = [&](uint32_t j) {
    const uint32_t b = j % NB;
    issued[b]++;
    if (TEAMS > 1) mbar_arrive(&sent[b]);
    duo_issue_load<F, LOGT, MODE>(&in_map, a, blockIdx.x + (uint64_t)j * gridDim.x, base + b * BB, &full[b]);
  };
  if (threadIdx.x == 0) {
    prefetch_tmap(&in_map);
    prefetch_tmap(&out_map);
    for (int b = 0; b < NB; b++) {
      mbar_init(&sent[b], 1);
      mbar_init(&full[b], 1);
      issued[b] = landed[b] = 0;
    }
    fence_mbar_init();
    fence_proxy_async();
    abort_flag = 0;
    // the previous pass's output is this one's input (and its input may be
    // this one's output): the loads and stores of the pass follow this wait
    grid_dep_wait();
    for (uint32_t j = 0; j < (uint32_t)NB && j < njobs; j++) issue(j);
  }
  grid_dep_launch();
  for (int i = threadIdx.x; i < 31 * L; i += TEAMS * NT) tab[i] = round_table<F, 5, LOGT - 5>(a)[L + i];
  __syncthreads();

  const int team = TEAMS == 1 ? 0 : (int)(threadIdx.x / NT);
  const bool leader = threadIdx.x % NT == 0;
  struct Ops {  // (team_ring.cuh)
    const CUtensorMap* out_map;
    const PassArgs<F>& a;
    unsigned char* base;
    const Tw* tab;
    uint64_t *sent, *full;
    uint32_t* landed_;
    volatile int* abort_flag;
    int* err;
    int team;
    const decltype(issue)& issue_;
    OMR_D uint64_t tile(uint32_t j) const { return blockIdx.x + (uint64_t)j * gridDim.x; }
    OMR_D bool wait_issued(uint32_t b, uint32_t parity) { return mbar_wait_bounded(&sent[b], parity); }
    OMR_D bool wait_landed(uint32_t b, uint32_t parity) { return mbar_wait_bounded(&full[b], parity); }
    OMR_D void gave_up() {
      atomicExch(err, OMR_NTT_ERR_TIMEOUT);
      *abort_flag = 1;
    }
    OMR_D bool aborted() { return *abort_flag != 0; }
    OMR_D void landed(uint32_t b) { landed_[b]++; }
    OMR_D void issue(uint32_t j) {
      fence_proxy_async();
      issue_(j);
    }
    OMR_D void transform(uint32_t j, uint32_t b) {
      uint32_t g, lm;
      uint64_t lb;
      tile_coords<F, C>(a, tile(j), g, lm, lb);
      duo_lines<F, LOGT, MODE, INV, TW>(a, base + b * BB, tab, g * C, lm, team);
      fence_proxy_async();  // this thread's writes become visible to the TMA store
    }
    OMR_D bool any(bool x) { return named_barrier_any(duo_team_barrier(team), NT, x); }
    OMR_D void store(uint32_t j, uint32_t b) {
      duo_issue_store<F, LOGT, MODE>(out_map, a, tile(j), base + b * BB);
    }
    OMR_D void store_read() { bulk_wait_read_all(); }
  } ops{&out_map, a, base, tab, sent, full, landed, &abort_flag, err, team, issue};
  team_ring_run<NB, TEAMS>(ops, (uint32_t)team, leader, njobs);
  if (leader) bulk_wait_all();
  __syncthreads();
  // after a wait that gave up, loads may still be in flight
  if (threadIdx.x == 0)
    for (int b = 0; b < NB; b++)
      if (issued[b] != landed[b]) mbar_wait_bounded(&full[b], landed[b] & 1);
}

}  // namespace omr
