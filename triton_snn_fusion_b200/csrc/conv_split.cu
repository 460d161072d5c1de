// 3x3 / 1x1 conv (+ bias, + residual or fused 1x1 shortcut conv) + LIF for calls with few output tiles: the reduction
// of a tile is split over a cluster of CTAs.
//
// What bounds such a call on the timestep-pair kernel (conv_pair_impl.cuh) is one serial chain: 512 -> 512 channels on
// the 7x7 maps of one image is four tiles, each 72 weight tiles x 4 instructions x 2 timestep pairs long, on 4 of 148
// SMs. Here the weight tiles (tap, 64-channel slab) of a tile are dealt to the S CTAs of a cluster in contiguous runs;
// each CTA multiplies its run with the halo tiles of up to four timesteps at once (512 columns of tensor memory; a weight
// tile is fetched once for all of them) and spills its partial sums to its own shared memory. After a cluster barrier every
// CTA collects a share of the tile's rows from all S CTAs over distributed shared memory, adds bias and residual and runs
// the LIF. More than four timesteps run as windows of four.
//
// The operand layout (128 output channels as M, 8 x 14 pixels of two timesteps as N = 256, taps as shifted descriptors
// into a 10 x 16 halo tile, two images per tile on maps of at most 7 x 8) is that of the timestep-pair kernel. Which
// calls come here: conv_split_plan() below.
#include <atomic>
#include <type_traits>

#include "conv.cuh"
#include "tmap.cuh"
#include "umma.cuh"

namespace snnb {

static __device__ int g_split_status = 0;

namespace {

constexpr int kPW = 10, kPH = 16, kRowBytes = kPW * 128, kHaloT = kPW * kPH * 128;
constexpr int kRows = 14;                 // output rows of a tile
constexpr int kWSlot = 128 * 128;
constexpr int kMaxTw = 4;                 // timesteps per window
constexpr int kMaxRing = 3, kMaxWRing = 8;
constexpr int kEpi = 8, kHaloWarp = 8, kWWarp = 9, kMmaWarp = 10, kThreads = 32 * 11;
constexpr uint32_t kStageT = kRows * 2 * 128 * 16;             // a timestep's partial sums: [row][half row][channel][4]
constexpr int kStageBytes = kMaxTw * kStageT;
constexpr int kSmem = kStageBytes + 1024;
constexpr int kMargin = 4 * kRowBytes;    // the last descriptor groups read (unused) rows past a slot
static_assert(2 * kMaxTw * kHaloT + 3 * kWSlot + kMargin <= kStageBytes, "rings fit under the staging area");
static_assert(kSmem <= 226 * 1024, "shared memory");

struct SplitGeom {
  int T, B, Cout, Ho, Wo;
  int kslabs, sc_slabs, ntaps, s2, stack;
  int nws;                    // weight tiles of a tile: kslabs * ntaps + sc_slabs
  int n_tiles_n, row_tiles, w_strips;
  int S, ring, wring, tw, nwin, lif, own, Cin;
  long long wait_limit;       // bound of every mbarrier wait, in SM cycles
  int drop_load;              // self-test: CTA 0 announces its first weight tile but never loads it
};

// Walks the weight tiles of a run: `slab` (64 input channels; slabs of the shortcut input follow those of the conv) and
// the position `r` in the slab's taps. Stride 2 deals the nine taps of a slab to four phase tiles (row parity a, column
// parity b; input row 2i - 1 + kh is row i - 1 of phase a = 1 for kh = 0, i of a = 0 for kh = 1, i of a = 1 for kh = 2):
// taps 4 | 3 5 | 1 7 | 0 2 6 8 read the tiles of phase 0 | 1 | 2 | 3.
struct Walk {
  int slab, r;
  __device__ __forceinline__ Walk(const SplitGeom &g, int ws) {
    const int main = g.kslabs * g.ntaps;
    if (ws >= main) { slab = g.kslabs + ws - main; r = 0; }
    else { slab = ws / g.ntaps; r = ws - slab * g.ntaps; }
  }
  __device__ __forceinline__ bool sc(const SplitGeom &g) const { return slab >= g.kslabs; }
  __device__ __forceinline__ int phase(const SplitGeom &g) const { return g.s2 && !sc(g) ? (r < 1 ? 0 : r < 3 ? 1 : r < 5 ? 2 : 3) : 0; }
  __device__ __forceinline__ int wtap(const SplitGeom &g) const { return g.s2 ? (int)(0x862071534ull >> (4 * r)) & 15 : r; }
  __device__ __forceinline__ int off(const SplitGeom &g) const {   // row offset in the halo tile
    if (g.ntaps == 1 || sc(g)) return kPW + 1;
    return g.s2 ? (int)(0xba10b1babull >> (4 * r)) & 15 : (r / 3) * kPW + r % 3;
  }
  // step to the next weight tile; true if it reads another input tile
  __device__ __forceinline__ bool next(const SplitGeom &g) {
    ++r;
    if (sc(g) || r == g.ntaps) { r = 0; ++slab; return true; }
    return g.s2 && (r == 1 || r == 3 || r == 5);
  }
};

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float4 ld_cluster(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void tmem_ld_x8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr) : "memory");
}

// Half a row (4 pixels) of one channel: sums of the S CTAs -> bias, residual, LIF over the window's steps. `mine`: which
// of the pixels are written; the others are computed on whatever lies at a valid address, so that only the stores are
// predicated. FAST: the common LIF kind (tau a power of two, hard reset).
template <bool FAST, typename XT, typename ST, typename VT>
__device__ __forceinline__ void split_unit(const SplitGeom &g, const LifParams &p, uint32_t src, int r, long long o, int mine,
                                           float (&v)[4], int win, int t0, int tw, float bias_c, const XT *__restrict__ res,
                                           const VT *v_init, ST *__restrict__ spikes, VT *v_out) {
  const long long frame_out = (long long)g.B * g.Ho * g.Wo * g.Cout;
  const long long o0 = t0 * frame_out + o;
  int po[4];   // pixel offsets; an absent pixel reads pixel 0 of the first channel, which exists
#pragma unroll
  for (int i = 0; i < 4; ++i) po[i] = i * g.Cout;
  auto at = [&](long long base, int i) { return (mine >> i & 1) ? base + po[i] : 0ll; };
  float rs[kMaxTw][4];
#pragma unroll
  for (int q = 0; q < kMaxTw; ++q)
#pragma unroll
    for (int i = 0; i < 4; ++i) rs[q][i] = 0.f;
  if (res != nullptr) {
#pragma unroll
    for (int q = 0; q < kMaxTw; ++q)
      if (q < tw) {
#pragma unroll
        for (int i = 0; i < 4; ++i) rs[q][i] = DT<XT>::to_f(res[at(o0 + q * frame_out, i)]);
      }
  }
  if (win == 0 && g.lif && v_init != nullptr) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      v[i] = DT<VT>::to_f(v_init[at(o, i)]);
  }
  float4 y[kMaxTw];
#pragma unroll
  for (int q = 0; q < kMaxTw; ++q) y[q] = make_float4(0.f, 0.f, 0.f, 0.f);
  // The sum of the S partial sums, each CTA starting with its own: at any time the CTAs of a cluster read different ones
  // (with all of them on rank 0 first the slowest took twice as long). Opposite partial sums are added first, then the sums a
  // quarter turn apart, and so on: a + b = b + a makes that the same number wherever one starts, so a pixel that two
  // shifted tiles compute, or an image in the other half of a tile, comes out the same.
  const int half = g.S >> 1, quarter = g.S >> 2;
  auto add = [](float4 &a, const float4 &b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; };
#pragma unroll
  for (int q0 = 0; q0 < kMaxTw; q0 += 2) {   // two timesteps at a time: eight loads in flight, which the registers hold
    if (q0 < tw) {
      const bool two = q0 + 1 < tw;
#pragma unroll 1
      for (int turn = 0; turn < (quarter > 1 ? 2 : 1); ++turn) {
        float4 part[4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < 2 || quarter) {
            const uint32_t from = map_rank(src, (uint32_t)((r + turn + (i & 1) * half + (i >> 1) * quarter) & (g.S - 1))) + (uint32_t)q0 * kStageT;
            part[i][0] = ld_cluster(from);
            if (two) part[i][1] = ld_cluster(from + kStageT);
          }
#pragma unroll
        for (int j = 0; j < 2; ++j)
          if (j == 0 || two) {
            add(part[0][j], part[1][j]);
            if (quarter) {
              add(part[2][j], part[3][j]);
              add(part[0][j], part[2][j]);
            }
            add(y[q0 + j], part[0][j]);
          }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < kMaxTw; ++q)
    if (q < tw) {
      const float cur[4] = {y[q].x, y[q].y, y[q].z, y[q].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float in = (cur[i] + bias_c) + rs[q][i];
        ST *to = spikes + (o0 + q * frame_out + po[i]);
        if (FAST || g.lif) {
          const ST spike = DT<ST>::from_f(FAST ? lif_step_t<1, true>(in, v[i], p) : lif_step(in, v[i], p));
          if (mine >> i & 1) *to = spike;
        } else if (mine >> i & 1) {
          reinterpret_cast<XT *>(spikes)[o0 + q * frame_out + po[i]] = DT<XT>::from_f(in);
        }
      }
    }
  if (win + 1 == g.nwin && g.lif && v_out != nullptr) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (mine >> i & 1) v_out[o + po[i]] = DT<VT>::from_f(v[i]);
  }
}

template <typename XT, typename ST, typename VT>
__global__ void __launch_bounds__(kThreads, 1)
conv_split_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                  const __grid_constant__ CUtensorMap scxmap, const __grid_constant__ CUtensorMap scwmap,
                  const __grid_constant__ CUtensorMap xmap01, const __grid_constant__ CUtensorMap xmap10,
                  const __grid_constant__ CUtensorMap xmap11, const XT *__restrict__ bias, const XT *__restrict__ bias2,
                  const XT *__restrict__ res, const VT *v_init, ST *__restrict__ spikes, VT *v_out, const SplitGeom g,
                  const LifParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * kMaxRing + 2 * kMaxWRing + 1];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  umma::pdl_trigger();

  const uint32_t smem_base = (umma::smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t w_base = smem_base, h_base = smem_base + (uint32_t)(g.wring * kWSlot);
  const uint32_t slot_bytes = (uint32_t)(g.tw * kHaloT);
  const uint32_t bar_base = umma::smem_u32(bars);
  auto hfull = [&](uint32_t s) { return bar_base + 8u * s; };
  auto hempty = [&](uint32_t s) { return bar_base + 8u * (kMaxRing + s); };
  auto wfull = [&](uint32_t s) { return bar_base + 8u * (2 * kMaxRing + s); };
  auto wempty = [&](uint32_t s) { return bar_base + 8u * (2 * kMaxRing + kMaxWRing + s); };
  const uint32_t accfull = bar_base + 8u * (2 * kMaxRing + 2 * kMaxWRing);
  volatile int *abort_flag = &abort_s;
  const long long wl = g.wait_limit;

  // this cluster's tile (channel tile fastest), this CTA's run of weight tiles
  const int rank = (int)(blockIdx.x % (unsigned)g.S), tile = (int)(blockIdx.x / (unsigned)g.S);
  const int n0 = (tile % g.n_tiles_n) * 128;
  int b, w0 = 0, h0 = 0, wlo = 0, hlo = 0;
  {
    int m = tile / g.n_tiles_n;
    if (g.stack) {
      b = 2 * m;
    } else {   // the last strip / row tile is shifted back inside the image and recomputes pixels of its neighbour
      const int strip = m % g.w_strips;
      m /= g.w_strips;
      const int rt = m % g.row_tiles;
      b = m / g.row_tiles;
      w0 = min(strip * 8, max(g.Wo - 8, 0));
      h0 = min(rt * kRows, max(g.Ho - kRows, 0));
      if (g.own) { wlo = strip * 8; hlo = rt * kRows; }   // membrane in place: shared pixels belong to one tile
    }
  }
  const int ws0 = (int)((long long)g.nws * rank / g.S), ws1 = (int)((long long)g.nws * (rank + 1) / g.S);

  if (threadIdx.x == 0) {
    abort_s = 0;
    for (int s = 0; s < g.ring; ++s) { umma::mbar_init(hfull(s), 1); umma::mbar_init(hempty(s), 1); }
    for (int s = 0; s < g.wring; ++s) { umma::mbar_init(wfull(s), 1); umma::mbar_init(wempty(s), 1); }
    umma::mbar_init(accfull, 1);
    umma::fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    umma::tmem_alloc(umma::smem_u32(&tmem_base_s), 512u);
    umma::tmem_relinquish();
  }
  if (warp == kHaloWarp && lane == 0) {
    umma::prefetch_tensormap(&xmap);
    umma::prefetch_tensormap(&wmap);
  }
  umma::tc_fence_before_sync();
  __syncthreads();
  umma::tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  umma::pdl_wait();   // from here on: reads what the predecessor in the stream wrote, writes what it may read

  uint32_t slot = 0, ws_slot = 0;
  uint32_t phase = warp == kMmaWarp ? 0u : 1u, wphase = phase;   // the producers' first waits pass
  bool ok = true;

  // ---- epilogue state: rows [vr0, vr1) of the tile's valid rows are this CTA's; a unit is half a row (4 pixels), the
  // two warps of a lane quarter take alternate units
  const int nimg = g.stack ? (b + 1 < g.B ? 2 : 1) : 1;
  const int rows_img = min(g.Ho, g.stack ? 7 : kRows);
  const int nvr = nimg * rows_img;
  const int rp = (nvr + g.S - 1) / g.S, vr0 = min(rank * rp, nvr), vr1 = min(vr0 + rp, nvr);
  const int quarter = warp & 3, ch = quarter * 32 + lane, c = n0 + ch;
  const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
  // where this thread's channel of half a row (4 pixels) lies: [timestep][row][half row][channel]
  auto stage_at = [&](int q, int row, int half) { return (uint32_t)q * kStageT + (uint32_t)((row * 2 + half) * 2048 + ch * 16); };
  constexpr int kUnits = 7;   // at S >= 2 a CTA owns at most seven rows: seven units per warp
  float v[kUnits][4];         // membranes between windows (thread-local memory: indexed by a real loop)
  const bool c_ok = warp < kEpi && c < g.Cout;
  const float bias_c = ((bias != nullptr && c_ok) ? DT<XT>::to_f(bias[c]) : 0.f) +
                       ((bias2 != nullptr && c_ok) ? DT<XT>::to_f(bias2[c]) : 0.f);
  for (int win = 0; win < g.nwin; ++win) {
    const int t0 = win * g.tw, tw = min(g.tw, g.T - t0);
    if (warp == kHaloWarp) {
      // ------------------------------------------------- halo producer: lane q loads timestep t0 + q
      Walk at(g, ws0);
      bool fresh = true;
      for (int ws = ws0; ws < ws1 && ok; ++ws) {
        const int ph = at.phase(g);
        const CUtensorMap *xm = at.sc(g) ? &scxmap : (ph == 0 ? &xmap : (ph == 1 ? &xmap01 : (ph == 2 ? &xmap10 : &xmap11)));
        const int c0 = (at.sc(g) ? at.slab - g.kslabs : at.slab) * 64;
        const bool load = fresh;
        fresh = at.next(g);
        if (!load) continue;
        if (lane == 0) {
          ok = umma::mbar_wait(hempty(slot), phase, abort_flag, wl);
          if (ok) umma::mbar_expect_tx(hfull(slot), (uint32_t)tw * (g.stack ? (uint32_t)nimg * 9u * kRowBytes : (uint32_t)kHaloT));
        }
        ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
        if (!ok) break;
        if (lane < tw) {
          const uint32_t dst = h_base + slot * slot_bytes + (uint32_t)lane * (uint32_t)kHaloT;
          umma::tma_load_5d(dst, xm, hfull(slot), c0, w0 - 1, h0 - 1, b, t0 + lane);
          if (g.stack && nimg == 2) umma::tma_load_5d(dst + 8u * kRowBytes, xm, hfull(slot), c0, -1, -1, b + 1, t0 + lane);
        }
        if (++slot == (uint32_t)g.ring) { slot = 0; phase ^= 1u; }
      }
      __syncwarp();
    } else if (warp == kWWarp) {
      // ---------------------------------------------------------- weight producer
      if (lane == 0) {
        Walk at(g, ws0);
        for (int ws = ws0; ws < ws1 && ok; ++ws, at.next(g)) {
          ok = umma::mbar_wait(wempty(ws_slot), wphase, abort_flag, wl);
          if (!ok) break;
          umma::mbar_expect_tx(wfull(ws_slot), (uint32_t)kWSlot);
          const uint32_t dst = w_base + ws_slot * (uint32_t)kWSlot;
          if (g.drop_load && blockIdx.x == 0 && win == 0 && ws == ws0) {
            // self-test of the bounded waits: this tile never arrives
          } else if (at.sc(g)) {
            umma::tma_load_2d(dst, &scwmap, wfull(ws_slot), (at.slab - g.kslabs) * 64, n0);
          } else {
            umma::tma_load_2d(dst, &wmap, wfull(ws_slot), at.wtap(g) * g.Cin + at.slab * 64, n0);
          }
          if (++ws_slot == (uint32_t)g.wring) { ws_slot = 0; wphase ^= 1u; }
        }
      }
      __syncwarp();
    } else if (warp == kMmaWarp) {
      // -------------------------------------------------------------- MMA issuer
      {
        const uint32_t leader = umma::elect_one() ? 1u : 0u;
        const bool bf16 = std::is_same<XT, __nv_bfloat16>::value;
        const uint32_t id256 = umma::make_idesc_f16(128, 256, bf16), id128 = umma::make_idesc_f16(128, 128, bf16);
        uint64_t hdesc0 = umma::make_sw128_kmajor_desc(h_base);
        hdesc0 = (hdesc0 & ~((uint64_t)0x3FFF << 32)) | ((uint64_t)(kRowBytes >> 4) << 32);
        const uint64_t wdesc0 = umma::make_sw128_kmajor_desc(w_base);
        Walk at(g, ws0);
        bool fresh = true;
        for (int ws = ws0; ws < ws1 && ok; ++ws) {
          if (fresh) {
            ok = umma::mbar_wait_warp(hfull(slot), phase, abort_flag, wl);
            if (!ok) break;
          }
          ok = umma::mbar_wait_warp(wfull(ws_slot), wphase, abort_flag, wl);
          if (!ok) break;
          umma::tc_fence_after_sync();
          const uint64_t wdesc = wdesc0 + (uint64_t)((ws_slot * (uint32_t)kWSlot) >> 4);
          const uint64_t xdesc = hdesc0 + (uint64_t)((slot * slot_bytes + (uint32_t)at.off(g) * 128u) >> 4);
#pragma unroll
          for (int q = 0; q < kMaxTw; q += 2)
            if (q < tw) {
#pragma unroll
              for (int k = 0; k < 4; ++k)
                umma::mma_f16_ss_by(leader, tmem_base + (uint32_t)(q * 128), wdesc + (uint64_t)(2 * k),
                                 xdesc + (uint64_t)((q * kHaloT >> 4) + 2 * k), q + 1 < tw ? id256 : id128,
                                 (ws > ws0 || k > 0) ? 1u : 0u);
            }
          umma::mma_commit_by(leader, wempty(ws_slot));
          if (++ws_slot == (uint32_t)g.wring) { ws_slot = 0; wphase ^= 1u; }
          fresh = at.next(g);
          if (fresh || ws + 1 == ws1) {
            umma::mma_commit_by(leader, hempty(slot));
            if (++slot == (uint32_t)g.ring) { slot = 0; phase ^= 1u; }
          }
        }
        if (ok) umma::mma_commit_by(leader, accfull);
      }
      __syncwarp();
    } else {
      // --------------------------- partial sums: tensor memory -> this CTA's shared memory (the rings are idle now)
      if (lane == 0) ok = umma::mbar_wait(accfull, (uint32_t)(win & 1), abort_flag, wl);
      ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
      umma::tc_fence_after_sync();
      if (ok) {
        for (int q = 0; q < tw; ++q)
          for (int vr = warp >> 2; vr < nvr; vr += 2) {
            uint32_t a[8];
            tmem_ld_x8(lane_base + (uint32_t)(q * 128 + (vr + ((g.stack && vr >= rows_img) ? 8 - rows_img : 0)) * 8), a);
            umma::tmem_ld_wait();
            const uint32_t dst = smem_base + stage_at(q, vr, 0);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]) : "memory");
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + 2048u), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]) : "memory");
          }
      }
      umma::tc_fence_before_sync();
    }
    __syncwarp();
    cluster_sync_all();   // every CTA's partial sums of this window are in its shared memory
    if (warp < kEpi) {
      // ------------------------------------------------------ collect, bias, residual, LIF, spikes out
      // A CTA has a few units per warp and nothing to overlap them with, so a unit is written for latency: no branch
      // per pixel, loads before their uses, a real loop over the units.
      const bool fast = g.lif && p.mode == 1 && p.hard;
#pragma unroll 1
      for (int k = 0; k < kUnits; ++k) {
        const int u = 2 * k + (warp >> 2), vr = vr0 + (u >> 1), half = u & 1;
        if (vr >= vr1) break;   // warp-uniform
        const int img = b + (vr >= rows_img ? 1 : 0);
        const int row = h0 + (vr >= rows_img ? vr - rows_img : vr), col = w0 + 4 * half;
        const long long o = (((long long)img * g.Ho + row) * g.Wo + col) * g.Cout + c;
        int mine = 0;   // which of the four pixels exist and are this tile's to write
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (c_ok && col + i < g.Wo && col + i >= wlo && row >= hlo) mine |= 1 << i;
        const uint32_t src = smem_base + stage_at(0, vr, half);
        float vk[4] = {0.f, 0.f, 0.f, 0.f};
        if (win > 0) {
#pragma unroll
          for (int i = 0; i < 4; ++i) vk[i] = v[k][i];
        }
        if (fast) split_unit<true>(g, p, src, rank, o, mine, vk, win, t0, tw, bias_c, res, v_init, spikes, v_out);
        else split_unit<false>(g, p, src, rank, o, mine, vk, win, t0, tw, bias_c, res, v_init, spikes, v_out);
        if (win + 1 < g.nwin) {
#pragma unroll
          for (int i = 0; i < 4; ++i) v[k][i] = vk[i];
        }
      }
    }
    if (win + 1 < g.nwin) umma::fence_proxy_async_smem();   // the next window's copies overwrite the staging area
    __syncwarp();
    cluster_sync_all();   // nobody reads this CTA's shared memory any more
    umma::tc_fence_after_sync();
  }

  umma::tc_fence_before_sync();
  __syncthreads();
  if (abort_s && threadIdx.x == 0) atomicExch(&g_split_status, 1);
  if (warp == kMmaWarp) {
    umma::tc_fence_after_sync();
    umma::tmem_dealloc(tmem_base, 512u);
  }
}

template <typename XT, typename ST, typename VT>
int launch(const ConvArgs &a, int S, cudaStream_t stream) {
  SplitGeom g;
  g.T = a.T; g.B = a.B; g.Cout = a.Cout; g.Ho = a.Ho; g.Wo = a.Wo; g.Cin = a.Cin;
  g.kslabs = (a.Cin + 63) / 64;
  g.sc_slabs = a.sc_x != nullptr ? a.sc_cin / 64 : 0;
  g.ntaps = a.KH * a.KW;
  g.s2 = a.stride == 2 ? 1 : 0;
  g.stack = (a.Ho <= 7 && a.Wo <= 8) ? 1 : 0;
  g.nws = g.kslabs * g.ntaps + g.sc_slabs;
  g.n_tiles_n = (a.Cout + 127) / 128;
  g.row_tiles = (a.Ho + kRows - 1) / kRows;
  g.w_strips = (a.Wo + 7) / 8;
  g.S = S;
  g.tw = a.T < kMaxTw ? a.T : kMaxTw;
  g.nwin = (a.T + g.tw - 1) / g.tw;
  g.ring = g.tw > 2 ? 2 : 3;
  g.wring = g.tw > 3 ? 3 : (g.tw > 2 ? 4 : 5);
  g.lif = a.lif;
  g.own = (a.lif && a.v_init != nullptr && a.v_init == a.v_out) ? 1 : 0;
  g.wait_limit = 4000000000ll;
  g.drop_load = 0;
  consume_wait_selftest(&g.wait_limit, &g.drop_load);
  const long long tiles = g.stack ? (long long)((a.B + 1) / 2) * g.n_tiles_n
                                  : (long long)a.B * g.row_tiles * g.w_strips * g.n_tiles_n;
  const int es = 2;
  CUtensorMap xph[4], wm, scx, scw;
  const cuuint64_t frame_bytes = (cuuint64_t)a.B * a.H * a.W * a.Cin * es;
  const cuuint32_t box_h = (cuuint32_t)(g.stack ? 9 : kPH);
  const int st = g.s2 ? 2 : 1;
  for (int ph = 0; ph < (g.s2 ? 4 : 1); ++ph) {
    const int pa = ph >> 1, pb = ph & 1;
    cuuint64_t dims[5] = {(cuuint64_t)a.Cin, (cuuint64_t)((a.W - pb + st - 1) / st), (cuuint64_t)((a.H - pa + st - 1) / st),
                          (cuuint64_t)a.B, (cuuint64_t)a.T};
    cuuint64_t strides[4] = {(cuuint64_t)st * a.Cin * es, (cuuint64_t)st * a.W * a.Cin * es, (cuuint64_t)a.H * a.W * a.Cin * es,
                             a.T > 1 ? (cuuint64_t)a.x_t_stride * es : frame_bytes};
    cuuint32_t box[5] = {64, kPW, box_h, 1, 1};
    const int rc = encode_tmap(&xph[ph], a.dtype, 5, static_cast<const char *>(a.x) + ((size_t)pa * a.W + pb) * a.Cin * es, dims, strides, box);
    if (rc != SNNB_OK) return rc;
  }
  if (!g.s2) xph[1] = xph[2] = xph[3] = xph[0];
  auto weight_map = [&](CUtensorMap *m, const void *w, cuuint64_t K) {
    cuuint64_t dims[2] = {K, (cuuint64_t)a.Cout};
    cuuint64_t strides[1] = {K * es};
    cuuint32_t box[2] = {64, 128};
    return encode_tmap(m, a.dtype, 2, w, dims, strides, box);
  };
  int rc = weight_map(&wm, a.w, (cuuint64_t)g.ntaps * a.Cin);
  if (rc != SNNB_OK) return rc;
  scx = xph[0];
  scw = wm;
  if (g.sc_slabs) {
    const cuuint64_t sC = (cuuint64_t)a.sc_cin, s_ = (cuuint64_t)a.sc_stride;
    cuuint64_t dims[5] = {sC, (cuuint64_t)a.Wo, (cuuint64_t)a.Ho, (cuuint64_t)a.B, (cuuint64_t)a.T};
    cuuint64_t strides[4] = {s_ * sC * es, s_ * (cuuint64_t)a.sc_W * sC * es, (cuuint64_t)a.sc_H * a.sc_W * sC * es,
                             (cuuint64_t)a.sc_t_stride * es};
    cuuint32_t box[5] = {64, kPW, box_h, 1, 1};
    rc = encode_tmap(&scx, a.dtype, 5, a.sc_x, dims, strides, box);
    if (rc != SNNB_OK) return rc;
    rc = weight_map(&scw, a.sc_w, sC);
    if (rc != SNNB_OK) return rc;
  }
  auto kern = conv_split_kernel<XT, ST, VT>;
  const cudaError_t e = raise_smem_limit_once<conv_split_kernel<XT, ST, VT>>(kSmem);
  if (e != cudaSuccess) return fail(SNNB_ERR_CUDA, "conv_lif: cannot raise the shared-memory limit: %s", cudaGetErrorString(e));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * S));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)S;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t le = cudaLaunchKernelEx(&cfg, kern, xph[0], wm, scx, scw, xph[1], xph[2], xph[3],
                                            static_cast<const XT *>(a.b), static_cast<const XT *>(a.b2),
                                            static_cast<const XT *>(a.res), static_cast<const VT *>(a.v_init),
                                            static_cast<ST *>(a.spikes), static_cast<VT *>(a.v_out), g, a.p);
  if (le != cudaSuccess) return fail(SNNB_ERR_CUDA, "conv_split: launch failed: %s", cudaGetErrorString(le));
  return SNNB_OK;
}

template <typename XT>
int dispatch(const ConvArgs &a, int S, cudaStream_t stream) {
  const bool s_u8 = a.lif && a.spike_dtype == SNNB_U8, v_f32 = a.lif && a.v_dtype == SNNB_F32;
  if (s_u8) return v_f32 ? launch<XT, uint8_t, float>(a, S, stream) : launch<XT, uint8_t, XT>(a, S, stream);
  return v_f32 ? launch<XT, XT, float>(a, S, stream) : launch<XT, XT, XT>(a, S, stream);
}

// How many clusters of S CTAs run at once, one CTA per SM. A cluster stays inside a GPC, and which SMs a GPC has differs
// from one GPU to the next, so this is asked of the device: 33 and 15 for S = 4 and 8 on the B200 that the figures below were
// taken on, not 148 / S. One tile more is a second wave: 128 -> 496 with a shortcut from 128, T = 6, 16 tiles with S = 8
// took 51 us, the timestep-pair kernel 34. Without a device the figures of that GPU.
int clusters_at_once(int S) {
  static std::atomic<int> known[64][3];
  const int si = S == 2 ? 0 : (S == 4 ? 1 : 2), fallback = S == 2 ? 72 : (S == 4 ? 33 : 15);
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    (void)cudaGetLastError();
    return fallback;
  }
  int n = known[dev][si].load(std::memory_order_relaxed);
  if (n > 0) return n;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(S * 148));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)S;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  using BF = __nv_bfloat16;   // every instantiation has the same block and shared memory, one block per SM
  if (raise_smem_limit_once<conv_split_kernel<BF, BF, BF>>(kSmem) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, conv_split_kernel<BF, BF, BF>, &cfg) != cudaSuccess || n < 1) {
    (void)cudaGetLastError();
    n = fallback;
  }
  known[dev][si].store(n, std::memory_order_relaxed);
  return n;
}

}  // namespace

// Cluster size for a call, 0 where splitting does not pay. Times in microseconds of one launch, measured on B200 and the
// same for all shapes within 15 %. Whole tiles: the timestep-pair kernel takes 6.5 + 0.41 per weight tile and timestep
// pair of a wave, 4.6 a pair at least (0.3 and two thirds of the tiles in its two-kernel-rows form for at most 64
// channels), 17.5 + 11 a pair at least where the LIF divides, 10 + 10 with a soft reset (6.5 a pair in the
// two-kernel-rows form, whose epilogue has twice the warps); odd T on the halo kernel as much per pair of steps; the 1x1
// kernel 4.5 + 0.95 per pair (3 more where the LIF divides; 2.0, 0.8 or 0.3 more with a residual whose rows are off
// 64-byte boundaries, are on them, or have at most 64 channels) + 0.38 per pair and slab. A cluster takes 4.3 (1x1: 3) +
// per window of up to four steps 2.2 (2.5) + its share of the weight tiles (0.55 each at three or four timesteps at once,
// 0.41 at one or two) + the exchange, 0.8 + 0.6 per timestep + 0.33 per timestep and row that a CTA owns (1.05 where the
// LIF divides, 0.6 with a soft reset, 0.45 for more than two rows at 1x1 in several windows; this part has nothing to
// hide behind, which is why two CTAs with seven rows each rarely pay). 512 -> 512 on one 7x7 map, T = 4: 59 us against 36
// / 23 / 16 with S = 2 / 4 / 8; 256 -> 512 stride 2 on one 14x14 map: 36 against 22 / 16 / 13; 256 -> 256 on nine 8x8
// maps, T = 1: 23 against 15 / 11 / 17 (144 CTAs in clusters of eight do not fit at once); 128 -> 128 stride 2 to 7x7,
// 116 images: 29 against 37 with S = 2. 1x1: 1408 -> 72 on 14 pixels, T = 12: 59 whole, 28 with S = 8; 640 -> 48 on 120
// tokens, T = 8: 23 whole, 29 with S = 8 (two windows for ten weight tiles: left whole). Split only for a clear gain (a
// tenth).
// A sum over S partial sums rounds elsewhere than the pair kernel's chain, so outputs of a small batch agree with those of
// a large one to fp32 rounding of the currents, not always bit for bit. Within a batch an image's place does not matter.
int conv_split_plan(const ConvArgs &a) {
  if (!pair_shape_supported(a) || a.T > 64) return 0;
  const bool stack = a.Ho <= 7 && a.Wo <= 8;
  const double tiles = (stack ? (a.B + 1) / 2 : (double)a.B * ((a.Ho + kRows - 1) / kRows) * ((a.Wo + 7) / 8)) * ((a.Cout + 127) / 128);
  const int sms = sm_count() > 0 ? sm_count() : 148;
  if (tiles > sms / 2) return 0;
  const int ntaps = a.KH * a.KW, kslabs = (a.Cin + 63) / 64, pairs = (a.T + 1) / 2;
  const int nws = kslabs * ntaps + (a.sc_x != nullptr ? a.sc_cin / 64 : 0);
  const bool twin = a.Cout <= 64 && ntaps == 9 && a.stride == 1 && a.sc_x == nullptr;
  // LIF kinds with a longer epilogue: 2 with a division, 1 with a soft reset
  const int kind = !a.lif ? 0 : (a.p.mode == 2 ? 2 : (a.p.hard ? 0 : 1));
  const double mma = twin ? 6 * kslabs * 0.3 : nws * 0.41;
  const double epilogue = twin ? (kind ? 6.5 : 0.0) : (kind == 2 ? 11.0 : (kind == 1 ? 10.0 : 4.6));
  double whole = (twin || kind == 0 ? 6.5 : (kind == 2 ? 17.5 : 10.0)) + pairs * (mma > epilogue ? mma : epilogue);   // conv_pair_impl.cuh
  if (ntaps == 1) {                                                                            // conv_pw.cu, one wave
    const double residual = a.res == nullptr ? 0.0 : (a.Cout <= 64 ? 0.3 : (a.Cout % 32 != 0 ? 2.0 : 0.8));
    whole = 4.5 + pairs * (0.95 + 0.38 * kslabs + (kind == 2 ? 3.0 : 0.0) + residual);
  }
  const int nwin = (a.T + kMaxTw - 1) / kMaxTw;
  const int rows = (a.Ho < kRows ? a.Ho : kRows) * (stack && a.B > 1 ? 2 : 1);
  // odd T, where the channel counts rule out the halo and the general kernel too: the CUDA cores take twenty times as long
  const char *why = "";
  const bool alone = ntaps == 9 && a.T % 2 != 0 && a.T != 1 && !conv3x3_halo_supported(a) && !conv_lif_tc_supported(a, &why);
  int best = 0;
  double best_us = alone ? 1e300 : 0.9 * whole;
  for (int S = 2; S <= 8 && S <= nws; S *= 2) {
    const int at_once = clusters_at_once(S), waves = ((int)tiles + at_once - 1) / at_once;
    const int share = (nws + S - 1) / S, owned = (rows + S - 1) / S;
    const double row_us = kind == 2 ? 1.05 : kind == 1 ? 0.6 : (ntaps == 1 && nwin > 1 && owned > 2 ? 0.45 : 0.33);
    double us = ntaps == 1 ? 3.0 + 2.5 * nwin : 4.3 + 2.2 * nwin;
    for (int win = 0; win < nwin; ++win) {
      const int tw = a.T - win * kMaxTw < kMaxTw ? a.T - win * kMaxTw : kMaxTw;
      us += share * (tw > 2 ? 0.55 : 0.41) + 0.8 + tw * (0.6 + row_us * owned);
    }
    if (us * waves < best_us) {
      best_us = us * waves;
      best = S;
    }
  }
  return best;
}

int conv_split(const ConvArgs &a, int S, cudaStream_t stream) {
  return a.dtype == SNNB_BF16 ? dispatch<__nv_bfloat16>(a, S, stream) : dispatch<__half>(a, S, stream);
}

int split_device_status(int *out) {
  int h = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&h, g_split_status, sizeof(int));
  if (e != cudaSuccess) return fail(SNNB_ERR_CUDA, "device_status: %s", cudaGetErrorString(e));
  if (h != 0) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_split_status, &zero, sizeof(int));
  }
  *out = h;
  return SNNB_OK;
}

}  // namespace snnb
