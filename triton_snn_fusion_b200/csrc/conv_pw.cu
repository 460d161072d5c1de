// 1x1 / stride 1 conv and linear (+ bias, + residual) + LIF over T steps on the tensor cores, 16-bit data: a GEMM over
// the pixels (tokens) of all images in a row.
//
//   D_pair[cout][tq * 128 + pixel] = sum_slab  W[cout][slab] . X_(2*pair+tq)[pixel][slab]^T
//
// A tile is 128 output channels (M) x 128 consecutive pixels of two timesteps (N = 256), whatever the map's shape: no
// rows or columns of a small map are wasted, and the last tile is shifted back to end with the last pixel. Timestep pairs
// alternate between two accumulators (TMEM columns 0..255 and 256..511), the membrane stays in registers over all pairs,
// an odd T ends with a pair of one (N = 128).
//
// Bound: with K = 32 .. 1024 the multiply-adds of a pair are short and its epilogue (32768 outputs: bias, LIF, one
// two-byte store each, 64 contiguous bytes per warp) is the longer part. In the timestep-pair kernel of the 3x3 convs,
// which these calls ran before, eight epilogue warps of 168 registers took 12.5 k cycles a pair, two thirds of their issue
// slots empty. Here sixteen warps share it, each thread one channel of 32 pixels; a spike is selected as the 16-bit
// pattern of 1.0, so an output is about seven instructions. Weights stay in shared memory for all tiles of a block when
// they fit beside the pixel ring (K <= 512; the block then walks the pixel tiles of one channel tile), which leaves only
// pixels to be fetched per pair.
#include <type_traits>

#include "conv.cuh"
#include "tmap.cuh"
#include "umma.cuh"

namespace snnb {

static __device__ int g_pw_status = 0;

namespace {

constexpr int kTile = 128 * 128;        // bytes of 128 rows x 64 channels
constexpr int kMaxStages = 6;
constexpr int kEpi = 16, kTmaWarp = 16, kMmaWarp = 17, kThreads = 32 * 18;
constexpr int kSmemData = 224 * 1024;
constexpr int kResidentSlabs = 8;       // weights of up to 512 input channels (128 KB) stay; the ring has three stages then
constexpr int kResAhead = 3, kResSlots = 4, kResWarp = kResSlots * 1024;   // residuals: steps fetched ahead, a warp's ring

struct PwGeom {
  int T, npairs, kslabs, Cout, n_tiles_n, m_tiles, stages, resident, lif, own;
  int kind;                 // what the epilogue computes (kLean ...)
  int res_staged;           // residuals pass through shared memory (Residuals below)
  int dup;                  // Cout <= 64: the weight rows twice (M rows 64..127 repeat 0..63), so that all epilogue warps have work
  long long P, frame_out;   // pixels of a frame; elements of an output frame
  long long wait_limit;     // bound of every mbarrier wait, in SM cycles
  int drop_load;            // self-test: block 0 announces its first stage but does not load its pixels
};

__device__ __forceinline__ long long first_pixel(const PwGeom &g, int m) { return max(0ll, min((long long)m * 128, g.P - 128)); }

// What the epilogue computes, fixed at compile time (a branch per output on the LIF's mode took four times as long): the
// common LIF (tau a power of two, hard reset to zero), the other LIF kinds as 1 + 2 * mode + hard, or no LIF.
constexpr int kLean = 0, kOff = 7;

// 16 pixels of one timestep. Common LIF: h = v + (y - v) * inv_tau; the product with a power of two is exact, so the fused
// multiply-add rounds the same sum as lif_step's separately rounded operations. MASK: only pixels whose bit is set are
// written. RES: r is added. WALK: the row pointer walks (in a loop over the steps the compiler would keep all 16 row offsets,
// which do not fit).
template <int KIND, bool MASK, bool RES, bool WALK, typename XT, typename ST>
__device__ __forceinline__ void lif16(const uint32_t (&a)[16], const XT (&r)[16], float bias, const LifParams &p, float *v, ST *out,
                                      int cs, uint32_t mask) {
  constexpr uint32_t one = std::is_same<ST, uint8_t>::value ? 1u : (std::is_same<ST, __half>::value ? 0x3C00u : 0x3F80u);
  using Bits = typename std::conditional<sizeof(ST) == 1, uint8_t, uint16_t>::type;
  ST *row = out;
  const float2 b2 = make_float2(bias, bias), it2 = make_float2(p.inv_tau, p.inv_tau);
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    float2 y = __fadd2_rn(make_float2(__uint_as_float(a[i]), __uint_as_float(a[i + 1])), b2);
    if (RES) y = __fadd2_rn(y, make_float2(DT<XT>::to_f(r[i]), DT<XT>::to_f(r[i + 1])));
    const bool w0 = !MASK || (mask >> i & 1u), w1 = !MASK || (mask >> (i + 1) & 1u);
    Bits *const to = reinterpret_cast<Bits *>(row);
    row += WALK ? 2 * cs : 0;
    const int at0 = WALK ? 0 : i, at1 = WALK ? 1 : i + 1;
    if constexpr (KIND == kOff) {
      XT *const plain = reinterpret_cast<XT *>(to);
      if (w0) plain[0] = DT<XT>::from_f(y.x);
      if (w1) plain[cs] = DT<XT>::from_f(y.y);
    } else {
      bool s0 = false, s1 = false;
      if constexpr (KIND == kLean) {
        const float2 d = __fadd2_rn(y, make_float2(-v[i], -v[i + 1]));
        const float2 h = __ffma2_rn(d, it2, make_float2(v[i], v[i + 1]));
        s0 = h.x >= p.v_th;
        s1 = h.y >= p.v_th;
        v[i] = s0 ? 0.f : h.x;
        v[i + 1] = s1 ? 0.f : h.y;
      } else {   // (absent pixels of the kinds with a division are not worth computing)
        if (KIND < 5 || w0) s0 = lif_step_t<(KIND - 1) / 2, (KIND - 1) % 2 == 1>(y.x, v[i], p) != 0.f;
        if (KIND < 5 || w1) s1 = lif_step_t<(KIND - 1) / 2, (KIND - 1) % 2 == 1>(y.y, v[i + 1], p) != 0.f;
      }
      if (w0) to[(long long)at0 * cs] = (Bits)(s0 ? one : 0u);
      if (w1) to[(long long)at1 * cs] = (Bits)(s1 ? one : 0u);
    }
  }
}

// A warp's residuals on their way to it. A thread's own are 2-byte reads from 16 rows, whose latency nothing covers (the
// registers hold one step's at most), and where the rows do not lie on 64-byte boundaries every one of them touches two or
// three lines more. There (`on`: Cout % 32 != 0; the copies also need Cout % 8 == 0 and a 16-byte aligned tensor) the
// steps of 16 pixels x 32 channels (1 KB) are copied to shared memory kResAhead steps before they are used: 0.73 of the
// time of direct reads over drawn calls (64 -> 136, 27900 pixels, T = 4: 68 -> 38 us). On 64-byte
// boundaries direct reads are the faster ones by 5 to 10 %, and with K > 512 the ring of operands needs the room.
template <typename XT>
struct Residuals {
  const XT *res;          // the whole tensor
  long long o0;           // this thread's first pixel and channel of the tile at timestep 0
  uint32_t smem;          // this warp's ring
  int nch, exist, npx;    // channels and pixels of the warp that exist; pixels of a full tile
  bool on;
  int t, half;            // the next step to be fetched
  uint32_t in, out;       // steps fetched and taken; slots are taken in turn, across tiles too
  __device__ __forceinline__ void fetch(const PwGeom &g) {   // the next step, if the tile has one
    const int lane = threadIdx.x & 31;
    if (t < g.T) {
      const uint32_t slot = smem + (in % kResSlots << 10);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int row = (lane >> 2) + 8 * k, ch = (lane & 3) * 8;
        const bool ok = half * 16 + row < exist && ch < nch;
        const XT *src = res + (ok ? o0 - lane + t * g.frame_out + (long long)(half * 16 + row) * g.Cout + ch : 0ll);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(slot + (uint32_t)(row * 64 + ch * 2)), "l"(src), "r"(ok ? 16 : 0) : "memory");
      }
      ++in;
      // both timesteps of a pair for the first 16 pixels, then for the second, then the next pair
      if ((t & 1) == 0 && t + 1 < g.T) ++t;
      else if (half == 0 && npx > 16) { half = 1; t &= ~1; }
      else { half = 0; ++t; }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  __device__ __forceinline__ void start(const PwGeom &g) {   // the first steps of a tile
    t = half = 0;
    if (!on) return;
    __syncwarp();
#pragma unroll 1
    for (int i = 0; i < kResAhead; ++i) fetch(g);
  }
  __device__ __forceinline__ void take(XT (&r)[16], const PwGeom &g, long long frame, int h, uint32_t mask) {
    if (on) {
      __syncwarp();   // everybody has read the slot that is filled now
      fetch(g);
      asm volatile("cp.async.wait_group %0;" ::"n"(kResAhead) : "memory");
      __syncwarp();
      const uint32_t at = smem + (out++ % kResSlots << 10) + (threadIdx.x & 31) * 2;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        uint16_t bits;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(bits) : "r"(at + (uint32_t)(i * 64)) : "memory");
        r[i] = __builtin_bit_cast(XT, bits);
      }
    } else {
      int pitch = g.Cout;
      asm volatile("" : "+r"(pitch));
      const XT *from = res + o0 + frame + (long long)(h * 16) * pitch;
#pragma unroll
      for (int i = 0; i < 16; ++i, from += pitch) r[i] = *((mask >> i & 1u) ? from : res);
    }
  }
};

// 16 pixels (half HALF of the warp's 32) of one (TQ = 1) or two timesteps of this thread's channel: tensor memory -> LIF ->
// spikes. `out` points at the first pixel of the first timestep. Both timesteps' sums travel together.
template <bool MASK, int TQ, typename XT, typename ST>
__device__ __forceinline__ void pair16(uint32_t taddr, float bias, const LifParams &p, float *v, ST *out, long long frame_out, int cs,
                                       uint32_t mask) {
  uint32_t a0[16], a1[16];
  const XT none[16] = {};
  umma::tmem_ld_x16(taddr, a0);
  if (TQ == 2) umma::tmem_ld_x16(taddr + 128u, a1);
  umma::tmem_ld_wait();
  lif16<kLean, MASK, false, false, XT, ST>(a0, none, bias, p, v, out, cs, mask);
  if (TQ == 2) lif16<kLean, MASK, false, false, XT, ST>(a1, none, bias, p, v, out + frame_out, cs, mask);
}
// The same with a residual that is read directly, one timestep after the other, which keeps the registers free of spills. A
// masked pixel's residual is read from `any`, an element that exists.
template <bool MASK, typename XT, typename ST>
__device__ __forceinline__ void pair16_res(uint32_t taddr, int tq, float bias, const LifParams &p, float *v, ST *out, const XT *res,
                                           const XT *any, long long frame_out, int cs, uint32_t mask) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    if (q < tq) {
      uint32_t a[16];
      XT r[16];
      umma::tmem_ld_x16(taddr + (uint32_t)(q * 128), a);
#pragma unroll
      for (int i = 0; i < 16; ++i) r[i] = *(!MASK || (mask >> i & 1u) ? res + q * frame_out + (long long)i * cs : any);
      umma::tmem_ld_wait();
      lif16<kLean, MASK, true, false, XT, ST>(a, r, bias, p, v, out + q * frame_out, cs, mask);
    }
  }
}
// The general form: any kind, with or without residuals, one timestep after the other. `frame`: offset of the pair's first
// timestep.
template <int KIND, bool MASK, bool RES, typename XT, typename ST>
__device__ __forceinline__ void pair_steps(uint32_t taddr, int tq, int npx, float bias, const PwGeom &g, const LifParams &p, float (&v)[32],
                                           ST *out, Residuals<XT> &res, long long frame, uint32_t mask) {
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    if (half * 16 < npx) {
#pragma unroll 1
      for (int q = 0; q < tq; ++q) {
        __syncwarp();   // predicated work of the step before; the load from tensor memory is the whole warp's
        uint32_t a[16], mk = mask >> (half * 16);
        int pitch = g.Cout;
        asm volatile("" : "+r"(mk), "+r"(pitch));   // what follows from them stays in the loop: 96 registers do not hold it
        XT r[16] = {};
        umma::tmem_ld_x16(taddr + (uint32_t)(q * 128 + half * 16), a);
        if (RES) res.take(r, g, frame + q * g.frame_out, half, mk);
        umma::tmem_ld_wait();
        lif16<KIND, MASK, RES, true, XT, ST>(a, r, bias, p, v + half * 16, out + q * g.frame_out + (long long)(half * 16) * pitch, pitch, mk);
      }
    }
  }
}

// The epilogue of a warp: all its tiles. Warp w reads lane quarter w % 4, pixels 32 (w / 4) .. + 31 (dup: quarters 2, 3 hold
// the channels of quarters 0, 1 again, and the eight warps of a channel group take 16 each).
template <int KIND, bool RES, bool DIRECT, typename XT, typename ST, typename VT>
__device__ __forceinline__ void epilogue(const PwGeom &g, const LifParams &p, const XT *__restrict__ bias, const XT *__restrict__ res,
                                         const VT *v_init, ST *__restrict__ spikes, VT *v_out, uint32_t tmem_base, uint32_t bar_base,
                                         uint32_t staging, volatile int *abort_flag) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, total = g.m_tiles * g.n_tiles_n;
  const long long wl = g.wait_limit;
  auto accfull = [&](uint32_t s) { return bar_base + 8u * (2 * kMaxStages + s); };
  auto accempty = [&](uint32_t s) { return bar_base + 8u * (2 * kMaxStages + 2 + s); };
  const int quarter = warp & 3;
  const int ch = (g.dup ? (quarter & 1) : quarter) * 32 + lane;
  const int px0 = g.dup ? ((warp >> 2) * 2 + (quarter >> 1)) * 16 : (warp >> 2) * 32;
  const int npx = g.dup ? 16 : 32;
  const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)px0;
  const int cs = g.Cout;
  Residuals<XT> rs;
  rs.res = res;
  rs.smem = staging + (uint32_t)(warp * kResWarp);
  rs.npx = npx;
  rs.on = g.res_staged != 0;
  rs.in = rs.out = 0;
  bool ok = true;
  uint32_t count = 0;
  for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
    const int m = tile / g.n_tiles_n, n0 = (tile % g.n_tiles_n) * 128;
    const long long m0 = first_pixel(g, m);
    const int c = n0 + ch;
    // which of this thread's pixels are written: those of the map; with the membrane in place the pixels that a shifted
    // tile shares with its neighbour belong to the neighbour (one thread reads and writes each value)
    uint32_t mask = 0;
    if (c < g.Cout) {
      const int hi = (int)max(0ll, min((long long)npx, g.P - m0 - px0));
      const int lo = g.own ? (int)max(0ll, min((long long)npx, (long long)m * 128 - m0 - px0)) : 0;
      if (hi > lo) mask = (hi - lo == 32 ? 0xffffffffu : ((1u << (hi - lo)) - 1u)) << lo;
    }
    const bool all = __all_sync(0xffffffffu, mask == (npx == 32 ? 0xffffffffu : 0xffffu));
    const bool none = __all_sync(0xffffffffu, mask == 0u);
    const float bias_c = (bias != nullptr && c < g.Cout) ? DT<XT>::to_f(bias[c]) : 0.f;
    const long long o0 = (m0 + px0) * cs + c;
    if (RES && !DIRECT && !none) {
      rs.o0 = o0;
      rs.nch = g.Cout - (c - lane);
      rs.exist = (int)max(0ll, min((long long)npx, g.P - m0 - px0));
      rs.start(g);
    }
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = 0.f;
    if (g.lif && v_init != nullptr) {
      const VT *from = v_init + o0;
      int pitch = cs;
      asm volatile("" : "+r"(pitch));   // the 32 offsets are not kept for the stores at the end
#pragma unroll
      for (int i = 0; i < 32; ++i, from += pitch)
        if (mask >> i & 1u) v[i] = DT<VT>::to_f(*from);
    }
    for (int pair = 0; pair < g.npairs && ok; ++pair, ++count) {
      const uint32_t acc = count & 1u, use = count >> 1;
      if (lane == 0) ok = umma::mbar_wait(accfull(acc), use & 1u, abort_flag, wl);
      ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
      if (!ok) break;
      umma::tc_fence_after_sync();
      const int tq = min(2, g.T - 2 * pair);
      const uint32_t taddr = lane_base + acc * 256u;
      const long long op = (2 * pair) * g.frame_out + o0;
      if (none) {
        // a warp without a channel or pixel of its own
      } else if constexpr (KIND == kLean && (!RES || DIRECT)) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          if (half * 16 < npx) {
            const uint32_t ta = taddr + (uint32_t)(half * 16), mk = mask >> (half * 16);
            const long long o = op + (long long)(half * 16) * cs;
            float *vh = v + half * 16;
            if constexpr (RES) {
              if (all) pair16_res<false, XT, ST>(ta, tq, bias_c, p, vh, spikes + o, res + o, res, g.frame_out, cs, mk);
              else pair16_res<true, XT, ST>(ta, tq, bias_c, p, vh, spikes + o, res + o, res, g.frame_out, cs, mk);
            } else if (tq == 2) {
              if (all) pair16<false, 2, XT, ST>(ta, bias_c, p, vh, spikes + o, g.frame_out, cs, mk);
              else pair16<true, 2, XT, ST>(ta, bias_c, p, vh, spikes + o, g.frame_out, cs, mk);
            } else {
              if (all) pair16<false, 1, XT, ST>(ta, bias_c, p, vh, spikes + o, g.frame_out, cs, mk);
              else pair16<true, 1, XT, ST>(ta, bias_c, p, vh, spikes + o, g.frame_out, cs, mk);
            }
          }
        }
      } else {
        ST *const out = spikes + op;
        const long long frame = (2 * pair) * g.frame_out;
        if (KIND == kLean && all) pair_steps<KIND, false, RES, XT, ST>(taddr, tq, npx, bias_c, g, p, v, out, rs, frame, mask);
        else pair_steps<KIND, true, RES, XT, ST>(taddr, tq, npx, bias_c, g, p, v, out, rs, frame, mask);
      }
      umma::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) umma::mbar_arrive(accempty(acc));
    }
    if (ok && g.lif && v_out != nullptr) {
      VT *to = v_out + o0;
      int pitch = cs;
      asm volatile("" : "+r"(pitch));
#pragma unroll
      for (int i = 0; i < 32; ++i, to += pitch)
        if (mask >> i & 1u) *to = DT<VT>::from_f(v[i]);
    }
  }
  if (RES && !DIRECT) asm volatile("cp.async.wait_all;" ::: "memory");   // what a wait that gave up left behind
}

// FORM: the common LIF without a residual, or with one that is read directly, each alone in its kernel; or everything else.
// In one kernel they do not fit 96 registers.
enum Form { kPlain, kDirect, kGeneral };
template <int FORM, typename XT, typename ST, typename VT>
__global__ void __launch_bounds__(kThreads, 1)
conv_pw_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const XT *__restrict__ bias,
               const XT *__restrict__ res, const VT *v_init, ST *__restrict__ spikes, VT *v_out, const PwGeom g, const LifParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * kMaxStages + 5];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  umma::pdl_trigger();

  // [resident weights: kslabs tiles] [ring of stages: pixels of two timesteps (+ the weight tile, when not resident)]
  const uint32_t w_base = (umma::smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t ring = w_base + (g.resident ? (uint32_t)(g.kslabs * kTile) : 0u);
  const uint32_t stage_bytes = (uint32_t)((g.resident ? 2 : 3) * kTile);
  const uint32_t bar_base = umma::smem_u32(bars);
  auto full = [&](uint32_t s) { return bar_base + 8u * s; };
  auto empty = [&](uint32_t s) { return bar_base + 8u * (kMaxStages + s); };
  auto accfull = [&](uint32_t s) { return bar_base + 8u * (2 * kMaxStages + s); };
  auto accempty = [&](uint32_t s) { return bar_base + 8u * (2 * kMaxStages + 2 + s); };
  const uint32_t wfull = bar_base + 8u * (2 * kMaxStages + 4);
  volatile int *abort_flag = &abort_s;
  const long long wl = g.wait_limit;

  if (threadIdx.x == 0) {
    abort_s = 0;
    for (int s = 0; s < g.stages; ++s) { umma::mbar_init(full(s), 1); umma::mbar_init(empty(s), 1); }
    for (int s = 0; s < 2; ++s) { umma::mbar_init(accfull(s), 1); umma::mbar_init(accempty(s), kEpi); }
    umma::mbar_init(wfull, 1);
    umma::fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    umma::tmem_alloc(umma::smem_u32(&tmem_base_s), 512u);
    umma::tmem_relinquish();
  }
  if (warp == kTmaWarp && lane == 0) {
    umma::prefetch_tensormap(&xmap);
    umma::prefetch_tensormap(&wmap);
  }
  umma::tc_fence_before_sync();
  __syncthreads();
  umma::tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  umma::pdl_wait();   // from here on: reads what the predecessor in the stream wrote, writes what it may read

  // Resident weights: this block keeps channel tile blockIdx % n_tiles_n and walks the pixel tiles. Otherwise the channel
  // tile is the fastest index, so that neighbouring blocks share their pixels in L2.
  const int total = g.m_tiles * g.n_tiles_n;

  if (warp == kTmaWarp) {
    if (lane == 0) {
      bool ok = true;
      uint32_t slot = 0, phase = 1;
      auto load_w = [&](uint32_t dst, uint32_t bar, int slab, int n0) {   // a box of 128 rows, or (dup) one of 64 twice
        umma::tma_load_2d(dst, &wmap, bar, slab * 64, n0);
        if (g.dup) umma::tma_load_2d(dst + (uint32_t)(kTile / 2), &wmap, bar, slab * 64, 0);
      };
      if (g.resident && (int)blockIdx.x < total) {
        umma::mbar_expect_tx(wfull, (uint32_t)(g.kslabs * kTile));
        for (int s = 0; s < g.kslabs; ++s) load_w(w_base + (uint32_t)(s * kTile), wfull, s, ((int)blockIdx.x % g.n_tiles_n) * 128);
      }
      for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
        const int m0 = (int)first_pixel(g, tile / g.n_tiles_n), n0 = (tile % g.n_tiles_n) * 128;
        for (int pair = 0; pair < g.npairs && ok; ++pair) {
          const int tq = min(2, g.T - 2 * pair);
          for (int s = 0; s < g.kslabs; ++s) {
            ok = umma::mbar_wait(empty(slot), phase, abort_flag, wl);
            if (!ok) break;
            umma::mbar_expect_tx(full(slot), (uint32_t)((tq + (g.resident ? 0 : 1)) * kTile));
            const uint32_t dst = ring + slot * stage_bytes;
            if (!g.resident) load_w(dst + 2u * kTile, full(slot), s, n0);
            if (!(g.drop_load && blockIdx.x == 0 && tile == 0 && pair == 0 && s == 0))
              for (int q = 0; q < tq; ++q) umma::tma_load_3d(dst + (uint32_t)(q * kTile), &xmap, full(slot), s * 64, m0, 2 * pair + q);
            if (++slot == (uint32_t)g.stages) { slot = 0; phase ^= 1u; }
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == kMmaWarp) {
    const uint32_t leader = umma::elect_one() ? 1u : 0u;
    const bool bf16 = std::is_same<XT, __nv_bfloat16>::value;
    const uint32_t id256 = umma::make_idesc_f16(128, 256, bf16), id128 = umma::make_idesc_f16(128, 128, bf16);
    const uint64_t rdesc = umma::make_sw128_kmajor_desc(ring), wdesc0 = umma::make_sw128_kmajor_desc(w_base);
    bool ok = true;
    uint32_t slot = 0, phase = 0, count = 0;   // count: pairs so far; they alternate between the accumulators across tiles too
    if (g.resident && (int)blockIdx.x < total) ok = umma::mbar_wait_warp(wfull, 0u, abort_flag, wl);
    for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
      for (int pair = 0; pair < g.npairs && ok; ++pair, ++count) {
        const uint32_t acc = count & 1u, use = count >> 1;
        ok = umma::mbar_wait_warp(accempty(acc), (use & 1u) ^ 1u, abort_flag, wl);   // its previous sums have been read
        if (!ok) break;
        umma::tc_fence_after_sync();
        const uint32_t d = tmem_base + acc * 256u, idesc = 2 * pair + 1 < g.T ? id256 : id128;
        for (int s = 0; s < g.kslabs; ++s) {
          ok = umma::mbar_wait_warp(full(slot), phase, abort_flag, wl);
          if (!ok) break;
          umma::tc_fence_after_sync();
          const uint64_t xdesc = rdesc + (uint64_t)((slot * stage_bytes) >> 4);
          const uint64_t wdesc = g.resident ? wdesc0 + (uint64_t)((uint32_t)(s * kTile) >> 4) : xdesc + (uint64_t)(2 * kTile >> 4);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma::mma_f16_ss_by(leader, d, wdesc + (uint64_t)(2 * k), xdesc + (uint64_t)(2 * k), idesc, (s > 0 || k > 0) ? 1u : 0u);
          umma::mma_commit_by(leader, empty(slot));
          if (++slot == (uint32_t)g.stages) { slot = 0; phase ^= 1u; }
        }
        if (ok) umma::mma_commit_by(leader, accfull(acc));
      }
    }
    __syncwarp();
  } else {
    const uint32_t staging = ring + (uint32_t)g.stages * stage_bytes;
    auto run = [&](auto kind, auto with_res) {
      epilogue<decltype(kind)::value, decltype(with_res)::value, FORM == kDirect, XT, ST, VT>(g, p, bias, res, v_init, spikes, v_out, tmem_base, bar_base, staging, abort_flag);
    };
    using std::integral_constant;
    // One branch around everything: inside the loop over the pairs the compiler computes for all kinds at once what only one
    // of them needs (500 bytes of spills).
    auto any_kind = [&](auto with_res) {
      switch (g.kind) {
        case kLean: run(integral_constant<int, kLean>{}, with_res); break;
        case 1: run(integral_constant<int, 1>{}, with_res); break;
        case 2: run(integral_constant<int, 2>{}, with_res); break;
        case 3: run(integral_constant<int, 3>{}, with_res); break;
        case 4: run(integral_constant<int, 4>{}, with_res); break;
        case 5: run(integral_constant<int, 5>{}, with_res); break;
        case 6: run(integral_constant<int, 6>{}, with_res); break;
        default: run(integral_constant<int, kOff>{}, with_res); break;
      }
    };
    if constexpr (FORM != kGeneral) run(integral_constant<int, kLean>{}, std::integral_constant<bool, FORM == kDirect>{});
    else if (res != nullptr) any_kind(std::true_type{});
    else any_kind(std::false_type{});
  }

  umma::tc_fence_before_sync();
  __syncthreads();
  if (abort_s && threadIdx.x == 0) atomicExch(&g_pw_status, 1);
  if (warp == kMmaWarp) {
    umma::tc_fence_after_sync();
    umma::tmem_dealloc(tmem_base, 512u);
  }
}

// Whether residuals pass through shared memory (Residuals above).
bool copies_residuals(const ConvArgs &a) {
  return a.res != nullptr && a.Cout % 32 != 0 && a.Cout % 8 == 0 && aligned16(a.res) && a.Cin <= kResidentSlabs * 64;
}

int lif_kind(const ConvArgs &a) {
  return !a.lif ? kOff : (a.p.mode == 1 && a.p.hard && a.p.v_reset == 0.f ? kLean : 1 + 2 * a.p.mode + (a.p.hard ? 1 : 0));
}

template <int FORM, typename XT, typename ST, typename VT>
int launch_form(const ConvArgs &a, cudaStream_t stream) {
  PwGeom g;
  g.T = a.T;
  g.npairs = (a.T + 1) / 2;
  g.kslabs = (a.Cin + 63) / 64;
  g.Cout = a.Cout;
  g.P = (long long)a.B * a.H * a.W;
  g.frame_out = g.P * a.Cout;
  g.n_tiles_n = (a.Cout + 127) / 128;
  g.m_tiles = (int)((g.P + 127) / 128);
  g.lif = a.lif;
  g.kind = lif_kind(a);
  g.dup = a.Cout <= 64 ? 1 : 0;
  g.own = (a.lif && a.v_init != nullptr && a.v_init == a.v_out) ? 1 : 0;
  g.wait_limit = 4000000000ll;
  g.drop_load = 0;
  consume_wait_selftest(&g.wait_limit, &g.drop_load);
  const int sms = sm_count();
  if (sms < 1) return fail(SNNB_ERR_CUDA, "conv_lif: cannot query the SM count");
  const long long total = (long long)g.m_tiles * g.n_tiles_n;
  if (total > 0x7fffffffLL) return fail(SNNB_ERR_INVALID, "conv_lif: problem too large for the grid");
  g.res_staged = copies_residuals(a) ? 1 : 0;
  const int data = kSmemData - (g.res_staged ? kEpi * kResWarp : 0);
  // three stages have to be left beside resident weights (with copied residuals: K <= 256)
  g.resident = g.kslabs <= kResidentSlabs && data - g.kslabs * kTile >= 3 * 2 * kTile && g.n_tiles_n <= sms ? 1 : 0;
  long long grid = total < sms ? total : sms;
  if (g.resident && grid > g.n_tiles_n) grid -= grid % g.n_tiles_n;   // every block keeps its channel tile
  const int fixed = g.resident ? g.kslabs * kTile : 0, stage = (g.resident ? 2 : 3) * kTile;
  g.stages = (data - fixed) / stage;
  if (g.stages > kMaxStages) g.stages = kMaxStages;
  const int smem = fixed + g.stages * stage + (g.res_staged ? kEpi * kResWarp : 0) + 1024;
  const int es = 2;
  CUtensorMap xm, wm;
  {
    cuuint64_t dims[3] = {(cuuint64_t)a.Cin, (cuuint64_t)g.P, (cuuint64_t)a.T};
    cuuint64_t strides[2] = {(cuuint64_t)a.Cin * es, a.T > 1 ? (cuuint64_t)a.x_t_stride * es : (cuuint64_t)g.P * a.Cin * es};
    cuuint32_t box[3] = {64, 128, 1};
    const int rc = encode_tmap(&xm, a.dtype, 3, a.x, dims, strides, box);
    if (rc != SNNB_OK) return rc;
  }
  {
    cuuint64_t dims[2] = {(cuuint64_t)a.Cin, (cuuint64_t)a.Cout};
    cuuint64_t strides[1] = {(cuuint64_t)a.Cin * es};
    cuuint32_t box[2] = {64, (cuuint32_t)(g.dup ? 64 : 128)};
    const int rc = encode_tmap(&wm, a.dtype, 2, a.w, dims, strides, box);
    if (rc != SNNB_OK) return rc;
  }
  const cudaError_t e = raise_smem_limit_once<conv_pw_kernel<FORM, XT, ST, VT>>(kSmemData + 1024);
  if (e != cudaSuccess) return fail(SNNB_ERR_CUDA, "conv_lif: cannot raise the shared-memory limit: %s", cudaGetErrorString(e));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t le = cudaLaunchKernelEx(&cfg, conv_pw_kernel<FORM, XT, ST, VT>, xm, wm, static_cast<const XT *>(a.b),
                                            static_cast<const XT *>(a.res), static_cast<const VT *>(a.v_init),
                                            static_cast<ST *>(a.spikes), static_cast<VT *>(a.v_out), g, a.p);
  if (le != cudaSuccess) return fail(SNNB_ERR_CUDA, "conv_pw: launch failed: %s", cudaGetErrorString(le));
  return SNNB_OK;
}

template <typename XT, typename ST, typename VT>
int launch(const ConvArgs &a, cudaStream_t stream) {
  if (lif_kind(a) != kLean || copies_residuals(a)) return launch_form<kGeneral, XT, ST, VT>(a, stream);
  return a.res == nullptr ? launch_form<kPlain, XT, ST, VT>(a, stream) : launch_form<kDirect, XT, ST, VT>(a, stream);
}

template <typename XT>
int dispatch(const ConvArgs &a, cudaStream_t stream) {
  const bool s_u8 = a.lif && a.spike_dtype == SNNB_U8, v_f32 = a.lif && a.v_dtype == SNNB_F32;
  if (s_u8) return v_f32 ? launch<XT, uint8_t, float>(a, stream) : launch<XT, uint8_t, XT>(a, stream);
  return v_f32 ? launch<XT, XT, float>(a, stream) : launch<XT, XT, XT>(a, stream);
}

}  // namespace

bool conv_pw_supported(const ConvArgs &a) {
  if (a.dtype != SNNB_BF16 && a.dtype != SNNB_F16) return false;
  if (a.KH != 1 || a.KW != 1 || a.stride != 1 || a.pad != 0 || a.sc_x != nullptr) return false;
  if (a.Cin % 8 != 0 || a.x_t_stride % 8 != 0 || (a.x_t_stride == 0 && a.T > 1)) return false;
  if (a.xs_w || a.xs_h || a.xs_b || a.xd_w || a.xd_h) return false;
  return aligned16(a.x) && aligned16(a.w);
}

// Calls that the general kernel of conv_tc.cu, which takes all timesteps of a tile at once and stores 32 bytes of a pixel at
// a time, does better (measured on B200 over drawn calls, geometric means): at most 16 channels out use 16 of the 128 rows
// here and a warp's stores fill half a sector pair (Cin 64: its time 0.82 of this kernel's, Cin 128: 0.95, Cin 192: 1.1);
// with one slab and T >= 9 a tile that has an SM to itself is a chain of five or more epilogues (0.68 with at most a quarter
// as many tiles as SMs, 1.4 with more; T 7, 8: 0.95; T 5, 6: 1.05).
bool conv_tc_beats_pw(const ConvArgs &a) {
  const int sms = sm_count() > 0 ? sm_count() : 148;
  const long long tiles = ((long long)a.B * a.H * a.W + 127) / 128 * ((a.Cout + 127) / 128);
  return (tiles <= sms && a.Cout <= 16 && a.Cin <= 128) || (tiles <= sms / 4 && a.Cin <= 64 && a.T >= 9);
}

int conv_pw(const ConvArgs &a, cudaStream_t stream) {
  return a.dtype == SNNB_BF16 ? dispatch<__nv_bfloat16>(a, stream) : dispatch<__half>(a, stream);
}

int pw_device_status(int *out) {
  int h = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&h, g_pw_status, sizeof(int));
  if (e != cudaSuccess) return fail(SNNB_ERR_CUDA, "device_status: %s", cudaGetErrorString(e));
  if (h != 0) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_pw_status, &zero, sizeof(int));
  }
  *out = h;
  return SNNB_OK;
}

}  // namespace snnb
