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

struct PwGeom {
  int T, npairs, kslabs, Cout, n_tiles_n, m_tiles, stages, resident, lif, own;
  int dup;                  // Cout <= 64: the weight rows twice (M rows 64..127 repeat 0..63), so that all epilogue warps have work
  long long P, frame_out;   // pixels of a frame; elements of an output frame
  long long wait_limit;     // bound of every mbarrier wait, in SM cycles
  int drop_load;            // self-test: block 0 announces its first stage but does not load its pixels
};

// The spikes of 16 pixels of one timestep, common case: tau a power of two, hard reset to zero.
// h = v + (y - v) * inv_tau: the product with a power of two is exact, so the fused multiply-add rounds the same sum as
// lif_step's separately rounded operations. MASK: only pixels whose bit is set are written. RES: r is added.
template <bool MASK, bool RES, typename XT, typename ST>
__device__ __forceinline__ void lif16(const uint32_t (&a)[16], const XT (&r)[16], float2 b2, float2 it2, float v_th, float *v,
                                      ST *out, int cs, uint32_t mask) {
  constexpr uint32_t one = std::is_same<ST, uint8_t>::value ? 1u : (std::is_same<ST, __half>::value ? 0x3C00u : 0x3F80u);
  using Bits = typename std::conditional<sizeof(ST) == 1, uint8_t, uint16_t>::type;
  Bits *to = reinterpret_cast<Bits *>(out);
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    float2 y = __fadd2_rn(make_float2(__uint_as_float(a[i]), __uint_as_float(a[i + 1])), b2);
    if (RES) y = __fadd2_rn(y, make_float2(DT<XT>::to_f(r[i]), DT<XT>::to_f(r[i + 1])));
    const float2 d = __fadd2_rn(y, make_float2(-v[i], -v[i + 1]));
    const float2 h = __ffma2_rn(d, it2, make_float2(v[i], v[i + 1]));
    const bool s0 = h.x >= v_th, s1 = h.y >= v_th;
    v[i] = s0 ? 0.f : h.x;
    v[i + 1] = s1 ? 0.f : h.y;
    if (!MASK || (mask >> i & 1u)) to[(long long)i * cs] = (Bits)(s0 ? one : 0u);
    if (!MASK || (mask >> (i + 1) & 1u)) to[(long long)(i + 1) * cs] = (Bits)(s1 ? one : 0u);
  }
}

// 16 pixels of one (TQ = 1) or two timesteps of this thread's channel: tensor memory -> LIF -> spikes. `out` / `res` point
// at the first pixel of the first timestep; a masked pixel's residual is read from `res_any`, an element that exists. Both
// timesteps' sums travel together; with a residual one after the other, which keeps the registers free of spills.
template <bool MASK, int TQ, typename XT, typename ST>
__device__ __forceinline__ void pair16(uint32_t taddr, float2 b2, float2 it2, float v_th, float *v, ST *out, long long frame_out,
                                       int cs, uint32_t mask) {
  uint32_t a0[16], a1[16];
  const XT none[16] = {};
  umma::tmem_ld_x16(taddr, a0);
  if (TQ == 2) umma::tmem_ld_x16(taddr + 128u, a1);
  umma::tmem_ld_wait();
  lif16<MASK, false, XT, ST>(a0, none, b2, it2, v_th, v, out, cs, mask);
  if (TQ == 2) lif16<MASK, false, XT, ST>(a1, none, b2, it2, v_th, v, out + frame_out, cs, mask);
}
template <bool MASK, typename XT, typename ST>
__device__ __forceinline__ void pair16_res(uint32_t taddr, int tq, float2 b2, float2 it2, float v_th, float *v, ST *out,
                                           const XT *res, const XT *res_any, long long frame_out, int cs, uint32_t mask) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    if (q < tq) {
      uint32_t a[16];
      XT r[16];
      umma::tmem_ld_x16(taddr + (uint32_t)(q * 128), a);
#pragma unroll
      for (int i = 0; i < 16; ++i) r[i] = *(!MASK || (mask >> i & 1u) ? res + q * frame_out + (long long)i * cs : res_any);
      umma::tmem_ld_wait();
      lif16<MASK, true, XT, ST>(a, r, b2, it2, v_th, v, out + q * frame_out, cs, mask);
    }
  }
}

template <typename XT, typename ST, typename VT>
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
  auto first_pixel = [&](int m) { return max(0ll, min((long long)m * 128, g.P - 128)); };

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
        const int m0 = (int)first_pixel(tile / g.n_tiles_n), n0 = (tile % g.n_tiles_n) * 128;
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
    // ------------------------------------------------ epilogue: warp w reads lane quarter w % 4, pixels 32 (w / 4) .. + 31
    // (dup: quarters 2, 3 hold the channels of quarters 0, 1 again, and the eight warps of a channel group take 16 each)
    const int quarter = warp & 3;
    const int ch = (g.dup ? (quarter & 1) : quarter) * 32 + lane;
    const int px0 = g.dup ? ((warp >> 2) * 2 + (quarter >> 1)) * 16 : (warp >> 2) * 32;
    const int npx = g.dup ? 16 : 32;
    const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)px0;
    const bool lean = g.lif && p.mode == 1 && p.hard && p.v_reset == 0.f;
    const float2 it2 = make_float2(p.inv_tau, p.inv_tau);
    const int cs = g.Cout;
    bool ok = true;
    uint32_t count = 0;
    for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
      const int m = tile / g.n_tiles_n, n0 = (tile % g.n_tiles_n) * 128;
      const long long m0 = first_pixel(m);
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
      const float2 b2 = make_float2(bias_c, bias_c);
      const long long o0 = (m0 + px0) * cs + c;
      float v[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = 0.f;
      if (g.lif && v_init != nullptr) {
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (mask >> i & 1u) v[i] = DT<VT>::to_f(v_init[o0 + (long long)i * cs]);
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
        } else if (lean) {
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            if (half * 16 < npx) {
              const uint32_t ta = taddr + (uint32_t)(half * 16), mk = mask >> (half * 16);
              const long long o = op + (long long)(half * 16) * cs;
              float *vh = v + half * 16;
              if (res != nullptr) {
                if (all) pair16_res<false, XT, ST>(ta, tq, b2, it2, p.v_th, vh, spikes + o, res + o, res, g.frame_out, cs, mk);
                else pair16_res<true, XT, ST>(ta, tq, b2, it2, p.v_th, vh, spikes + o, res + o, res, g.frame_out, cs, mk);
              } else if (tq == 2) {
                if (all) pair16<false, 2, XT, ST>(ta, b2, it2, p.v_th, vh, spikes + o, g.frame_out, cs, mk);
                else pair16<true, 2, XT, ST>(ta, b2, it2, p.v_th, vh, spikes + o, g.frame_out, cs, mk);
              } else {
                if (all) pair16<false, 1, XT, ST>(ta, b2, it2, p.v_th, vh, spikes + o, g.frame_out, cs, mk);
                else pair16<true, 1, XT, ST>(ta, b2, it2, p.v_th, vh, spikes + o, g.frame_out, cs, mk);
              }
            }
          }
        } else {   // other LIF kinds, or none
#pragma unroll
          for (int half = 0; half < 2; ++half)
            for (int q = 0; q < tq && half * 16 < npx; ++q) {
              uint32_t a[16];
              umma::tmem_ld_x16(taddr + (uint32_t)(q * 128 + half * 16), a);
              umma::tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                const int px = half * 16 + i;
                if (!(mask >> px & 1u)) continue;
                const long long o = op + q * g.frame_out + (long long)px * cs;
                float y = __uint_as_float(a[i]) + bias_c;
                if (res != nullptr) y += DT<XT>::to_f(res[o]);
                if (g.lif) spikes[o] = DT<ST>::from_f(lif_step(y, v[px], p));
                else reinterpret_cast<XT *>(spikes)[o] = DT<XT>::from_f(y);
              }
            }
        }
        umma::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) umma::mbar_arrive(accempty(acc));
      }
      if (ok && g.lif && v_out != nullptr) {
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (mask >> i & 1u) v_out[o0 + (long long)i * cs] = DT<VT>::from_f(v[i]);
      }
    }
  }

  umma::tc_fence_before_sync();
  __syncthreads();
  if (abort_s && threadIdx.x == 0) atomicExch(&g_pw_status, 1);
  if (warp == kMmaWarp) {
    umma::tc_fence_after_sync();
    umma::tmem_dealloc(tmem_base, 512u);
  }
}

template <typename XT, typename ST, typename VT>
int launch(const ConvArgs &a, cudaStream_t stream) {
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
  g.dup = a.Cout <= 64 ? 1 : 0;
  g.own = (a.lif && a.v_init != nullptr && a.v_init == a.v_out) ? 1 : 0;
  g.wait_limit = 4000000000ll;
  g.drop_load = 0;
  consume_wait_selftest(&g.wait_limit, &g.drop_load);
  const int sms = sm_count();
  if (sms < 1) return fail(SNNB_ERR_CUDA, "conv_lif: cannot query the SM count");
  const long long total = (long long)g.m_tiles * g.n_tiles_n;
  if (total > 0x7fffffffLL) return fail(SNNB_ERR_INVALID, "conv_lif: problem too large for the grid");
  g.resident = g.kslabs <= kResidentSlabs && g.n_tiles_n <= sms ? 1 : 0;
  long long grid = total < sms ? total : sms;
  if (g.resident && grid > g.n_tiles_n) grid -= grid % g.n_tiles_n;   // every block keeps its channel tile
  g.stages = (kSmemData - (g.resident ? g.kslabs * kTile : 0)) / ((g.resident ? 2 : 3) * kTile);
  if (g.stages > kMaxStages) g.stages = kMaxStages;
  const int smem = (g.resident ? g.kslabs * kTile : 0) + g.stages * (g.resident ? 2 : 3) * kTile + 1024;
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
  const cudaError_t e = raise_smem_limit_once<conv_pw_kernel<XT, ST, VT>>(kSmemData + 1024);
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
  const cudaError_t le = cudaLaunchKernelEx(&cfg, conv_pw_kernel<XT, ST, VT>, xm, wm, static_cast<const XT *>(a.b),
                                            static_cast<const XT *>(a.res), static_cast<const VT *>(a.v_init),
                                            static_cast<ST *>(a.spikes), static_cast<VT *>(a.v_out), g, a.p);
  if (le != cudaSuccess) return fail(SNNB_ERR_CUDA, "conv_pw: launch failed: %s", cudaGetErrorString(le));
  return SNNB_OK;
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
