// fp32 dense conv / linear (+ bias, + residual) + LIF over T on the CUDA cores: an implicit GEMM whose rows are
// (pixel, timestep) pairs, fed by asynchronous copies, on the packed fp32 multiply-add.
//
// Bound: the FMA pipe (128 fp32 FMA per SM and cycle = 74 TFLOP/s on 148 SMs at 1.965 GHz); TF32 cannot hold the 1e-4
// membrane bound, so fp32 stays off the tensor cores. What the layout is chosen for:
//
//  * Rows = pixels x TT timesteps. A thread's eight rows are TT consecutive steps of 8 / TT pixels, so the LIF of a
//    pixel runs inside one thread straight from the accumulators, the weights staged for a tile serve all TT steps, and
//    a layer has T times as many tiles' worth of rows to spread over the SMs (16 x 16 maps, batch 16, 128 channels:
//    256 blocks). Longer sequences walk windows of TT steps with the membrane in shared memory (pick_tile). One frame
//    for all steps (direct encoding) is convolved once (TT = 1) and its LIF repeated.
//  * Both operands keep K contiguous in shared memory (what 16-byte cp.async delivers, with zero fill for padding, the
//    last K chunk and rows past the end), rows 20 words apart: the 16-byte fragment reads of eight neighbouring rows
//    touch all 32 banks once.
//  * The packed multiply-add (two fp32 FMA per instruction) works on neighbouring K values: an accumulator is a pair
//    (sum over even K, sum over odd K), which needs no broadcast moves, and the two chains of half the length round
//    less than one.
//
// Measured on B200 against the kernel of conv_simt.cu (4 x 4 outputs per thread, element-wise loads, one timestep at a
// time), which these calls ran before: 3x3 128 -> 128 on 16 x 16 maps, batch 16, T = 4, with its 1x1 shortcut conv 621 ->
// 152 us; 64 -> 64, batch 25, T = 8 601 -> 116 us; 256 -> 512 on one 28 x 28 map, T = 8 2292 -> 386 us (38 TFLOP/s); linear
// 22 x 1024 -> 4096, T = 4 493 -> 59 us. What is left: the packed FMA pipe is busy half of the time, its warps wait for
// their own fixed latencies (two warps per scheduler at 255 registers; four at 128 registers gain nothing, because the
// smaller tile reads more shared memory per multiply-add).
//
// Calls with Cin % 4 != 0 or operands off the 16-byte grid stay on the kernel of conv_simt.cu, and so do those that are mostly
// stores (conv_f32_pays).
#include "conv.cuh"

namespace snnb {
namespace {

constexpr int kBM = 128, kBK = 16, kPitch = 20, kThreads = 128, kStages = 4;

struct F32Geom {
  int T, nwin, Cin, H, W, Cout, KH, KW, stride, pad, Ho, Wo, K, lif, alias, vec;
  long long x_t_stride, M, frame_out;
};

__device__ __forceinline__ void cp16(uint32_t dst, const float *src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

template <int TT, int TN, typename ST>
__global__ void __launch_bounds__(kThreads, TN == 4 && TT >= 4 ? 4 : 2)
conv_lif_f32_kernel(const float *__restrict__ x, const float *__restrict__ w, const float *__restrict__ bias,
                    const float *__restrict__ res, const float *v_init, ST *__restrict__ spikes, float *v_out,
                    const F32Geom g, const LifParams p) {
  constexpr int NP = 8 / TT;             // pixels per thread
  constexpr int BN = 8 * TN;             // channels per block
  constexpr int PIX = 16 * NP;           // pixels per block
  constexpr int kStage = (kBM + BN) * kPitch * 4;   // bytes
  extern __shared__ __align__(16) float smem[];
  float *vs = smem + kStages * kStage / 4 + threadIdx.x;   // [NP * TN][kThreads]: membranes between windows

  const int tid = threadIdx.x;
  const int ty = ((tid >> 5) << 2 & 8) | (tid & 7), tx = ((tid >> 5 & 1) << 2) | (tid >> 3 & 3);   // a warp is 8 x 4
  const long long m0 = (long long)blockIdx.x * PIX;
  const int n0 = blockIdx.y * BN;

  // ---- loaders: this thread copies 16-byte piece `piece` of rows lrow + 32 i (activations) / channels lrow + 32 i
  // A row is described by its first tap's offset from the tile's first image and by (hi0, wi0); the tap offset is
  // common to all rows and added per chunk.
  const int piece = tid & 3, lrow = tid >> 2;
  const long long hw = (long long)g.Ho * g.Wo;
  const long long img0 = m0 / hw;
  const float *ximg = x + img0 * g.H * (long long)g.W * g.Cin;
  int xoff[4], hw0[4];   // hw0: hi0 in the upper, wi0 in the lower 16 bits
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = lrow + 32 * i;
    const long long m = m0 + (row >> 4) / TT * 16 + (row & 15);
    hw0[i] = (int)0x80000000;   // rows past the end: every tap lies above the image
    xoff[i] = 0;
    if (m < g.M) {
      const int q = (int)(m - img0 * hw);
      const int im = q / (int)hw, r = q - im * (int)hw;
      const int ho = r / g.Wo, wo = r - ho * g.Wo;
      const int hi0 = ho * g.stride - g.pad, wi0 = wo * g.stride - g.pad;
      hw0[i] = (int)((uint32_t)hi0 << 16 | ((uint32_t)wi0 & 0xFFFFu));
      xoff[i] = ((im * g.H + hi0) * g.W + wi0) * g.Cin;
    }
  }
  constexpr int WROWS = BN / 32;   // weight rows per thread and chunk
  const float *wrow[WROWS];
  uint32_t wdst[WROWS];
  bool wok[WROWS];
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
#pragma unroll
  for (int i = 0; i < WROWS; ++i) {
    const int c = lrow + 32 * i;   // channel c of the tile lies in row (c % TN) * 8 + c / TN: a thread's TN channels
                                   // are neighbours in memory, its fragment reads 8 rows apart
    wok[i] = n0 + c < g.Cout;
    wrow[i] = w + (long long)(wok[i] ? n0 + c : 0) * g.K + piece * 4;
    wdst[i] = sbase + (uint32_t)((kBM + (c % TN) * 8 + c / TN) * kPitch + piece * 4) * 4u;
  }
  const uint32_t adst = sbase + (uint32_t)(lrow * kPitch + piece * 4) * 4u;
  const int nchunks = (g.K + kBK - 1) / kBK;

  float bj[TN];
#pragma unroll
  for (int j = 0; j < TN; ++j) {
    const int n = n0 + tx * TN + j;
    bj[j] = (bias != nullptr && n < g.Cout) ? bias[n] : 0.f;
  }

  for (int win = 0; win < g.nwin; ++win) {
    // position of this thread's piece in K: tap (kh, kw) and channel
    int ci = piece * 4, kh = 0, kw = 0, kpos = piece * 4;
    while (ci >= g.Cin) { ci -= g.Cin; if (++kw == g.KW) { kw = 0; ++kh; } }
    auto load = [&](int chunk) {
      const uint32_t st = (uint32_t)((chunk % kStages) * kStage);
      const bool kok = kpos < g.K;
      const int tap = (kh * g.W + kw) * g.Cin + ci;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int hi = (hw0[i] >> 16) + kh, wi = (int)(int16_t)hw0[i] + kw;
        const bool ok = kok && (unsigned)hi < (unsigned)g.H && (unsigned)wi < (unsigned)g.W;
        // a step past the end reads the last one; its rows are not evaluated
        const int t = TT == 1 ? win : min(win * TT + ((lrow >> 4) + 2 * i) % TT, g.T - 1);
        cp16(adst + st + (uint32_t)(32 * i * kPitch * 4), ok ? ximg + (long long)t * g.x_t_stride + (xoff[i] + tap) : x, ok);
      }
#pragma unroll
      for (int i = 0; i < WROWS; ++i) cp16(wdst[i] + st, wok[i] && kok ? wrow[i] + (long long)chunk * kBK : w, wok[i] && kok);
      ci += kBK;
      kpos += kBK;
      while (ci >= g.Cin) { ci -= g.Cin; if (++kw == g.KW) { kw = 0; ++kh; } }
    };

    float2 acc[8][TN];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) {
      if (s < nchunks) load(s);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int chunk = 0; chunk < nchunks; ++chunk) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
      __syncthreads();   // chunk has arrived for everybody; everybody is done with the stage the next load overwrites
      if (chunk + kStages - 1 < nchunks) load(chunk + kStages - 1);
      asm volatile("cp.async.commit_group;" ::: "memory");
      const float *as = smem + (chunk % kStages) * (kStage / 4) + ty * kPitch;
      const float *bs = smem + (chunk % kStages) * (kStage / 4) + (kBM + tx) * kPitch;
#pragma unroll
      for (int kk = 0; kk < kBK; kk += 4) {
        float4 a[8], b[TN];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const float4 *>(as + i * 16 * kPitch + kk);
#pragma unroll
        for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4 *>(bs + j * 8 * kPitch + kk);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) acc[i][j] = __ffma2_rn(make_float2(a[i].x, a[i].y), make_float2(b[j].x, b[j].y), acc[i][j]);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) acc[i][j] = __ffma2_rn(make_float2(a[i].z, a[i].w), make_float2(b[j].z, b[j].w), acc[i][j]);
      }
    }
    __syncthreads();   // the next window's first loads overwrite stages that may still be read

    // ---- epilogue: row i of the thread is step i % TT of pixel i / TT
    const int nb = n0 + tx * TN;
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      const long long m = m0 + q * 16 + ty;
      if (m >= g.M) continue;
      const long long o = m * g.Cout + nb;
      float v[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        if (win > 0) v[j] = vs[(q * TN + j) * kThreads];
        else v[j] = (g.lif && v_init != nullptr && nb + j < g.Cout) ? v_init[o + j] : 0.f;
      }
      for (int rep = 0; rep < (g.alias ? g.T : 1); ++rep) {   // direct encoding: the one conv serves every step
#pragma unroll
        for (int t = 0; t < TT; ++t) {
          const int step = g.alias ? rep : win * TT + t;
          if (step >= g.T) break;
          const long long os = (long long)step * g.frame_out + o;
          float y[TN];
#pragma unroll
          for (int j = 0; j < TN; ++j) y[j] = (acc[q * TT + t][j].x + acc[q * TT + t][j].y) + bj[j];
#pragma unroll
          for (int j0 = 0; j0 < TN; j0 += 4) {
            if (g.vec && nb + j0 + 3 < g.Cout) {
              if (res != nullptr) {
                float r[4];
                load_pack<float, 4>(res + os + j0, r);
#pragma unroll
                for (int j = 0; j < 4; ++j) y[j0 + j] += r[j];
              }
              float s[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) s[j] = g.lif ? lif_step(y[j0 + j], v[j0 + j], p) : y[j0 + j];
              if (g.lif) store_pack<ST, 4, false>(spikes + os + j0, s);
              else store_pack<float, 4, false>(reinterpret_cast<float *>(spikes) + os + j0, s);
            } else {
#pragma unroll
              for (int j = j0; j < j0 + 4; ++j) {
                if (nb + j >= g.Cout) continue;
                float yy = y[j];
                if (res != nullptr) yy += res[os + j];
                if (g.lif) spikes[os + j] = DT<ST>::from_f(lif_step(yy, v[j], p));
                else reinterpret_cast<float *>(spikes)[os + j] = yy;
              }
            }
          }
        }
      }
      if (win + 1 < g.nwin) {
#pragma unroll
        for (int j = 0; j < TN; ++j) vs[(q * TN + j) * kThreads] = v[j];
      } else if (g.lif && v_out != nullptr) {
#pragma unroll
        for (int j0 = 0; j0 < TN; j0 += 4) {
          if (g.vec && nb + j0 + 3 < g.Cout && (reinterpret_cast<uintptr_t>(v_out) & 15u) == 0) {
            *reinterpret_cast<float4 *>(v_out + o + j0) = make_float4(v[j0], v[j0 + 1], v[j0 + 2], v[j0 + 3]);
          } else {
#pragma unroll
            for (int j = j0; j < j0 + 4; ++j)
              if (nb + j < g.Cout) v_out[o + j] = v[j];
          }
        }
      }
    }
  }
}

template <int TT, int TN, typename ST>
int launch_f32(const ConvArgs &a, const F32Geom &g, cudaStream_t stream) {
  constexpr int PIX = 16 * (8 / TT), BN = 8 * TN;
  const long long gx = (g.M + PIX - 1) / PIX;
  const int gy = (g.Cout + BN - 1) / BN;
  if (gx > 0x7fffffffLL || gy > 65535) return fail(SNNB_ERR_INVALID, "conv_lif: problem too large for the grid");
  const int smem = kStages * (kBM + BN) * kPitch * 4 + (g.nwin > 1 ? (8 / TT) * TN * kThreads * 4 : 0);
  constexpr int smem_max = kStages * (kBM + BN) * kPitch * 4 + (8 / TT) * TN * kThreads * 4;
  const cudaError_t e = raise_smem_limit_once<conv_lif_f32_kernel<TT, TN, ST>>(smem_max);
  if (e != cudaSuccess) return fail(SNNB_ERR_CUDA, "conv_lif: cannot raise the shared-memory limit: %s", cudaGetErrorString(e));
  conv_lif_f32_kernel<TT, TN, ST><<<dim3((unsigned)gx, (unsigned)gy), kThreads, smem, stream>>>(
      static_cast<const float *>(a.x), static_cast<const float *>(a.w), static_cast<const float *>(a.b),
      static_cast<const float *>(a.res), static_cast<const float *>(a.v_init), static_cast<ST *>(a.spikes),
      static_cast<float *>(a.v_out), g, a.p);
  SNNB_CHECK_LAUNCH("conv_lif_f32");
  return SNNB_OK;
}

// Which tile: TT steps per window and 64 or 32 channels per block, by the time that the fullest SM needs per K chunk
// (measured in microseconds, the same for all shapes to within 10 %: a block of 64 channels 1.15 alone on its SM and
// 1.0 each beside others; a block of 32 channels 0.85 and 0.6), times the windows that a block walks. 16 x 16 maps,
// batch 16, 128 -> 128 channels, T = 4: predicted 2.0 / 2.4 / 2.3 / 4.0 for (steps, channels) = (4, 64) / (4, 32) /
// (2, 64) / (8, 64), measured 152 / 182 / 188 / 276 us. Odd T is rounded up to whole windows by the same estimate:
// T = 3, 28 x 28, 512 -> 1024 takes 756 us with a window of four, 932 us with three windows of one.
F32Tile pick_tile(const F32Geom &g) {
  const int sms = sm_count() > 0 ? sm_count() : 148;
  F32Tile best = {1, 8};
  double best_cost = 1e300;
  for (int TT = g.alias ? 1 : 8; TT >= 1; TT /= 2)
    for (int TN = 8; TN >= 4; TN -= 4) {
      const int pix = 16 * (8 / TT);
      const long long blocks = ((g.M + pix - 1) / pix) * ((g.Cout + 8 * TN - 1) / (8 * TN));
      const double per_sm = (double)((blocks + sms - 1) / sms);
      const int nwin = g.alias ? 1 : (g.T + TT - 1) / TT;
      const double cost = nwin * (per_sm > 1 ? per_sm * (TN == 8 ? 1.0 : 0.6) : (TN == 8 ? 1.15 : 0.85));
      if (cost < best_cost) {
        best_cost = cost;
        best = {TT, TN};
      }
    }
  return best;
}

template <int TT, typename ST>
int launch_tn(const ConvArgs &a, F32Geom &g, int TN, cudaStream_t stream) {
  g.nwin = g.alias ? 1 : (g.T + TT - 1) / TT;
  return TN == 8 ? launch_f32<TT, 8, ST>(a, g, stream) : launch_f32<TT, 4, ST>(a, g, stream);
}

template <typename ST>
int launch_tt(const ConvArgs &a, F32Geom &g, cudaStream_t stream) {
  const F32Tile t = pick_tile(g);
  switch (t.TT) {
    case 8: return launch_tn<8, ST>(a, g, t.TN, stream);
    case 4: return launch_tn<4, ST>(a, g, t.TN, stream);
    case 2: return launch_tn<2, ST>(a, g, t.TN, stream);
    default: return launch_tn<1, ST>(a, g, t.TN, stream);
  }
}

}  // namespace

bool conv_f32_supported(const ConvArgs &a) {
  return a.dtype == SNNB_F32 && a.Cin % 4 == 0 && a.x_t_stride % 4 == 0 && aligned16(a.x) && aligned16(a.w) &&
         a.pad < a.KH && a.pad < a.KW && a.KH <= 128 && a.KW <= 128 && a.H < 16384 && a.W < 16384 && a.stride * (long long)a.Ho < 32768 && a.stride * (long long)a.Wo < 32768 &&
         (128 / ((long long)a.Ho * a.Wo) + 2) * a.H * a.W * a.Cin < (1LL << 31) && !a.xs_w && !a.xs_h && !a.xs_b && !a.xd_w && !a.xd_h && a.sc_x == nullptr;
}

// Where the kernel of conv_simt.cu is the faster one: with a short K a call is its stores, which that kernel's small blocks
// (64 pixels, eight to an SM) keep going while these have two to four blocks of 128 rows. Measured on B200, its time against
// this one's: 8 -> 336 channels, 36504 pixels, T = 5 209 and 346 us; 8 -> 1106, 1452 tokens, T = 2 18 and 34 us; 16 -> 192, 4116
// pixels, T = 6 29 and 35 us; with few channels out or K = 28 .. 64 about as often one as the other (16 -> 4, 87025 pixels
// 88 and 49 us; 32 -> 328, 2009 pixels 49 and 41 us). One frame for all steps, where T frames are stored per convolution:
// K = 16, 126 channels, 6720 pixels, T = 4 17 and 35 us; K = 80, 312 channels, 8325 pixels, T = 6 66 and 107 us; K = 64,
// 48 channels, 8112 pixels, T = 4 21 and 18 us; 24 -> 37, 14 pixels, T = 12 36 and 9 us.
bool conv_f32_pays(const ConvArgs &a) {
  const long long K = (long long)a.KH * a.KW * a.Cin;
  const long long pixels = (long long)a.B * a.Ho * a.Wo;
  if (a.x_t_stride == 0 && a.T > 1) return K > 16 * a.T || pixels < 128;
  const long long blocks = (pixels + 63) / 64 * ((a.Cout + 63) / 64);   // of conv_simt.cu
  return !(K <= 24 && a.Cout > 96 && blocks >= (sm_count() > 0 ? sm_count() : 148));
}

namespace {
F32Geom make_geom(const ConvArgs &a) {
  F32Geom g;
  g.T = a.T; g.nwin = 1; g.Cin = a.Cin; g.H = a.H; g.W = a.W; g.Cout = a.Cout; g.KH = a.KH; g.KW = a.KW;
  g.stride = a.stride; g.pad = a.pad; g.Ho = a.Ho; g.Wo = a.Wo; g.K = a.KH * a.KW * a.Cin; g.lif = a.lif;
  g.alias = (a.x_t_stride == 0 && a.T > 1) ? 1 : 0;
  g.x_t_stride = a.x_t_stride;
  g.M = (long long)a.B * a.Ho * a.Wo;
  g.frame_out = g.M * a.Cout;
  g.vec = a.Cout % 4 == 0 && aligned16(a.spikes) && (a.res == nullptr || aligned16(a.res));
  return g;
}
}  // namespace

F32Tile conv_f32_tile(const ConvArgs &a) { return pick_tile(make_geom(a)); }

int conv_f32(const ConvArgs &a, cudaStream_t stream) {
  F32Geom g = make_geom(a);
  if (a.lif && a.spike_dtype == SNNB_U8) return launch_tt<uint8_t>(a, g, stream);
  return launch_tt<float>(a, g, stream);
}

}  // namespace snnb
