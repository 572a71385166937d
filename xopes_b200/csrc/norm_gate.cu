// Fused normalisation + gate: the op that follows lightning attention in a model block
// (xopes/ops/normalize/normalize/normalize_torch.py:9-111, the gate branch):
//
//   a  = act(gate)                                   act in {none, relu, sigmoid, silu}
//   z  = x (.) a   (gate_pos = pre)   or   x         per group of e features (a head):
//   zc = z - mean(z)  (use_mean)      or   z
//   y  = c zc / sqrt(sum zc^2 + eps) (.) weight + bias
//   o  = y            (gate_pos = pre, or no gate)   or   y (.) a   (gate_pos = post)
//
// One pass over x and gate in, o out (forward), and one pass over x, gate, do in, dx, dgate out
// (backward), all arithmetic in fp32: pure HBM streaming, 3 x 2e bytes per group forward and
// 5 x 2e backward.  LPG lanes own one (row, group) at a time, so a warp works on 32 / LPG rows of ONE
// group; the weight / bias gradients accumulate in registers, meet in shared memory once at the
// end and leave with one atomicAdd per feature and CTA.
#include "common.cuh"

namespace la {
namespace {

constexpr int kMaxFeatures = 512;
constexpr int kThreads = 256, kWarps = kThreads / 32;

enum { kActNone = 0, kActRelu = 1, kActSigmoid = 2, kActSilu = 3 };

// act[j] = activation of g[j]; dact[j] = its derivative (only when asked for).  The activation is
// the same for the whole launch, so the choice is a branch around the loops.
template <bool GRAD, int N>
__device__ __forceinline__ void activate(const float (&g)[N], int kind, float (&act)[N], float (&dact)[N]) {
  if (kind == kActSigmoid || kind == kActSilu) {
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const float s = 1.f / (1.f + __expf(-g[j]));
      if (kind == kActSigmoid) {
        act[j] = s;
        if (GRAD) dact[j] = s * (1.f - s);
      } else {
        act[j] = g[j] * s;
        if (GRAD) dact[j] = s * (1.f + g[j] * (1.f - s));
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < N; ++j) {
      act[j] = kind == kActRelu ? fmaxf(g[j], 0.f) : g[j];
      if (GRAD) dact[j] = (kind == kActRelu && !(g[j] >= 0.f)) ? 0.f : 1.f;
    }
  }
}

// sum over the LPG consecutive lanes that share a (row, group)
template <int LPG>
__device__ __forceinline__ float lane_sum(float v) {
#pragma unroll
  for (int off = LPG / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

struct NormArgs {
  const void *x, *gate;
  const float *weight, *bias;  // (G * e) fp32 or null
  void *out;
  const void *d_out;
  void *dx, *dgate;
  float *dweight, *dbias;      // (G * e) fp32 accumulators (zeroed by the caller) or null
  long long rows;
  int G, e, act, post, use_mean;
  float c, eps;
};

// VEC consecutive elements of type T as one aligned access.
template <int BYTES> struct Raw;
template <> struct Raw<16> { typedef uint4 type; };
template <> struct Raw<8> { typedef uint2 type; };
template <typename T, int VEC> struct Pack {
  typedef typename Raw<VEC * (int)sizeof(T)>::type R;
  static __device__ __forceinline__ void unpack(const R &raw, float *v) {
    const T *h = reinterpret_cast<const T *>(&raw);
#pragma unroll
    for (int j = 0; j < VEC; ++j) v[j] = Cvt<T>::to_f(h[j]);
  }
  static __device__ __forceinline__ R pack(const float *v) {
    R raw;
    T *h = reinterpret_cast<T *>(&raw);
#pragma unroll
    for (int j = 0; j < VEC; ++j) h[j] = Cvt<T>::from_f(v[j]);
    return raw;
  }
};

// resident CTAs per SM (almost) without spills (N = features per lane)
template <typename T, bool BWD, bool POST, int N> constexpr int ctas_per_sm() {
  if (N <= 4 && sizeof(T) == 2) return BWD ? 4 : 8;
  return N <= (BWD && POST ? 4 : 8) ? 3 : (N <= 8 ? 2 : 1);
}

// Grid (CTAs over rows, G).  Lane l of the LPG lanes of a (row, group) owns NP packs of VEC features,
// pack p being features [(p LPG + l) VEC, +VEC); packs past e are zero.  The rows of a warp's next
// step are loaded before the current step is worked on.
//
// Bound by HBM: 75 MB forward / 126 MB backward at 16384 rows of 12 groups of 64 (bf16) are 11.5 / 19 us
// at the measured copy bandwidth; 22 / 39 us here, 52 / 198 with a whole warp per group, which left half its
// lanes idle at 64 features, had one 8-byte load per operand in flight and sent one atomic per warp and
// feature.  Groups that are no multiple of 8 features have 4 a lane and more CTAs per SM: 100 features, 32768 rows
// of 8 groups, 65 / 112 us (77 / 293 with a warp per group, 125 / 262 here with three CTAs).
//
// POST = false: no gate behind the norm (the backward then needs neither y nor the bias, which is
// what lets a third CTA onto the SM).
template <typename T, bool BWD, bool POST, int VEC, int LPG, int NP>
__global__ void __launch_bounds__(kThreads, (ctas_per_sm<T, BWD, POST, VEC * NP>())) norm_gate_kernel(const NormArgs a) {
  typedef Pack<T, VEC> P;
  typedef typename P::R R;
  constexpr int N = VEC * NP, RPW = 32 / LPG;
  // the next rows are loaded ahead, except where eight CTAs per SM cover the latency and leave no registers for it
  constexpr bool kAhead = BWD || N > 4 || sizeof(T) > 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gl = lane % LPG, sub = lane / LPG;
  const int g = blockIdx.y, e = a.e;
  const long long stride = (long long)a.G * e;
  const bool has_gate = a.gate != nullptr;
  float w[N], b[N], dw[N], db[N];
#pragma unroll
  for (int p = 0; p < NP; ++p)
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
      const int f = (p * LPG + gl) * VEC + j, i = p * VEC + j;
      w[i] = (a.weight != nullptr && f < e) ? a.weight[(long long)g * e + f] : 1.f;
      b[i] = ((POST || !BWD) && a.bias != nullptr && f < e) ? a.bias[(long long)g * e + f] : 0.f;
      dw[i] = db[i] = 0.f;
    }
  const float inv_e = 1.f / (float)e;
  const T *xp = static_cast<const T *>(a.x), *gp = static_cast<const T *>(a.gate), *dp = static_cast<const T *>(a.d_out);
  const long long step = (long long)gridDim.x * kWarps * RPW;
  R rx[NP], rg[NP], rd[NP];
  const R zero = {};
  auto fetch = [&](long long r) {
    // past the end: the last row again, with do = 0, so that such a lane adds 0 times a value of that row to the
    // gradient sums (x = 0 in its place would make that 0 * inf at eps = 0)
    const bool in = r < a.rows;
    const long long off = (in ? r : a.rows - 1) * stride + (long long)g * e;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const int f = (p * LPG + gl) * VEC;
      const bool on = f < e;
      rx[p] = on ? *reinterpret_cast<const R *>(xp + off + f) : zero;
      rg[p] = (on && has_gate) ? *reinterpret_cast<const R *>(gp + off + f) : zero;
      if (BWD) rd[p] = (on && in) ? *reinterpret_cast<const R *>(dp + off + f) : zero;
    }
  };
  const long long first = ((long long)blockIdx.x * kWarps + warp) * RPW;  // uniform over the warp
  if (kAhead) fetch(first + sub);
  for (long long r0 = first; r0 < a.rows; r0 += step) {
    const long long r = r0 + sub;
    const bool live = r < a.rows;
    const long long off = r * stride + (long long)g * e;
    if (!kAhead) fetch(r);
    float x[N], gt[N], d_o[N], act[N], dact[N], z[N];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      P::unpack(rx[p], x + p * VEC);
      P::unpack(rg[p], gt + p * VEC);
      if (BWD) P::unpack(rd[p], d_o + p * VEC);
    }
    if (kAhead) fetch(r + step);
    if (has_gate) {
      activate<BWD, N>(gt, a.act, act, dact);
    } else {
#pragma unroll
      for (int j = 0; j < N; ++j) { act[j] = 1.f; dact[j] = 0.f; }
    }
    const bool pre = has_gate && !a.post, post = POST && has_gate && a.post;
    float s1 = 0.f, s2 = 0.f, mean = 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      z[j] = pre ? x[j] * act[j] : x[j];
      s1 += z[j];
    }
    if (a.use_mean) mean = lane_sum<LPG>(s1) * inv_e;
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
      for (int j = p * VEC; j < (p + 1) * VEC; ++j) {
        z[j] = (p * LPG + gl) * VEC < e ? z[j] - mean : 0.f;  // zc (e is a multiple of VEC)
        s2 += z[j] * z[j];
      }
    const float rsig = rsqrtf(lane_sum<LPG>(s2) + a.eps);
    if (!BWD) {
      float o[N];
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const float y = a.c * z[j] * rsig * w[j] + b[j];
        o[j] = post ? y * act[j] : y;
      }
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const int f = (p * LPG + gl) * VEC;
        if (live && f < e) *reinterpret_cast<R *>(static_cast<T *>(a.out) + off + f) = P::pack(o + p * VEC);
      }
    } else {
      float dxh[N], dga[N];
      float dot = 0.f;
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const float xh = z[j] * rsig;                    // normalised value
        const float y = a.c * xh * w[j] + b[j];
        const float dy = post ? d_o[j] * act[j] : d_o[j];
        dga[j] = post ? d_o[j] * y : 0.f;                // d loss / d act(gate), post-gate part
        dw[j] += dy * a.c * xh;                          // rows past the end add zero (fetch)
        db[j] += dy;
        dxh[j] = dy * w[j] * a.c;
        dot += dxh[j] * xh;
      }
      dot = lane_sum<LPG>(dot);
      float s3 = 0.f;
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int j = p * VEC; j < (p + 1) * VEC; ++j) {
          const float xh = z[j] * rsig;
          dxh[j] = (p * LPG + gl) * VEC < e ? (dxh[j] - xh * dot) * rsig : 0.f;  // d loss / d zc
          s3 += dxh[j];
        }
      float dmean = 0.f;
      if (a.use_mean) dmean = lane_sum<LPG>(s3) * inv_e;
      float gx[N], gg[N];
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const float dz = dxh[j] - dmean;                 // d loss / d z
        gx[j] = pre ? dz * act[j] : dz;
        if (pre) dga[j] = dz * x[j];
        gg[j] = dga[j] * dact[j];
      }
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const int f = (p * LPG + gl) * VEC;
        if (live && f < e) {
          *reinterpret_cast<R *>(static_cast<T *>(a.dx) + off + f) = P::pack(gx + p * VEC);
          if (has_gate) *reinterpret_cast<R *>(static_cast<T *>(a.dgate) + off + f) = P::pack(gg + p * VEC);
        }
      }
    }
  }
  if (BWD && (a.dweight != nullptr || a.dbias != nullptr)) {  // uniform over the grid
    __shared__ float part[2][kWarps][LPG * N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
#pragma unroll
      for (int o = LPG; o < 32; o <<= 1) {
        dw[j] += __shfl_xor_sync(0xffffffffu, dw[j], o);
        db[j] += __shfl_xor_sync(0xffffffffu, db[j], o);
      }
      const int f = ((j / VEC) * LPG + gl) * VEC + j % VEC;
      if (sub == 0) {
        part[0][warp][f] = dw[j];
        part[1][warp][f] = db[j];
      }
    }
    __syncthreads();
    for (int f = threadIdx.x; f < e; f += kThreads) {
      float sw = 0.f, sb = 0.f;
#pragma unroll
      for (int k = 0; k < kWarps; ++k) {
        sw += part[0][k][f];
        sb += part[1][k][f];
      }
      if (a.dweight != nullptr) atomicAdd(a.dweight + (long long)g * e + f, sw);
      if (a.dbias != nullptr) atomicAdd(a.dbias + (long long)g * e + f, sb);
    }
  }
}

template <typename T, int VEC, int LPG, int NP>
int launch_cfg(const NormArgs &a, bool bwd, cudaStream_t st) {
  static int sms[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return LA_ERR_CUDA;
  if (sms[dev] == 0 && cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return LA_ERR_CUDA;
  const long long rows_per_cta = (long long)kWarps * (32 / LPG);
  long long blocks = (a.rows + rows_per_cta - 1) / rows_per_cta;
  // one wave over all groups: each CTA ends with its gradient sums, so few CTAs that walk many rows
  const bool post = a.gate != nullptr && a.post;
  const int resident = !bwd ? ctas_per_sm<T, false, true, VEC * NP>()
                            : (post ? ctas_per_sm<T, true, true, VEC * NP>() : ctas_per_sm<T, true, false, VEC * NP>());
  const long long cap = ((long long)sms[dev] * resident + a.G - 1) / a.G;
  if (blocks > cap) blocks = cap;
  dim3 grid((unsigned)blocks, (unsigned)a.G);
  if (!bwd) norm_gate_kernel<T, false, true, VEC, LPG, NP><<<grid, kThreads, 0, st>>>(a);
  else if (post) norm_gate_kernel<T, true, true, VEC, LPG, NP><<<grid, kThreads, 0, st>>>(a);
  else norm_gate_kernel<T, true, false, VEC, LPG, NP><<<grid, kThreads, 0, st>>>(a);
  return launch_status();
}

// VEC = features per access.  16-byte accesses (8 features of a 16-bit type) need groups of a multiple
// of 8 features and 16-byte aligned tensors; 16-bit tensors that have neither take 8-byte accesses.
template <typename T, int VEC>
int launch_vec(const NormArgs &a, bool bwd, cudaStream_t st) {
  const int lanes = (a.e + VEC - 1) / VEC;
  if (lanes <= 8) return launch_cfg<T, VEC, 8, 1>(a, bwd, st);
  if (lanes <= 16) return launch_cfg<T, VEC, 16, 1>(a, bwd, st);
  if (lanes <= 32) return launch_cfg<T, VEC, 32, 1>(a, bwd, st);
  if (lanes <= 64) return launch_cfg<T, VEC, 32, 2>(a, bwd, st);
  if constexpr (VEC == 4) return launch_cfg<T, VEC, 32, 4>(a, bwd, st);
  return LA_ERR_UNSUPPORTED;
}

template <typename T>
int launch_t(const NormArgs &a, bool bwd, cudaStream_t st) {
  if constexpr (sizeof(T) == 2) {
    const uintptr_t all = reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.gate) |
                          reinterpret_cast<uintptr_t>(a.out) | reinterpret_cast<uintptr_t>(a.d_out) |
                          reinterpret_cast<uintptr_t>(a.dx) | reinterpret_cast<uintptr_t>(a.dgate);
    if (a.e % 8 == 0 && (all & 15u) == 0) return launch_vec<T, 8>(a, bwd, st);
  }
  return launch_vec<T, 4>(a, bwd, st);
}

int dispatch(const NormArgs &a, int dtype, bool bwd, cudaStream_t st) {
  switch (dtype) {
    case LA_F32: return launch_t<float>(a, bwd, st);
    case LA_BF16: return launch_t<__nv_bfloat16>(a, bwd, st);
    case LA_F16: return launch_t<__half>(a, bwd, st);
  }
  return LA_ERR_UNSUPPORTED;
}

int check(const void *x, int64_t rows, int64_t G, int64_t e, int dtype, int act, int gate_pos) {
  cudaGetLastError();
  if (x == nullptr) return LA_ERR_NULL_POINTER;
  if (rows <= 0 || G <= 0 || e <= 0) return LA_ERR_BAD_SHAPE;
  if (e % 4 != 0 || e > kMaxFeatures || G > 65535) return LA_ERR_UNSUPPORTED;
  if (act < 0 || act > 3 || gate_pos < 0 || gate_pos > 1) return LA_ERR_UNSUPPORTED;
  if (!(dtype == LA_F32 || dtype == LA_BF16 || dtype == LA_F16)) return LA_ERR_UNSUPPORTED;
  return LA_OK;
}

}  // namespace
}  // namespace la

using namespace la;

extern "C" {

int la_normalize_gate_fwd(const void *x, const void *gate, const float *weight, const float *bias, void *out,
                          int64_t rows, int64_t G, int64_t e, int dtype, int act, int gate_pos, float c, float eps,
                          int use_mean, void *stream) {
  const int rc = check(x, rows, G, e, dtype, act, gate_pos);
  if (rc != LA_OK) return rc;
  if (out == nullptr) return LA_ERR_NULL_POINTER;
  NormArgs a = {};
  a.x = x; a.gate = gate; a.weight = weight; a.bias = bias; a.out = out;
  a.rows = rows; a.G = (int)G; a.e = (int)e; a.act = act; a.post = gate_pos; a.use_mean = use_mean;
  a.c = c; a.eps = eps;
  return dispatch(a, dtype, false, static_cast<cudaStream_t>(stream));
}

int la_normalize_gate_bwd(const void *x, const void *gate, const float *weight, const float *bias, const void *d_out,
                          void *dx, void *dgate, float *dweight, float *dbias, int64_t rows, int64_t G, int64_t e,
                          int dtype, int act, int gate_pos, float c, float eps, int use_mean, void *stream) {
  const int rc = check(x, rows, G, e, dtype, act, gate_pos);
  if (rc != LA_OK) return rc;
  if (d_out == nullptr || dx == nullptr || (gate != nullptr && dgate == nullptr)) return LA_ERR_NULL_POINTER;
  NormArgs a = {};
  a.x = x; a.gate = gate; a.weight = weight; a.bias = bias; a.d_out = d_out; a.dx = dx; a.dgate = dgate;
  a.dweight = dweight; a.dbias = dbias;
  a.rows = rows; a.G = (int)G; a.e = (int)e; a.act = act; a.post = gate_pos; a.use_mean = use_mean;
  a.c = c; a.eps = eps;
  return dispatch(a, dtype, true, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
