// Chunk-parallel scalar-decay forward in fp32 arithmetic on the CUDA cores.
//
// Serves what the tcgen05 kernels do not take and the token-by-token scan is slow at: fp32 inputs and
// 16-bit sequences shorter than one 128-token tile, head dimensions up to 128.  Same recurrence and
// the same fp32 products and sums as scan.cu, grouped by chunks of 64 tokens:
//
//   o_i = sum_{j <= i} (q_i . k_j) e^{c_i - c_j} v_j + e^{c_i} q_i S_in,    S_out = e^g S_in + sum_j e^{g - c_j} k_j v_j^T
//
// with c the cumulative log decay inside the chunk, held in double so that a difference of two large
// sums keeps its relative accuracy; e^{c_i - c_j} is one fp32 exponential of that difference, the 64 factors of
// a chunk's state update are rounded once from double.
//
// The sequence is cut into segments of whole chunks, one CTA per (segment, head) in each of three
// launches: (1) every segment's own state from a zero start, (2) a fold that turns those into the
// states entering the segments (and the final state), (3) the outputs.  The scan walks the tokens one
// by one, 0.77 us each whatever the GPU could hold (394 us for B 2, H 8, N 512, D 64; 24 us here); a segment
// costs a few 64 x 64 x D products, which the fp32 pipes bound.  All long sums run in blocks of 16 terms
// whose totals are then added up: the rounding error of a sum grows with its longest chain, and in
// one chain of 64 or 128 these products came out less exact than the scan, whose threads add 32.
#include <mutex>

#include "chunk.cuh"
#include "scan.cuh"

namespace la {
namespace {

constexpr int kC = 64;        // tokens per chunk
constexpr int kThreads = 256;  // 16 x 16
constexpr int kBlock = 16;     // terms of a sum added in one chain
constexpr int kPt = kC + 4;    // row pitch of P^T: float4 accesses, rows four banks apart

struct Args {
  const void *q, *k, *v;
  const float *ld;
  int64_t ld_sb, ld_sn, ld_sh;
  const float *s0;   // (B,H,D,E) or null
  float *s_fin;      // (B,H,D,E) or null
  void *o;
  float *seg_state;  // (B*H, nseg, D, E): own states, then (in place) entering states; null with one segment
  float *seg_decay;  // (B*H, nseg): e^{total log decay}
  int B, N, H, D, E, nseg, seg_tokens, ld_act;
};

template <int DT> struct Tile {
  static constexpr int kPitch = DT + 4;
  static constexpr int kFloats = kC * kPitch;
};

// rows [t0, t0 + 64) x F features of one head -> shared memory in fp32, zero past `rows` and F
template <typename T, int DT>
__device__ __forceinline__ void load_tile(float *dst, const T *src, int64_t row_stride, int rows, int F) {
  constexpr int kVec = 16 / (int)sizeof(T) < 8 ? 4 : 8, kPer = DT / kVec;
  for (int idx = threadIdx.x; idx < kC * kPer; idx += kThreads) {
    const int r = idx / kPer, f = (idx - r * kPer) * kVec;
    float *p = dst + r * Tile<DT>::kPitch + f;
#pragma unroll
    for (int h = 0; h < kVec; h += 4) {
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < rows && f + h < F) {  // F is a multiple of 4
        const T *s = src + r * row_stride + f + h;
        if (sizeof(T) == 4) {
          x = *reinterpret_cast<const float4 *>(s);
        } else {
          const uint2 u = *reinterpret_cast<const uint2 *>(s);
          const T *e = reinterpret_cast<const T *>(&u);
          x = make_float4(Cvt<T>::to_f(e[0]), Cvt<T>::to_f(e[1]), Cvt<T>::to_f(e[2]), Cvt<T>::to_f(e[3]));
        }
      }
      *reinterpret_cast<float4 *>(p + h) = x;
    }
  }
}

// Cumulative log decays of a chunk's rows (double, natural log) into cs[64]; rows past the end add
// nothing.  e^x is 0 in fp32 far above x = -1e4, so the clamp changes no factor; it keeps the
// differences of the cumulative sums defined (and exact to 1e-10) where a decay is -inf.
__device__ __forceinline__ void chunk_decays(const Args &a, int64_t b, int h, int t, int rows, double *cs) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    double x[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = 2 * lane + u;
      double l = 0.0;
      if (r < rows) {
        l = (double)a.ld[b * a.ld_sb + (int64_t)(t + r) * a.ld_sn + h * a.ld_sh];
        if (a.ld_act) l = l < 0.0 ? l - log1p(exp(l)) : -log1p(exp(-l));
        if (l < -1e4) l = -1e4;
      }
      x[u] = l;
    }
    double s = x[0] + x[1];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const double n = __shfl_up_sync(0xffffffffu, s, off);
      if (lane >= off) s += n;
    }
    // the sum before this lane's rows is the lane before's, not s minus the own part: that would carry a decay
    // that is not finite from an odd row to the even one before it
    double pre = __shfl_up_sync(0xffffffffu, s, 1);
    if (lane == 0) pre = 0.0;
    cs[2 * lane] = pre + x[0];
    cs[2 * lane + 1] = s;
  }
}

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void fma4(float (&acc)[4], float s, const float4 &x) {
  acc[0] = fmaf(s, x.x, acc[0]);
  acc[1] = fmaf(s, x.y, acc[1]);
  acc[2] = fmaf(s, x.z, acc[2]);
  acc[3] = fmaf(s, x.w, acc[3]);
}

__device__ __forceinline__ void mul4(float (&acc)[4], float s, const float4 &x) {
  acc[0] = s * x.x;
  acc[1] = s * x.y;
  acc[2] = s * x.z;
  acc[3] = s * x.w;
}

// Thread (ty, tx) owns state rows {ty 4 + r + 64 u} and columns {tx 4 + c + 64 w} (DT 128: u, w = 0, 1;
// DT 32: threads outside the 8 x 8 corner idle).
template <int DT> struct StateAcc {
  static constexpr int kU = DT > 64 ? 2 : 1;
  float v[kU][4][kU][4];
};
template <int DT>
__device__ __forceinline__ bool owns_state(int ty, int tx) { return DT >= 64 || (ty < DT / 4 && tx < DT / 4); }

// acc = sum_j w_j k_j v_j^T over the chunk
template <int DT>
__device__ __forceinline__ void state_product(StateAcc<DT> &acc, const float *ks, const float *vs, const float *wj,
                                              int ty, int tx) {
  constexpr int P = Tile<DT>::kPitch, U = StateAcc<DT>::kU;
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int w = 0; w < U; ++w)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc.v[u][r][w][c] = 0.f;
  if (!owns_state<DT>(ty, tx)) return;
#pragma unroll 1
  for (int j0 = 0; j0 < kC; j0 += kBlock) {
    StateAcc<DT> t;
#pragma unroll 4
    for (int jj = 0; jj < kBlock; ++jj) {
      const int j = j0 + jj;
      const float wt = wj[j];
      float4 vv[U];
#pragma unroll
      for (int w = 0; w < U; ++w) vv[w] = ld4(vs + j * P + tx * 4 + 64 * w);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float4 kk = ld4(ks + j * P + ty * 4 + 64 * u);
        const float kr[4] = {kk.x * wt, kk.y * wt, kk.z * wt, kk.w * wt};
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int w = 0; w < U; ++w) {
            if (jj == 0) mul4(t.v[u][r][w], kr[r], vv[w]);
            else fma4(t.v[u][r][w], kr[r], vv[w]);
          }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int w = 0; w < U; ++w)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc.v[u][r][w][c] += t.v[u][r][w][c];
  }
}

// Launch 1: the state a segment's own tokens build from a zero start, and its total decay.
template <typename T, int DT>
__global__ void __launch_bounds__(kThreads) seg_state_kernel(const Args a) {
  extern __shared__ __align__(16) float smem[];
  constexpr int U = StateAcc<DT>::kU;
  float *ks = smem, *vs = ks + Tile<DT>::kFloats, *wj = vs + Tile<DT>::kFloats;
  double *cs = reinterpret_cast<double *>(wj + kC);
  const int seg = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh - b * a.H;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int t_end = min(a.N, (seg + 1) * a.seg_tokens);
  StateAcc<DT> st;
  double total = 0.0;
  for (int t = seg * a.seg_tokens; t < t_end; t += kC) {
    const int rows = min(kC, t_end - t);
    const int64_t row = ((int64_t)b * a.N + t) * a.H + h;
    __syncthreads();  // the previous chunk's tiles have been read
    load_tile<T, DT>(ks, static_cast<const T *>(a.k) + row * a.D, (int64_t)a.H * a.D, rows, a.D);
    load_tile<T, DT>(vs, static_cast<const T *>(a.v) + row * a.E, (int64_t)a.H * a.E, rows, a.E);
    chunk_decays(a, b, h, t, rows, cs);
    __syncthreads();
    const double g = cs[kC - 1];
    if (threadIdx.x < kC) wj[threadIdx.x] = (float)exp(g - cs[threadIdx.x]);
    __syncthreads();
    StateAcc<DT> acc;
    state_product<DT>(acc, ks, vs, wj, ty, tx);
    const float eg = (float)exp(g);
    const bool first = t == seg * a.seg_tokens;
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int w = 0; w < U; ++w)
#pragma unroll
          for (int c = 0; c < 4; ++c)
            st.v[u][r][w][c] = first ? acc.v[u][r][w][c] : fmaf(st.v[u][r][w][c], eg, acc.v[u][r][w][c]);
    total += g;
  }
  if (owns_state<DT>(ty, tx)) {
    float *dst = a.seg_state + ((int64_t)bh * a.nseg + seg) * a.D * a.E;
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int w = 0; w < U; ++w) {
          const int d = ty * 4 + r + 64 * u, e = tx * 4 + 64 * w;
          if (d < a.D && e < a.E)
            *reinterpret_cast<float4 *>(dst + (int64_t)d * a.E + e) =
                make_float4(st.v[u][r][w][0], st.v[u][r][w][1], st.v[u][r][w][2], st.v[u][r][w][3]);
        }
  }
  if (threadIdx.x == 0) a.seg_decay[(int64_t)bh * a.nseg + seg] = (float)exp(total);
}

// Launch 2: own states -> entering states, in place; the end of the last segment is the final state.
// One thread per four state elements; the loads of a group of segments are issued together.
__global__ void __launch_bounds__(kThreads) seg_fold_kernel(const Args a) {
  const int quads = a.D * a.E / 4;
  const int64_t idx = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (idx >= (int64_t)a.B * a.H * quads) return;
  const int64_t bh = idx / quads;
  const int qd = (int)(idx - bh * quads);
  const int64_t slot = (int64_t)quads;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (a.s0 != nullptr) s = reinterpret_cast<const float4 *>(a.s0)[bh * quads + qd];
  float4 *p = reinterpret_cast<float4 *>(a.seg_state) + bh * a.nseg * slot + qd;
  const float *dec = a.seg_decay + bh * a.nseg;
  constexpr int kGroup = 8;
  for (int k0 = 0; k0 < a.nseg; k0 += kGroup) {
    float4 own[kGroup];
    float e[kGroup];
#pragma unroll
    for (int u = 0; u < kGroup; ++u)
      if (k0 + u < a.nseg) {
        own[u] = p[(k0 + u) * slot];
        e[u] = dec[k0 + u];
      }
#pragma unroll
    for (int u = 0; u < kGroup; ++u)
      if (k0 + u < a.nseg) {
        p[(k0 + u) * slot] = s;
        s = make_float4(fmaf(s.x, e[u], own[u].x), fmaf(s.y, e[u], own[u].y), fmaf(s.z, e[u], own[u].z),
                        fmaf(s.w, e[u], own[u].w));
      }
  }
  if (a.s_fin != nullptr) reinterpret_cast<float4 *>(a.s_fin)[bh * quads + qd] = s;
}

// Launch 3: outputs of a segment from its entering state (with one segment: from the caller's, and the
// final state as well).  Thread (ty, tx) owns output rows 4 ty .. 4 ty + 3 and columns tx 4 (+ 64).
template <typename T, int DT>
__global__ void __launch_bounds__(kThreads) seg_out_kernel(const Args a) {
  extern __shared__ __align__(16) float smem[];
  constexpr int P = Tile<DT>::kPitch, U = StateAcc<DT>::kU;
  float *qs = smem, *ks = qs + Tile<DT>::kFloats, *vs = ks + Tile<DT>::kFloats;
  float *ss = vs + Tile<DT>::kFloats;  // [DT][DT] running state
  float *pt = ss + DT * DT;            // [64 j][kPt]: masked P, transposed
  float *wj = pt + kC * kPt;
  double *cs = reinterpret_cast<double *>(wj + kC);
  const int seg = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh - b * a.H;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int t_begin = seg * a.seg_tokens, t_end = min(a.N, t_begin + a.seg_tokens);
  const float *s_in = a.nseg > 1 ? a.seg_state + ((int64_t)bh * a.nseg + seg) * a.D * a.E
                                 : (a.s0 != nullptr ? a.s0 + (int64_t)bh * a.D * a.E : nullptr);
  for (int idx = threadIdx.x; idx < DT * DT / 4; idx += kThreads) {
    const int d = idx / (DT / 4), e = (idx - d * (DT / 4)) * 4;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (s_in != nullptr && d < a.D && e < a.E) x = ld4(s_in + (int64_t)d * a.E + e);
    *reinterpret_cast<float4 *>(ss + d * DT + e) = x;
  }
  const bool keep_state = a.nseg == 1 && a.s_fin != nullptr;
  for (int t = t_begin; t < t_end; t += kC) {
    const int rows = min(kC, t_end - t);
    const int64_t row = ((int64_t)b * a.N + t) * a.H + h;
    load_tile<T, DT>(qs, static_cast<const T *>(a.q) + row * a.D, (int64_t)a.H * a.D, rows, a.D);
    load_tile<T, DT>(ks, static_cast<const T *>(a.k) + row * a.D, (int64_t)a.H * a.D, rows, a.D);
    load_tile<T, DT>(vs, static_cast<const T *>(a.v) + row * a.E, (int64_t)a.H * a.E, rows, a.E);
    chunk_decays(a, b, h, t, rows, cs);
    __syncthreads();
    if (threadIdx.x < kC) wj[threadIdx.x] = (float)exp(cs[kC - 1] - cs[threadIdx.x]);
    // ---- P = Q K^T, rows 4 ty + r, columns tx + 16 s (the row pitch spreads these over the banks)
    {
      float p[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int s = 0; s < 4; ++s) p[r][s] = 0.f;
#pragma unroll 1
      for (int d0 = 0; d0 < DT; d0 += kBlock) {
        float t[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int s = 0; s < 4; ++s) t[r][s] = 0.f;
#pragma unroll
        for (int d = d0; d < d0 + kBlock; d += 4) {
          float4 qv[4], kv[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) qv[r] = ld4(qs + (4 * ty + r) * P + d);
#pragma unroll
          for (int s = 0; s < 4; ++s) kv[s] = ld4(ks + (tx + 16 * s) * P + d);
#pragma unroll
          for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int s = 0; s < 4; ++s) {
              t[r][s] = fmaf(qv[r].x, kv[s].x, t[r][s]);
              t[r][s] = fmaf(qv[r].y, kv[s].y, t[r][s]);
              t[r][s] = fmaf(qv[r].z, kv[s].z, t[r][s]);
              t[r][s] = fmaf(qv[r].w, kv[s].w, t[r][s]);
            }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int s = 0; s < 4; ++s) p[r][s] += t[r][s];
      }
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const int j = tx + 16 * s;
        float m[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int i = 4 * ty + r;
          m[r] = j <= i ? p[r][s] * expf((float)(cs[i] - cs[j])) : 0.f;
        }
        *reinterpret_cast<float4 *>(pt + j * kPt + 4 * ty) = make_float4(m[0], m[1], m[2], m[3]);
      }
    }
    __syncthreads();
    if (owns_state<DT>(0, tx)) {
      float o[4][U][4];
      // ---- e^{c_i} q_i S_in
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int w = 0; w < U; ++w)
#pragma unroll
          for (int c = 0; c < 4; ++c) o[r][w][c] = 0.f;
      float t[4][U][4];
      auto clear = [&]() {
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int w = 0; w < U; ++w)
#pragma unroll
            for (int c = 0; c < 4; ++c) t[r][w][c] = 0.f;
      };
      auto fold = [&]() {
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int w = 0; w < U; ++w)
#pragma unroll
            for (int c = 0; c < 4; ++c) o[r][w][c] += t[r][w][c];
      };
#pragma unroll 1
      for (int d0 = 0; d0 < DT; d0 += kBlock) {
        clear();
#pragma unroll
        for (int d = d0; d < d0 + kBlock; d += 4) {
          float4 qv[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) qv[r] = ld4(qs + (4 * ty + r) * P + d);
#pragma unroll
          for (int dd = 0; dd < 4; ++dd)
#pragma unroll
            for (int w = 0; w < U; ++w) {
              const float4 sv = ld4(ss + (d + dd) * DT + tx * 4 + 64 * w);
#pragma unroll
              for (int r = 0; r < 4; ++r)
                fma4(t[r][w], dd == 0 ? qv[r].x : dd == 1 ? qv[r].y : dd == 2 ? qv[r].z : qv[r].w, sv);
            }
        }
        fold();
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float e = (float)exp(cs[4 * ty + r]);
#pragma unroll
        for (int w = 0; w < U; ++w)
#pragma unroll
          for (int c = 0; c < 4; ++c) o[r][w][c] *= e;
      }
      // ---- P~ V over j <= i only, so that a later token's v never meets an earlier row (0 * inf)
#pragma unroll 1
      for (int j0 = 0; j0 <= 4 * ty; j0 += kBlock) {
        clear();
        const int j1 = min(j0 + kBlock, 4 * ty);
#pragma unroll 4
        for (int j = j0; j < j1; ++j) {
          const float4 pv = ld4(pt + j * kPt + 4 * ty);
#pragma unroll
          for (int w = 0; w < U; ++w) {
            const float4 vv = ld4(vs + j * P + tx * 4 + 64 * w);
            fma4(t[0][w], pv.x, vv);
            fma4(t[1][w], pv.y, vv);
            fma4(t[2][w], pv.z, vv);
            fma4(t[3][w], pv.w, vv);
          }
        }
        if (j0 + kBlock > 4 * ty) {  // the block with the diagonal
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            const float4 pv = ld4(pt + (4 * ty + jj) * kPt + 4 * ty);
            const float pr[4] = {pv.x, pv.y, pv.z, pv.w};
#pragma unroll
            for (int w = 0; w < U; ++w) {
              const float4 vv = ld4(vs + (4 * ty + jj) * P + tx * 4 + 64 * w);
#pragma unroll
              for (int r = jj; r < 4; ++r) fma4(t[r][w], pr[r], vv);
            }
          }
        }
        fold();
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int w = 0; w < U; ++w) {
          const int i = 4 * ty + r, e = tx * 4 + 64 * w;
          if (i < rows && e < a.E) {
            T *dst = static_cast<T *>(a.o) + (row + (int64_t)i * a.H) * a.E + e;
            if (sizeof(T) == 4) {
              *reinterpret_cast<float4 *>(dst) = make_float4(o[r][w][0], o[r][w][1], o[r][w][2], o[r][w][3]);
            } else {
              T x[4] = {Cvt<T>::from_f(o[r][w][0]), Cvt<T>::from_f(o[r][w][1]), Cvt<T>::from_f(o[r][w][2]),
                        Cvt<T>::from_f(o[r][w][3])};
              *reinterpret_cast<uint2 *>(dst) = *reinterpret_cast<const uint2 *>(x);
            }
          }
        }
    }
    // ---- the state after this chunk, if anything reads it
    if (t + kC < t_end || keep_state) {  // uniform over the CTA
      StateAcc<DT> acc;
      state_product<DT>(acc, ks, vs, wj, ty, tx);
      const float eg = (float)exp(cs[kC - 1]);
      __syncthreads();  // S_in and the tiles have been read
      if (owns_state<DT>(ty, tx)) {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int w = 0; w < U; ++w) {
              float4 *p = reinterpret_cast<float4 *>(ss + (ty * 4 + r + 64 * u) * DT + tx * 4 + 64 * w);
              const float4 x = *p;
              *p = make_float4(fmaf(x.x, eg, acc.v[u][r][w][0]), fmaf(x.y, eg, acc.v[u][r][w][1]),
                               fmaf(x.z, eg, acc.v[u][r][w][2]), fmaf(x.w, eg, acc.v[u][r][w][3]));
            }
      }
    }
  }
  if (keep_state) {
    __syncthreads();
    float *dst = a.s_fin + (int64_t)bh * a.D * a.E;
    for (int idx = threadIdx.x; idx < DT * DT / 4; idx += kThreads) {
      const int d = idx / (DT / 4), e = (idx - d * (DT / 4)) * 4;
      if (d < a.D && e < a.E) *reinterpret_cast<float4 *>(dst + (int64_t)d * a.E + e) = ld4(ss + d * DT + e);
    }
  }
}

template <int DT> constexpr int state_smem() {
  return (int)sizeof(float) * (2 * Tile<DT>::kFloats + kC) + (int)sizeof(double) * kC;
}
template <int DT> constexpr int out_smem() {
  return (int)sizeof(float) * (3 * Tile<DT>::kFloats + DT * DT + kC * kPt + kC) + (int)sizeof(double) * kC;
}

template <typename T, int DT>
int launch_dt(Args &a, cudaStream_t st) {
  static std::mutex mu;
  static bool ready[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return LA_ERR_CUDA;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!ready[dev]) {
      if (cudaFuncSetAttribute(seg_state_kernel<T, DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, state_smem<DT>()) != cudaSuccess ||
          cudaFuncSetAttribute(seg_out_kernel<T, DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, out_smem<DT>()) != cudaSuccess)
        return LA_ERR_CUDA;
      ready[dev] = true;
    }
  }
  const dim3 grid((unsigned)a.nseg, (unsigned)(a.B * a.H));
  int rc;
  if (a.nseg > 1) {
    seg_state_kernel<T, DT><<<grid, kThreads, state_smem<DT>(), st>>>(a);
    if ((rc = launch_status()) != LA_OK) return rc;
    const int64_t quads = (int64_t)a.B * a.H * (a.D * a.E / 4);
    seg_fold_kernel<<<(unsigned)((quads + kThreads - 1) / kThreads), kThreads, 0, st>>>(a);
    if ((rc = launch_status()) != LA_OK) return rc;
  }
  seg_out_kernel<T, DT><<<grid, kThreads, out_smem<DT>(), st>>>(a);
  return launch_status();
}

template <typename T>
int launch_t(Args &a, cudaStream_t st) {
  const int f = a.D > a.E ? a.D : a.E;
  if (f <= 32) return launch_dt<T, 32>(a, st);
  if (f <= 64) return launch_dt<T, 64>(a, st);
  return launch_dt<T, 128>(a, st);
}

// How a call is cut: chunks per segment and segments per sequence; per = 0: a call for the scan.
struct Plan {
  int per, nseg;
};

// The shapes the chunk form takes (four features per access) and, of those, the ones it is quicker for.
// Below 16 tokens the scan's few steps are as quick as these launches.
//
// A CTA works on all 64 rows of a chunk and on a square tile of features however few of them there are, and
// holds 50, 86 or 185 KB of shared memory, so its time goes by chunks and by CTAs per SM.  The scan's goes by
// the tokens: a step's latency while the GPU has room (its CTAs grow once there are two per SM), then its
// arithmetic on the padded state.  The constants are fitted to 1193 calls (fp32 and bf16; 4 to 128 features, D
// and E equal or not; 16 to 2048 tokens; 1 to 8192 pairs), e.g., in us, chunk form / scan:
//   128 features   64 tokens, 16 pairs 31 / 95, 8192 pairs 1697 / 3531;  16 tokens, 8192 pairs 1553 / 1025
//    32 features   64 tokens, 16 pairs 13 / 37, 8192 pairs 452 / 282;  2048 tokens, 16 pairs 46 / 1081
// Among those the choice is never slower than the scan by more than 2 us, and where it stays with the scan that
// costs at most 1.24 times the chunk form's time (32 tokens of 192 pairs of 16 features, 21 us).
Plan plan_of(int64_t B, int64_t N, int64_t H, int64_t D, int64_t E, bool scratch) {
  if (D > 128 || E > 128 || D % 4 != 0 || E % 4 != 0 || N < 16 || B * H > 65535) return {0, 0};
  const int dev_sms = device_sms();
  const int64_t pairs = B * H, chunks = (N + kC - 1) / kC, sms = dev_sms > 0 ? dev_sms : 1;
  // with scratch, as many segments as keep about two CTAs per SM (the states of the segments are then at most
  // 2 x SMs + B H of D x E floats, whatever N is)
  int64_t parts = scratch ? (2 * sms + pairs - 1) / pairs : 1;
  if (parts > chunks) parts = chunks;
  const int64_t per = (chunks + parts - 1) / parts, nseg = (chunks + per - 1) / per;
  const int tile = D > 64 || E > 64 ? 2 : (D > 32 || E > 32 ? 1 : 0), cols = D > 64 ? 2 : (D > 32 ? 1 : 0);
  static const double kChunkUs[3] = {7.8, 11.8, 27.5}, kStartUs[3] = {5.0, 4.0, 1.5};
  const double ctas_per_sm = (double)((pairs * nseg + sms - 1) / sms);
  double chunk_us = kStartUs[tile] + kChunkUs[tile] * ctas_per_sm * per;
  if (nseg > 1) chunk_us = kStartUs[tile] + 6.0 + 1.2 * kChunkUs[tile] * ctas_per_sm * per;  // three launches
  // a scan step's latency: up to 32 pairs, fewer pairs than SMs, fewer than two per SM, more (with few rows
  // the CTAs of 128 columns stay small)
  static const double kStepUs[4][3] = {{0.53, 0.77, 1.35}, {0.47, 0.58, 0.9}, {0.45, 0.56, 1.5}, {0.47, 0.66, 1.6}};
  static const double kElementUs[3] = {5.0e-7, 3.45e-7, 3.9e-7};  // per state element of a pair and token
  int level = pairs <= 32 ? 0 : (pairs < sms ? 1 : (pairs < 2 * sms ? 2 : 3));
  if (cols == 2 && level > 1 && (E <= 32 || (E <= 64 && level == 2))) level = 1;
  int64_t rows = 8;
  while (rows < E) rows *= 2;
  const double work_us = kElementUs[cols] * (double)(32 << cols) * (double)rows * (double)pairs * 148.0 / (double)sms;
  const double step_us = kStepUs[level][cols];
  const double scan_us = 4.5 + (double)N * (work_us > step_us ? work_us : step_us);
  if (chunk_us > scan_us) return {0, 0};
  return {(int)per, (int)nseg};
}

int64_t plan_bytes(const Plan &p, int64_t pairs, int64_t D, int64_t E) {
  return p.nseg > 1 ? pairs * p.nseg * (D * E + 1) * (int64_t)sizeof(float) : 0;
}

}  // namespace

int64_t fp32_chunk_fwd_workspace(int64_t B, int64_t N, int64_t H, int64_t D, int64_t E) {
  return plan_bytes(plan_of(B, N, H, D, E, true), B * H, D, E);
}

// LA_ERR_UNSUPPORTED: the call is one for the scan kernels.  With neither a workspace nor the pool (or where that
// has no memory) the whole sequence is one segment: no scratch, one launch.
int launch_fp32_chunk_fwd(const void *q, const void *k, const void *v, const float *ld, int64_t ld_sb, int64_t ld_sn,
                          int64_t ld_sh, const float *s0, void *o, float *s_fin, void *workspace, int64_t workspace_bytes,
                          int use_pool, int B, int N, int H, int D, int E, int dtype, int ld_act, cudaStream_t st) {
  // one 16-byte aligned row start per tensor
  const uintptr_t rows = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
                         reinterpret_cast<uintptr_t>(o);
  const uintptr_t states = reinterpret_cast<uintptr_t>(s0) | reinterpret_cast<uintptr_t>(s_fin);
  if ((rows & (dtype == LA_F32 ? 15u : 7u)) != 0 || (states & 15u) != 0) return LA_ERR_UNSUPPORTED;
  const int64_t pairs = (int64_t)B * H;
  Plan p = plan_of(B, N, H, D, E, workspace != nullptr || use_pool);
  void *scratch = workspace, *pooled = nullptr;
  if (plan_bytes(p, pairs, D, E) > 0) {
    if (workspace != nullptr) {
      if (workspace_bytes < plan_bytes(p, pairs, D, E)) return LA_ERR_WORKSPACE;
      if ((reinterpret_cast<uintptr_t>(workspace) & 15u) != 0) return LA_ERR_MISALIGNED;
    } else if (scratch_alloc(&pooled, (size_t)plan_bytes(p, pairs, D, E), st) == LA_OK) {
      scratch = pooled;
    } else {
      p = plan_of(B, N, H, D, E, false);
    }
  }
  if (p.per == 0) return LA_ERR_UNSUPPORTED;
  Args a = {};
  a.q = q; a.k = k; a.v = v; a.ld = ld; a.ld_sb = ld_sb; a.ld_sn = ld_sn; a.ld_sh = ld_sh;
  a.s0 = s0; a.s_fin = s_fin; a.o = o;
  a.B = B; a.N = N; a.H = H; a.D = D; a.E = E; a.ld_act = ld_act;
  a.nseg = p.nseg;
  a.seg_tokens = p.per * kC;
  if (p.nseg > 1) {
    a.seg_state = static_cast<float *>(scratch);
    a.seg_decay = a.seg_state + pairs * a.nseg * D * E;
  }
  int rc = LA_ERR_UNSUPPORTED;
  switch (dtype) {
    case LA_F32: rc = launch_t<float>(a, st); break;
    case LA_BF16: rc = launch_t<__nv_bfloat16>(a, st); break;
    case LA_F16: rc = launch_t<__half>(a, st); break;
  }
  if (pooled != nullptr && cudaFreeAsync(pooled, st) != cudaSuccess && rc == LA_OK) rc = LA_ERR_CUDA;
  return rc;
}

}  // namespace la
