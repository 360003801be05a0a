// Register-resident FFT passes: an M-point complex Stockham transform by
// T = M / E threads that hold E complex values each, in passes of radix 4, 8 or
// 16 whose values meet in shared memory only between passes. A 512-point
// transform is three radix-8 passes with two exchanges; as radix-4 stages in
// place (tanb_fft.cuh) it is five stages with ten block barriers and five round
// trips through shared memory. What bounds these kernels is that chain of
// barriers (one transform per block) or the shared-memory pipe (thousands).
//
// The radices read the same forwards and backwards where that is possible
// (all sizes but 32 and 8192 points): then the inverse transform's first pass
// takes its inputs where the forward transform's last pass left its outputs,
// and of the bin pairs (k, M - k) that the real-transform steps and the
// spectral product need, each thread already holds the lower half.
//
// Every product and sum is an explicit round-to-nearest operation, so two
// kernels that run the same passes give the same bits whatever else they
// contain (the one-block and the many-block forms of the convolution rely on
// it).
//
// Twiddles: a table of 2M entries per size, W_2M^k = exp(-2 pi i k / 2M) for
// k < M (the real-transform steps), then for each pass after the first
// W_{R Ns}^{r k} stored [r - 1][k], k < Ns, so that a warp reads consecutive
// entries: sum (R - 1) Ns < M of them. All computed in double on the host.
#pragma once

#include "tanb_fft.cuh"

namespace tanb {

__host__ __device__ constexpr int reg_fft_passes(int l) { return l <= 6 ? 2 : (l <= 12 ? 3 : 4); }
// log2 of the radix of pass p
__host__ __device__ constexpr int reg_fft_lr(int l, int p) {
  constexpr int t[15][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}, {0, 0, 0, 0}, {0, 0, 0, 0}, {0, 0, 0, 0},
                            {2, 3, 0, 0}, {3, 3, 0, 0}, {2, 3, 2, 0}, {3, 2, 3, 0}, {3, 3, 3, 0},
                            {3, 4, 3, 0}, {4, 3, 4, 0}, {4, 4, 4, 0}, {4, 3, 3, 3}, {4, 3, 3, 4}};
  return t[l][p];
}
// span of pass p: the product of the radices before it
__host__ __device__ constexpr int reg_fft_span(int l, int p) {
  int s = 0;
  for (int q = 0; q < p; ++q) s += reg_fft_lr(l, q);
  return 1 << s;
}
// offset of pass p's twiddles (p >= 1) behind the first M entries of the table
__host__ __device__ constexpr int reg_fft_twoff(int l, int p) {
  int n = 0;
  for (int q = 1; q < p; ++q) n += ((1 << reg_fft_lr(l, q)) - 1) * reg_fft_span(l, q);
  return n;
}

// Entry i of the size's table is W_2M^j with this j (unused entries: 0).
__host__ __device__ inline int plan_twiddle_index(int l, int i) {
  const int M = 1 << l;
  if (i < M) return i;
  int q = i - M;
  for (int p = 1; p < reg_fft_passes(l); ++p) {
    const int R = 1 << reg_fft_lr(l, p), Ns = reg_fft_span(l, p);
    if (q < (R - 1) * Ns) return (1 + q / Ns) * (q % Ns) * (2 * M / (R * Ns));
    q -= (R - 1) * Ns;
  }
  return 0;
}

template <int LOG2M>
struct RegFft {
  static constexpr int M = 1 << LOG2M;
  // complex values per thread (16384 points: 512 threads, 128 registers each)
  static constexpr int E = LOG2M <= 9 ? 8 : (LOG2M <= 13 ? 16 : 32);
  static constexpr int T = M / E;
  static constexpr int NP = reg_fft_passes(LOG2M);
  static constexpr int R0 = 1 << reg_fft_lr(LOG2M, 0);
  static constexpr int RL = 1 << reg_fft_lr(LOG2M, NP - 1);
  static constexpr bool SYM = R0 == RL;
  // Shared-memory slots are padded by one per 2^PS so that the first pass's
  // stores (stride R0) spread over the banks.
  static constexpr int PS = R0 >= 16 ? 4 : 3;
  static constexpr int PM = M + (M >> PS);
  static __device__ __forceinline__ int pad(int i) { return i + (i >> PS); }
  static constexpr int radix(int p) { return 1 << reg_fft_lr(LOG2M, p); }
  static constexpr int span(int p) { return reg_fft_span(LOG2M, p); }
  static constexpr int twn(int p) { return (radix(p) - 1) * (E / radix(p)); }  // twiddles per thread of pass p
  static constexpr int tw_total() {
    int n = 0;
    for (int p = 1; p < NP; ++p) n += twn(p);
    return n;
  }
  static constexpr int TWT = tw_total();
  static constexpr int tw_base(int p) {
    int n = 0;
    for (int q = 1; q < p; ++q) n += twn(q);
    return n;
  }
};

__device__ __forceinline__ float2 x_add(float2 a, float2 b) {
  return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y));
}
__device__ __forceinline__ float2 x_sub(float2 a, float2 b) {
  return make_float2(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y));
}
__device__ __forceinline__ float2 x_mul(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}
// a * conj(b)
__device__ __forceinline__ float2 x_mulc(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, __fmul_rn(a.y, b.y)), __fmaf_rn(a.y, b.x, -__fmul_rn(a.x, b.y)));
}

// a, b, c, d -> their 4-point DFT (forward: exp(-i), inverse: exp(+i))
template <bool INV>
__device__ __forceinline__ void x_dft4(float2& a, float2& b, float2& c, float2& d) {
  const float2 t0 = x_add(a, c), t1 = x_sub(a, c), t2 = x_add(b, d), t3 = x_sub(b, d);
  a = x_add(t0, t2);
  c = x_sub(t0, t2);
  const float2 p = make_float2(__fadd_rn(t1.x, t3.y), __fsub_rn(t1.y, t3.x));  // t1 - i t3
  const float2 m = make_float2(__fsub_rn(t1.x, t3.y), __fadd_rn(t1.y, t3.x));  // t1 + i t3
  b = INV ? m : p;
  d = INV ? p : m;
}

template <bool INV>
__device__ __forceinline__ void x_dft8(float2* v) {
  float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  x_dft4<INV>(e0, e1, e2, e3);
  x_dft4<INV>(o0, o1, o2, o3);
  const float r = 0.70710678118654752f;
  // o1 W_8 = r s1, o2 W_8^2 = s2, o3 W_8^3 = r s3
  const float2 s1 = INV ? make_float2(__fsub_rn(o1.x, o1.y), __fadd_rn(o1.y, o1.x))
                        : make_float2(__fadd_rn(o1.x, o1.y), __fsub_rn(o1.y, o1.x));
  const float2 s2 = INV ? make_float2(-o2.y, o2.x) : make_float2(o2.y, -o2.x);
  const float2 s3 = INV ? make_float2(-__fadd_rn(o3.x, o3.y), __fsub_rn(o3.x, o3.y))
                        : make_float2(__fsub_rn(o3.y, o3.x), -__fadd_rn(o3.x, o3.y));
  v[0] = x_add(e0, o0);
  v[4] = x_sub(e0, o0);
  v[1] = make_float2(__fmaf_rn(r, s1.x, e1.x), __fmaf_rn(r, s1.y, e1.y));
  v[5] = make_float2(__fmaf_rn(-r, s1.x, e1.x), __fmaf_rn(-r, s1.y, e1.y));
  v[2] = x_add(e2, s2);
  v[6] = x_sub(e2, s2);
  v[3] = make_float2(__fmaf_rn(r, s3.x, e3.x), __fmaf_rn(r, s3.y, e3.y));
  v[7] = make_float2(__fmaf_rn(-r, s3.x, e3.x), __fmaf_rn(-r, s3.y, e3.y));
}

// v times W_16^n (inverse: its conjugate) for the n that a 16-point DFT needs
template <bool INV, int n>
__device__ __forceinline__ float2 x_w16(float2 v) {
  constexpr float c = 0.92387953251128674f, s = 0.38268343236508977f, r = 0.70710678118654752f;
  if constexpr (n == 0) {
    return v;
  } else if constexpr (n == 4) {
    return INV ? make_float2(-v.y, v.x) : make_float2(v.y, -v.x);
  } else {
    constexpr float wx = n == 1 ? c : n == 2 ? r : n == 3 ? s : n == 6 ? -r : /* 9 */ -c;
    constexpr float wy = n == 1 ? -s : n == 2 ? -r : n == 3 ? -c : n == 6 ? -r : /* 9 */ s;
    return INV ? x_mulc(v, make_float2(wx, wy)) : x_mul(v, make_float2(wx, wy));
  }
}

template <bool INV>
__device__ __forceinline__ void x_dft16(float2* v) {
#pragma unroll
  for (int r = 0; r < 4; ++r) x_dft4<INV>(v[r], v[r + 4], v[r + 8], v[r + 12]);
  // v[r + 4 q] = y_r[q]; times W_16^(r q)
  v[5] = x_w16<INV, 1>(v[5]);
  v[9] = x_w16<INV, 2>(v[9]);
  v[13] = x_w16<INV, 3>(v[13]);
  v[6] = x_w16<INV, 2>(v[6]);
  v[10] = x_w16<INV, 4>(v[10]);
  v[14] = x_w16<INV, 6>(v[14]);
  v[7] = x_w16<INV, 3>(v[7]);
  v[11] = x_w16<INV, 6>(v[11]);
  v[15] = x_w16<INV, 9>(v[15]);
  // X[q + 4 s] = sum_r W_4^(r s) y_r[q]
#pragma unroll
  for (int q = 0; q < 4; ++q) x_dft4<INV>(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
  // v[4 q + s] -> X[q + 4 s]: transpose
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int s = q + 1; s < 4; ++s) {
      const float2 t = v[4 * q + s];
      v[4 * q + s] = v[4 * s + q];
      v[4 * s + q] = t;
    }
}

template <int R, bool INV>
__device__ __forceinline__ void x_dft(float2* v) {
  if constexpr (R == 4) x_dft4<INV>(v[0], v[1], v[2], v[3]);
  else if constexpr (R == 8) x_dft8<INV>(v);
  else x_dft16<INV>(v);
}

// Pass P of the transform on registers: butterfly e of thread t is j = t + e T,
// v[e R + r] its inputs x[j + r M / R], on return its outputs
// X[((j - k) R + k) + r Ns], k = j mod Ns. `w`: the pass's twiddles of this
// thread in the same order (r = 1 .. R - 1), as reg_twiddles loads them.
template <int LOG2M, int P, bool INV>
__device__ __forceinline__ void reg_pass(float2* v, const float2* w) {
  using F = RegFft<LOG2M>;
  constexpr int R = F::radix(P);
#pragma unroll
  for (int e = 0; e < F::E / R; ++e) {
    if constexpr (P > 0) {
#pragma unroll
      for (int r = 1; r < R; ++r)
        v[e * R + r] = INV ? x_mulc(v[e * R + r], w[e * (R - 1) + r - 1]) : x_mul(v[e * R + r], w[e * (R - 1) + r - 1]);
    }
    x_dft<R, INV>(v + e * R);
  }
}

// The same with each butterfly's twiddles read from the table as it needs them.
template <int LOG2M, int P, bool INV>
__device__ __forceinline__ void reg_pass_table(float2* v, const float2* __restrict__ tw, int t) {
  using F = RegFft<LOG2M>;
  constexpr int R = F::radix(P), Ns = F::span(P);
  const float2* s = tw + F::M + reg_fft_twoff(LOG2M, P);
#pragma unroll
  for (int e = 0; e < F::E / R; ++e) {
    const int k = (t + e * F::T) & (Ns - 1);
#pragma unroll
    for (int r = 1; r < R; ++r) {
      const float2 w = s[(r - 1) * Ns + k];
      v[e * R + r] = INV ? x_mulc(v[e * R + r], w) : x_mul(v[e * R + r], w);
    }
    x_dft<R, INV>(v + e * R);
  }
}

// This thread's twiddles of pass P from the table (global or shared memory).
template <int LOG2M, int P>
__device__ __forceinline__ void reg_twiddles(float2* w, const float2* __restrict__ tw, int t) {
  using F = RegFft<LOG2M>;
  constexpr int R = F::radix(P), Ns = F::span(P);
  const float2* s = tw + F::M + reg_fft_twoff(LOG2M, P);
#pragma unroll
  for (int e = 0; e < F::E / R; ++e) {
    const int k = (t + e * F::T) & (Ns - 1);
#pragma unroll
    for (int r = 1; r < R; ++r) w[e * (R - 1) + r - 1] = s[(r - 1) * Ns + k];
  }
}

// Outputs of pass P to the padded buffer, inputs of pass P from it.
template <int LOG2M, int P>
__device__ __forceinline__ void reg_store(const float2* v, float2* buf, int t) {
  using F = RegFft<LOG2M>;
  constexpr int R = F::radix(P), Ns = F::span(P);
#pragma unroll
  for (int e = 0; e < F::E / R; ++e) {
    const int j = t + e * F::T, k = j & (Ns - 1), d = ((j - k) * R) + k;
#pragma unroll
    for (int r = 0; r < R; ++r) buf[F::pad(d + r * Ns)] = v[e * R + r];
  }
}
template <int LOG2M, int P>
__device__ __forceinline__ void reg_load(float2* v, const float2* buf, int t) {
  using F = RegFft<LOG2M>;
  constexpr int R = F::radix(P), S = F::M / R;
#pragma unroll
  for (int e = 0; e < F::E / R; ++e)
#pragma unroll
    for (int r = 0; r < R; ++r) v[e * R + r] = buf[F::pad(t + e * F::T + r * S)];
}

// Index of the value that register i holds before the first pass (and, with a
// symmetric plan, after the last one).
template <int LOG2M>
__device__ __forceinline__ int reg_in_index(int t, int i) {
  using F = RegFft<LOG2M>;
  return t + (i / F::R0) * F::T + (i % F::R0) * (F::M / F::R0);
}
// Index of the value that register i holds after the last pass.
template <int LOG2M>
__device__ __forceinline__ int reg_out_index(int t, int i) {
  using F = RegFft<LOG2M>;
  return t + (i / F::RL) * F::T + (i % F::RL) * (F::M / F::RL);
}

// Passes after the first (v holds pass 0's inputs), exchanging through buf0 and
// buf1 in turn (buf0 == buf1: one buffer, two barriers per exchange). `w`: all
// the passes' twiddles in registers when WREG, else read from the table `tw` as
// each pass needs them. `sync` is the barrier of the transform's threads. Ends
// with the outputs in registers and the last exchange's loads not yet fenced.
template <int LOG2M, bool INV, bool WREG, class Sync, int P = 0>
__device__ __forceinline__ void reg_fft(float2* v, const float2* w, const float2* __restrict__ tw, float2* buf0,
                                        float2* buf1, int t, Sync&& sync) {
  using F = RegFft<LOG2M>;
  if constexpr (P > 0 && !WREG) {
    reg_pass_table<LOG2M, P, INV>(v, tw, t);
  } else {
    reg_pass<LOG2M, P, INV>(v, w + F::tw_base(P));
  }
  if constexpr (P + 1 < F::NP) {
    reg_store<LOG2M, P>(v, buf0, t);
    sync();
    reg_load<LOG2M, P + 1>(v, buf0, t);
    if (buf0 == buf1) sync();
    reg_fft<LOG2M, INV, WREG, Sync, P + 1>(v, w, tw, buf1, buf0, t, sync);
  }
}

// Real-transform steps of the bin pair (k, M - k), 0 < k < M / 2: a = Z[k],
// b = Z[M - k], w = W_2M^k. W_2M^(M-k) = -conj(w), so one product serves both.
__device__ __forceinline__ void x_post(float2 a, float2 b, float2 w, float2& Xk, float2& Xm) {
  const float ex = __fmul_rn(0.5f, __fadd_rn(a.x, b.x)), ey = __fmul_rn(0.5f, __fsub_rn(a.y, b.y));
  const float2 d = make_float2(__fmul_rn(0.5f, __fsub_rn(a.x, b.x)), __fmul_rn(0.5f, __fadd_rn(a.y, b.y)));
  const float2 t = x_mul(w, d);
  Xk = make_float2(__fadd_rn(ex, t.y), __fsub_rn(ey, t.x));
  Xm = make_float2(__fsub_rn(ex, t.y), -__fadd_rn(ey, t.x));
}
// Mirror step: a = A[k], b = A[M - k] -> Z'[k], Z'[M - k], scaled by inv_n (a power of two).
__device__ __forceinline__ void x_pre(float2 a, float2 b, float2 w, float inv_n, float2& zk, float2& zm) {
  const float ex = __fadd_rn(a.x, b.x), ey = __fsub_rn(a.y, b.y);
  const float2 o = x_mulc(make_float2(__fsub_rn(a.x, b.x), __fadd_rn(a.y, b.y)), w);
  zk = make_float2(__fmul_rn(__fsub_rn(ex, o.y), inv_n), __fmul_rn(__fadd_rn(ey, o.x), inv_n));
  zm = make_float2(__fmul_rn(__fadd_rn(ex, o.y), inv_n), __fmul_rn(__fsub_rn(o.x, ey), inv_n));
}
// Packed bin 0 and bin M / 2 (W = -i): the pair k = 0 of the loops below.
__device__ __forceinline__ float2 x_post_dc(float2 z) {
  return make_float2(__fadd_rn(z.x, z.y), __fsub_rn(z.x, z.y));
}
__device__ __forceinline__ float2 x_pre_dc(float2 a, float inv_n) {
  return make_float2(__fmul_rn(__fadd_rn(a.x, a.y), inv_n), __fmul_rn(__fsub_rn(a.x, a.y), inv_n));
}
__device__ __forceinline__ float2 x_post_mid(float2 z) { return make_float2(z.x, -z.y); }
__device__ __forceinline__ float2 x_pre_mid(float2 a, float inv_n) {
  const float s = __fmul_rn(2.0f, inv_n);
  return make_float2(__fmul_rn(a.x, s), -__fmul_rn(a.y, s));
}

// Transforms side by side in a CTA: G groups of T threads.
template <int LOG2M>
struct RegGroups {
  using F = RegFft<LOG2M>;
  static constexpr int G = F::T >= 256 ? 1 : 256 / F::T;
  static constexpr int THREADS = G * F::T;
  static constexpr bool PP = LOG2M <= 12;    // two exchange buffers (larger: one)
  static constexpr bool WREG = F::E == 8;    // all twiddles in registers
  static constexpr int SMEM = G * (PP ? 2 : 1) * F::PM * (int)sizeof(float2);
};

// Barrier of the T threads of one group: a warp or part of one, a named barrier
// of whole warps, or the whole CTA.
template <int T, int G>
__device__ __forceinline__ void group_sync() {
  if constexpr (T < 32) {
    const unsigned lane = threadIdx.x & 31u;
    __syncwarp(((1u << T) - 1u) << (lane / T * T));
  } else if constexpr (T == 32) {
    __syncwarp();
  } else if constexpr (G > 1) {
    asm volatile("bar.sync %0, %1;" ::"r"((int)threadIdx.x / T + 1), "n"(T) : "memory");
  } else {
    __syncthreads();
  }
}

// Register that holds the lower bin of pair p after the last pass.
template <int LOG2M>
__device__ __forceinline__ constexpr int reg_pair(int p) {
  constexpr int RL = RegFft<LOG2M>::RL;
  return p / (RL / 2) * RL + p % (RL / 2);
}

}  // namespace tanb
