// TIME_DOMAIN method: direct FIR over a per-channel circular history, the GPU
// form of ProcessDirect / ovlTimeDomainCPU
// (tan/tanlibrary/src/TrueAudioNext/convolution/ConvolutionImpl.cpp:721-762,
// 2757-2782; the reference's OpenCL kernel is TimeDomainConvolution.cl:234-273,
// launched with one work-item per work-group).
//
//   out[c][j] = sum_{k=first}^{last-1} hist[c][(pos + j - k) mod len] * ir[c][k]
//
// with the call's n inputs already in the history at pos .. pos + n - 1 (mod
// len). One launch: a sample that this call writes is read from the caller's
// row, every other one from the history, so that no CTA waits for another's
// history stores. Where output rows overlap input rows the inputs enter the
// history in a launch of their own (td_insert_kernel), and every sample is then
// read from there.
//
// Taps are accumulated in increasing k with fused multiply-adds, the order of
// the reference's loop (another order differs from it by more than the 1e-5 of
// output RMS that it is held to: 1.7e-5 at 4096 taps). That makes one output a
// chain of dependent operations, four cycles a tap, which bounds calls of few
// outputs; four outputs a thread fill the chain's gaps. A warp takes 128 outputs,
// so that calls of a few thousand outputs still reach most schedulers (with 1024
// outputs per CTA, 32 CTAs took 116 us at 16 channels, 4096 taps and 2048
// samples, now 42). It keeps a chunk of taps and the samples they meet in shared
// memory and loads the next chunk's into registers meanwhile: per four taps one
// 16-byte load of taps and one of samples serve 16 products. Outputs leave through
// shared memory: written four to a thread straight into host rows they cross the
// bus four bytes at a time, 47.5 us where this takes 45. On a crossfade block a
// second IR is convolved and the two outputs blended with the reference's weights
// (ConvolutionImpl.cpp:1392-1408).
#include "tanb_internal.h"

namespace tanb {
namespace {

constexpr int kOut = 4;             // outputs per thread
constexpr int kTJ = 32 * kOut;      // outputs per warp
constexpr int kWarps = 4;           // per CTA, one for each scheduler of an SM
constexpr int kTK = 256;            // taps per chunk
constexpr int kRing = 512;          // samples in shared memory, a ring
constexpr int kPad = 16;
constexpr int kPer = kTK / 32;      // taps and samples each lane loads per chunk

// History index of offset o in [0, len) from pos in [0, len).
__device__ __forceinline__ int wrap(int pos, int o, int len) { return o >= len - pos ? o - (len - pos) : pos + o; }

struct TdSmem {
  // the sample at offset o - first from pos is in xs[kPad + o mod kRing]; the
  // pad repeats the ring's last slots
  float xs[kPad + kRing];
  float ws[kTK + 16];

  __device__ __forceinline__ void put(int o, float v) {
    const int i = o & (kRing - 1);
    xs[kPad + i] = v;
    if (i >= kRing - kPad) xs[i - (kRing - kPad)] = v;
  }
};

// Outputs j0 + 4 lane .. + 3 for one IR.
__device__ __forceinline__ void fir_tile(const float* __restrict__ h, int len, const TdChan& t,
                                         const float* __restrict__ ir, int n, int j0, TdSmem& sm, float (&acc)[kOut]) {
  const int lane = threadIdx.x & 31, taps = t.last - t.first;
  // the sample that output j0 + 4 l meets at tap first + kk, o = j0 + 4 l - kk
  auto sample = [&](int o) {
    o -= t.first;
    if (o >= n) return 0.f;  // outputs past the last one, not stored
    if (o < 0) o += len;     // o > -len: a tap's number is below len
    return (o < n && t.in) ? t.in[o] : h[wrap(t.pos, o, len)];
  };
#pragma unroll
  for (int q = 0; q < kOut; ++q) acc[q] = 0.f;
  float xr[kPer], wr[kPer];
  // taps [k0, k0 + kTK) and the oldest kTK samples they meet, in one run of the
  // caller's row or of the history where they lie so
  auto load = [&](int k0) {
    const int hi = j0 - k0 - t.first, lo = hi - (kTK - 1);  // offsets of the samples
    const float* src = nullptr;
    if (k0 + kTK <= taps) {
      if (lo >= 0 && hi < n && t.in) {
        src = t.in + hi;
      } else if (hi < 0 && lo + len >= n) {
        const int p = wrap(t.pos, hi + len, len);
        if (p >= kTK - 1) src = h + p;
      }
    }
    if (src) {
      const float* w = ir + t.first + k0 + lane;
      src -= lane;
#pragma unroll
      for (int e = 0; e < kPer; ++e) {
        wr[e] = w[32 * e];
        xr[e] = src[-32 * e];
      }
      return;
    }
#pragma unroll 1
    for (int e = 0; e < kPer; ++e) {
      const int k = lane + 32 * e;
      const float wk = (k0 + k < taps) ? ir[t.first + k0 + k] : 0.f;
      const float xk = (k0 + k < taps) ? sample(j0 - k0 - k) : 0.f;
#pragma unroll
      for (int q = 0; q < kPer; ++q) {
        wr[q] = q == e ? wk : wr[q];
        xr[q] = q == e ? xk : xr[q];
      }
    }
  };
  if (taps > 0) {
    load(0);
#pragma unroll
    for (int e = 0; e < kOut; ++e) {  // the samples ahead of the first chunk's oldest ones
      const int o = j0 + 1 + lane + 32 * e;
      if (o < j0 + kTJ) sm.put(o, sample(o));
    }
  }
  for (int k0 = 0; k0 < taps; k0 += kTK) {
    const int kn = min(kTK, taps - k0);
    __syncwarp();
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      const int k = lane + 32 * e;
      sm.ws[k] = wr[e];
      sm.put(j0 - k0 - k, xr[e]);
    }
    __syncwarp();
    if (k0 + kTK < taps) load(k0 + kTK);
    const int b = j0 + kOut * lane - k0;  // a multiple of four
    const float* xs = sm.xs + kPad;
    // four taps against the samples at b - kk .. + 3 (hi) and the four before (lo)
    auto four = [&](float4 hi, float4 lo, float4 w) {
      acc[0] = __fmaf_rn(hi.x, w.x, acc[0]);
      acc[1] = __fmaf_rn(hi.y, w.x, acc[1]);
      acc[2] = __fmaf_rn(hi.z, w.x, acc[2]);
      acc[3] = __fmaf_rn(hi.w, w.x, acc[3]);
      acc[0] = __fmaf_rn(lo.w, w.y, acc[0]);
      acc[1] = __fmaf_rn(hi.x, w.y, acc[1]);
      acc[2] = __fmaf_rn(hi.y, w.y, acc[2]);
      acc[3] = __fmaf_rn(hi.z, w.y, acc[3]);
      acc[0] = __fmaf_rn(lo.z, w.z, acc[0]);
      acc[1] = __fmaf_rn(lo.w, w.z, acc[1]);
      acc[2] = __fmaf_rn(hi.x, w.z, acc[2]);
      acc[3] = __fmaf_rn(hi.y, w.z, acc[3]);
      acc[0] = __fmaf_rn(lo.y, w.w, acc[0]);
      acc[1] = __fmaf_rn(lo.z, w.w, acc[1]);
      acc[2] = __fmaf_rn(lo.w, w.w, acc[2]);
      acc[3] = __fmaf_rn(hi.x, w.w, acc[3]);
    };
    // sixteen taps a step (hi: the samples at b - kk .. + 3), two steps' operands
    // in turn: the next step's are on their way while this one's are in use. Past
    // the chunk they come from slots that exist and are not used.
    float4 hi = *reinterpret_cast<const float4*>(xs + (b & (kRing - 1)));
    int kk = 0;
    if (kn >= 32) {
      float4 x0[4], w0[4], x1[4], w1[4];
      auto fetch = [&](int at, float4 (&x)[4], float4 (&w)[4]) {
        const float* xp = xs + ((b - at) & (kRing - 1));  // the pad below repeats the ring's top
        const float* wp = sm.ws + at;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          x[e] = *reinterpret_cast<const float4*>(xp - 4 * e - 4);
          w[e] = *reinterpret_cast<const float4*>(wp + 4 * e);
        }
      };
      auto sixteen = [&](const float4 (&x)[4], const float4 (&w)[4]) {
        four(hi, x[0], w[0]);
        four(x[0], x[1], w[1]);
        four(x[1], x[2], w[2]);
        four(x[2], x[3], w[3]);
        hi = x[3];
      };
      fetch(0, x0, w0);
#pragma unroll 1
      for (; kk + 32 <= kn; kk += 32) {
        fetch(kk + 16, x1, w1);
        sixteen(x0, w0);
        fetch(kk + 32, x0, w0);
        sixteen(x1, w1);
      }
    }
#pragma unroll 1
    for (; kk < kn; ++kk) {  // the last taps, fewer than 32
      const float w = sm.ws[kk];
#pragma unroll
      for (int q = 0; q < kOut; ++q) acc[q] = __fmaf_rn(xs[(b + q - kk) & (kRing - 1)], w, acc[q]);
    }
  }
}

// The n <= len samples of the rows from `at` on. `inserted`: the history already
// holds them.
__global__ void __launch_bounds__(32 * kWarps) td_fir_kernel(float* hist, int len, const TdChan* __restrict__ ch,
                                                             int C, int n, int at, int fade_len, int inserted) {
  __shared__ __align__(16) TdSmem sms[kWarps];
  // output tiles of all channels over the warps in turn
  const int tiles = (n + kTJ - 1) / kTJ, lane = threadIdx.x & 31;
  const long long id = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
  const int c = (int)(id / tiles), j0 = (int)(id % tiles) * kTJ;
  if (c >= C) return;
  TdSmem& sm = sms[threadIdx.x >> 5];
  TdChan t = ch[c];
  if (!t.run) return;
  t.in = (t.in && !inserted) ? t.in + at : nullptr;
  t.out = t.out ? t.out + at : nullptr;
  t.fade0 += at;
  float* h = hist + (size_t)c * len;
  float a[kOut], b[kOut];
  fir_tile(h, len, t, t.ir, n, j0, sm, a);
  if (t.swap) {
    __syncwarp();
    fir_tile(h, len, t, t.ir_new, n, j0, sm, b);
  }
  if (t.in)
    for (int j = j0 + lane; j < min(n, j0 + kTJ); j += 32) h[wrap(t.pos, j, len)] = t.in[j];
  if (!t.out) return;
  // outputs through shared memory, so that the row (which may be host memory
  // across the bus) is written in runs of 128 bytes
  const float step = 1.0f / (float)fade_len;
  __syncwarp();
#pragma unroll
  for (int q = 0; q < kOut; ++q) {
    const int j = j0 + lane * kOut + q;
    float o = t.swap ? b[q] : a[q];
    if (t.swap && t.fade0 + j < fade_len) {
      const float w1 = step * (float)(t.fade0 + j), w2 = step * (float)(fade_len - t.fade0 - j);
      o = b[q] * w1 + a[q] * w2;
    }
    sm.xs[lane * kOut + q] = o;
  }
  __syncwarp();
  for (int j = j0 + lane; j < min(n, j0 + kTJ); j += 32) t.out[j] = sm.xs[j - j0];
}

// hist[c][(pos + i) mod len] = in[c][at + i], i < n <= len.
__global__ void td_insert_kernel(float* hist, int len, const TdChan* __restrict__ ch, int n, int at) {
  const int c = blockIdx.y;
  const TdChan t = ch[c];
  if (!t.run || !t.in) return;
  float* h = hist + (size_t)c * len;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    h[wrap(t.pos, i, len)] = t.in[at + i];
}

}  // namespace

cudaError_t launch_td(float* hist, int len, const TdChan* ch, int C, int n, int fade_len, bool overlap,
                      cudaStream_t st) {
  // The history takes len samples at a time, after which its position is the same
  // again: a longer call (a block above the response's length rounded up) goes
  // through it in pieces, each with the samples and results of a call of its own.
  for (int at = 0; at < n; at += len) {
    const int m = n - at < len ? n - at : len;
    if (overlap) td_insert_kernel<<<dim3((m + 255) / 256, C), 256, 0, st>>>(hist, len, ch, m, at);
    const long long warps = (long long)C * ((m + kTJ - 1) / kTJ);
    td_fir_kernel<<<(unsigned)((warps + kWarps - 1) / kWarps), 32 * kWarps, 0, st>>>(hist, len, ch, C, m, at, fade_len,
                                                                                  overlap ? 1 : 0);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace tanb
