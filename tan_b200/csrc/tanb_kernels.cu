// sm_100a kernels of the uniformly-partitioned overlap-save convolution.
//
//   ir_spectrum_kernel  R2C of the IR partitions [h_i, 0^B], one per group of
//                       threads (tanb_fft_reg.cuh)
//   head_kernel         one CTA per channel: R2C of [x_{k-1}, x_k] into the
//                       delay line, MAC with partitions 0 and 1, add the
//                       precomputed tail, C2R, output the upper B samples
//                       (crossfading old and new IR on a swap block)
//   tail_kernel         streaming MAC over partitions 2..P-1 for the next block
//                       (the HBM-bound kernel): float4 loads of the IR spectrum
//                       and the delay line, partitions split across warps and
//                       reduced in shared memory in a fixed order
//   run_*_kernel        the same for a call over several blocks at once
//
// The reference computes the same sums on the CPU with an overlap-add form
// (tan/tanlibrary/src/TrueAudioNext/convolution/ConvolutionImpl.cpp:2380-2643);
// overlap-save needs no overlap buffer and gives the exact new-IR output on a
// swap block from the same delay line.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>
#include <utility>
#include <vector>

#include "tanb_fft_reg.cuh"
#include "tanb_internal.h"

namespace tanb {
namespace {

// Programmatic dependent launch (sm_90+): a kernel launched with
// cudaLaunchAttributeProgrammaticStreamSerialization may begin once every CTA
// of the kernel before it in the stream has executed launch_dependents (or
// exited). The head triggers at once; the tail launched behind it shares no
// data with it, so it never has to wait for the head grid. Without the
// attribute this is a no-op.
__device__ __forceinline__ void griddep_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Preferred shared-memory / L1 split (percent of the maximum shared memory)
// of a block's head and tail launches. Both carry the same value: an SM whose
// split has been set for one kernel cannot take CTAs of a kernel that asks
// for another split until it drains, and with the head's dynamic shared
// memory and the tail's small static buffers the driver's own choices differ
// (measured: the tail behind a head with 16 KB of dynamic shared memory ended
// 4 us later than the tail alone; with equal preferences, at the same time).
// 50% holds a head of up to 64 KB beside the tail's CTAs; the 128 KB head of
// 8192-sample blocks takes all of it. A kernel that needs more shared memory
// than its preference gets more regardless.
int pair_carveout(int log2B) { return log2B >= 13 ? 100 : 50; }

// Launch of `kernel`, with programmatic stream serialization when `pdl` is set
// and a preferred shared-memory split when `carveout` >= 0.
template <class... KArgs, class... Args>
cudaError_t launch_k(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, bool pdl,
                     int carveout, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (pdl) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  if (carveout >= 0) {
    attr[n].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attr[n].val.sharedMemCarveout = (unsigned)carveout;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// Descriptor sources for the head and tail kernels.
struct DevDesc {
  const ChanCtl* ctl;
  const float* const* in;
  float* const* out;
  __device__ __forceinline__ ChanCtl get_ctl(int c) const { return ctl[c]; }
  __device__ __forceinline__ const float* get_in(int c) const { return in[c]; }
  __device__ __forceinline__ float* get_out(int c) const { return out[c]; }
};
__device__ __forceinline__ ChanCtl unpack_ctl(uint8_t b) {
  return ChanCtl{(b & kCtlRun) ? 1 : 0, (b & kCtlSwap) ? 1 : 0, (b & kCtlSlotCur) ? 1 : 0, (b & kCtlSlotNew) ? 1 : 0};
}
struct ParDesc {
  ParamDesc p;
  __device__ __forceinline__ ChanCtl get_ctl(int c) const { return unpack_ctl(p.c.ctl[c]); }
  __device__ __forceinline__ const float* get_in(int c) const { return p.in[c]; }
  __device__ __forceinline__ float* get_out(int c) const { return p.out[c]; }
};
struct StgDesc {
  StageDesc p;
  __device__ __forceinline__ ChanCtl get_ctl(int c) const { return unpack_ctl(p.c.ctl[c]); }
  __device__ __forceinline__ const float* get_in(int c) const {
    return (p.c.ctl[c] & kCtlHasIn) ? p.in + c * p.stride : nullptr;
  }
  __device__ __forceinline__ float* get_out(int c) const { return p.out + c * p.ostride; }
};
// Channel states only (the tail reads no rows).
struct CtlDesc {
  CtlParam p;
  __device__ __forceinline__ ChanCtl get_ctl(int c) const { return unpack_ctl(p.ctl[c]); }
};


// R2C of each IR partition: z[n] = (h[t0 + 2n], h[t0 + 2n + 1]) for n < M / 2,
// zero above, through register passes (tanb_fft_reg.cuh). THREADS / T transforms
// run side by side in a CTA and each group of T threads takes several partitions
// of its channel in turn, so that the stage twiddles are loaded into registers
// once and the next partition's samples while the present one is transformed.
// The kernel is bound by the shared-memory pipe and the barriers rather than by
// the 12 bytes a sample it moves: with one partition per group, twiddles in
// shared memory and CTA-wide barriers it took 22 us for 8192 partitions of 512
// (50 MB).
template <int LOG2M>
__global__ void __launch_bounds__(RegGroups<LOG2M>::THREADS)
    ir_spectrum_kernel(DevState s, IrRows ir, const int* __restrict__ chans, const ChanCtl* __restrict__ ctl) {
  using Sh = RegGroups<LOG2M>;
  using F = RegFft<LOG2M>;
  constexpr int M = F::M, T = F::T, E = F::E, G = Sh::G, RL = F::RL, NPAIR = E / 2;
  extern __shared__ __align__(16) float2 sm[];
  auto sync = [] { group_sync<T, G>(); };
  const int grp = (int)threadIdx.x / T, t = (int)threadIdx.x % T;
  float2* buf0 = sm + (Sh::PP ? 2 : 1) * grp * F::PM;
  float2* buf1 = Sh::PP ? buf0 + F::PM : buf0;
  const int row = blockIdx.y;
  const int c = chans[row];
  const int slot = ctl[c].slot_new;
  const float* h = ir.ptrs ? ir.ptrs[row] : ir.base + (size_t)row * ir.stride;
  const float2* tw = s.tw;
  float2 w[Sh::WREG ? F::TWT : 1];
  if constexpr (Sh::WREG) {
    reg_twiddles<LOG2M, 1>(w, tw, t);
    if constexpr (F::NP > 2) reg_twiddles<LOG2M, 2>(w + F::tw_base(2), tw, t);
  }
  float2 wp[NPAIR];
#pragma unroll
  for (int p = 0; p < NPAIR; ++p) wp[p] = tw[reg_out_index<LOG2M>(t, p / (RL / 2) * RL + p % (RL / 2))];
  const bool h8 = (reinterpret_cast<uintptr_t>(h) & 7) == 0;  // sample pairs load as one float2
  // inputs below M / 2 of partition `part` (the rest of the frame is zero)
  auto load = [&](int part, float2 (&x)[NPAIR]) {
#pragma unroll
    for (int p = 0; p < NPAIR; ++p) {
      const int n = reg_in_index<LOG2M>(t, p / (F::R0 / 2) * F::R0 + p % (F::R0 / 2));
      const long long at = (long long)part * M + 2 * n;
      x[p] = make_float2(0.f, 0.f);
      if (h8 && at + 1 < ir.n) {
        x[p] = __ldg(reinterpret_cast<const float2*>(h + at));
      } else {
        if (at < ir.n) x[p].x = h[at];
        if (at + 1 < ir.n) x[p].y = h[at + 1];
      }
    }
  };
  int part = blockIdx.x * G + grp;
  const int step = gridDim.x * G;
  float2 x[NPAIR];
  if (part < s.P) load(part, x);
  for (; part < s.P; part += step) {
    float2 v[E];
#pragma unroll
    for (int i = 0; i < E; ++i)
      v[i] = (i % F::R0 < F::R0 / 2) ? x[i / F::R0 * (F::R0 / 2) + i % F::R0] : make_float2(0.f, 0.f);
    if (part + step < s.P) load(part + step, x);
    reg_fft<LOG2M, false, Sh::WREG>(v, w, tw, buf0, buf1, t, sync);
    // the upper half meets the lower one of the bin pairs in the next buffer
    float2* pb = (F::NP & 1) ? buf0 : buf1;
#pragma unroll
    for (int i = 0; i < E; ++i)
      if (i % RL >= RL / 2) pb[F::pad(reg_out_index<LOG2M>(t, i))] = v[i];
    sync();
    float2* H = s.H + h_index(s, c, slot, part);
#pragma unroll
    for (int p = 0; p < NPAIR; ++p) {
      const int i = p / (RL / 2) * RL + p % (RL / 2);
      const int k = reg_out_index<LOG2M>(t, i);
      const float2 b = pb[F::pad(k == 0 ? M / 2 : M - k)];
      if (k == 0) {
        H[0] = x_post_dc(v[i]);
        H[M / 2] = x_post_mid(b);
      } else {
        float2 Xk, Xm;
        x_post(v[i], b, wp[p], Xk, Xm);
        H[k] = Xk;
        H[M - k] = Xm;
      }
    }
    if constexpr (!Sh::PP) {
      sync();
    } else if constexpr ((F::NP & 1) != 0) {
      // an odd number of uses: the next partition starts with the other buffer
      float2* b = buf0;
      buf0 = buf1;
      buf1 = b;
    }
  }
}

// Swap-block output samples i and i + 1 (one packed pair): the new IR's output
// weighted by i / M, the old one's by (M - i) / M (ConvolutionImpl.cpp:1395-1407).
__device__ __forceinline__ float2 crossfade_pair(float2 o, float2 yn, int i, float step, int M) {
  const float a0 = step * (float)i, b0 = step * (float)(M - i);
  const float a1 = step * (float)(i + 1), b1 = step * (float)(M - i - 1);
  return make_float2(__fmaf_rn(yn.x, a0, __fmul_rn(o.x, b0)), __fmaf_rn(yn.y, a1, __fmul_rn(o.y, b1)));
}

// Fused PCM epilogue (MixEpi): the channel's output row is in epi.scratch; the
// last head CTA of the channel's group sums the group's rows and converts.
// The counter is an atomic taken once per CTA after a fence: no CTA waits.
template <int M, int T>
__device__ __forceinline__ void mix_epilogue(const MixEpi& epi, int c) {
  __shared__ int last;
  const int g = epi.chan_group[c];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned members = (unsigned)(epi.gstart[g + 1] - epi.gstart[g]);
    last = (atomicAdd(epi.count + g, 1u) == members - 1) ? 1 : 0;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  bool clip = false;
  for (int i = threadIdx.x; i < M; i += T) {
    float sum = 0.f;
    for (int j = epi.gstart[g]; j < epi.gstart[g + 1]; ++j)
      sum = __fadd_rn(sum, __ldcg(epi.scratch + (size_t)epi.gchan[j] * M + i));
    float f = __fmul_rn(sum, epi.out_scale);
    if (f > 32767.f) { f = 32767.f; clip = true; }
    if (f < -32768.f) { f = -32768.f; clip = true; }
    epi.out16[(size_t)g * M + i] = (int16_t)((f != f) ? 0 : __float2int_rz(f));
  }
  if (clip) atomicOr(epi.clip, 1);
  if (threadIdx.x == 0) epi.count[g] = 0u;  // every member has counted itself
}

// One block of one channel. Every global load of the prologue is issued before
// any of them is used, so the block waits for one memory round trip: the frame
// (caller rows may sit in pinned host memory, the longest latency), the
// twiddles, the tail, partitions 0 and 1 and X_{k-1}. The transforms run as
// register passes (tanb_fft_reg.cuh): a block of 512 meets seven barriers (one
// more where it signals the host), where radix-4 stages in shared memory met 24.
template <int LOG2M>
struct HeadShape {
  using F = RegFft<LOG2M>;
  static constexpr bool PP = LOG2M <= 11;    // two exchange buffers
  static constexpr bool WREG = LOG2M <= 12;  // all twiddles in registers
  static constexpr bool PRE = LOG2M <= 12;   // tail and H_0 prefetched (8192: 512 threads, 128 registers each)
  static constexpr int SMEM = (PP ? 3 : 2) * F::PM * (int)sizeof(float2);
};

template <int LOG2M, class D>
__device__ __forceinline__ void head_body(const DevState& s, const D& desc, int cur, int parity, const MixEpi& epi) {
  using F = RegFft<LOG2M>;
  using Sh = HeadShape<LOG2M>;
  constexpr int M = F::M, T = F::T, E = F::E, R0 = F::R0, RL = F::RL, NP = F::NP, NPAIR = E / 2;
  extern __shared__ __align__(16) float2 sm[];
  float2* bufs[2] = {sm, Sh::PP ? sm + F::PM : sm};
  float2* zb = sm + (Sh::PP ? 2 : 1) * F::PM;  // the new IR's bins on a swap block
  auto sync = [] { __syncthreads(); };
  const int t = threadIdx.x;
  const int c = blockIdx.x;
  const ChanCtl cc = desc.get_ctl(c);
  if (!cc.run) return;
  const bool swap = cc.swap != 0;
  const float* x = desc.get_in(c);
  float* y = desc.get_out(c);
  float* prev = s.prev + (size_t)c * M;
  const float2* h0 = s.H + h_index(s, c, cc.slot_cur, 0);
  const float2* h1 = s.H + h_index(s, c, cc.slot_new, 0);
  // tails of this block (partitions >= 2): the IR in use, by block parity, and
  // a pending IR's; partition 1 multiplies X_{k-1}, in the next delay-line slot
  const float2* t0 = s.tail + ((size_t)c * 3 + parity) * M;
  const float2* t1 = s.tail + ((size_t)c * 3 + 2) * M;
  const bool p1 = s.P > 1;
  const float2* xp = s.fdl + ((size_t)c * s.P + (cur + 1) % s.P) * M;

  // The new half of the frame, M / 2 complex pairs, goes through shared memory:
  // 16-byte loads when the caller's row allows (staging rows always do), half
  // the requests, which counts when the row is read over the host bus.
  const int16_t* x16 = epi.active ? reinterpret_cast<const int16_t*>(x) : nullptr;
  const bool x_v4 = !x16 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;  // also when x is null
  float2 xr[NPAIR];
  if (x_v4) {
#pragma unroll
    for (int e = 0; e < NPAIR / 2; ++e) {
      const float4 q = x ? reinterpret_cast<const float4*>(x)[t + e * T] : make_float4(0.f, 0.f, 0.f, 0.f);
      xr[2 * e] = make_float2(q.x, q.y);
      xr[2 * e + 1] = make_float2(q.z, q.w);
    }
  } else {
    const bool x_vec = (reinterpret_cast<uintptr_t>(x) & 7) == 0;
#pragma unroll
    for (int e = 0; e < NPAIR; ++e) {
      const int n = t + e * T;
      if (x16) xr[e] = make_float2(__fmul_rn((float)x16[2 * n], epi.in_scale), __fmul_rn((float)x16[2 * n + 1], epi.in_scale));
      else if (x_vec) xr[e] = reinterpret_cast<const float2*>(x)[n];
      else xr[e] = make_float2(x[2 * n], x[2 * n + 1]);
    }
  }
  // the old half where pass 0 takes it
  float2 v[E];
#pragma unroll
  for (int i = 0; i < E; ++i)
    if (i % R0 < R0 / 2) v[i] = reinterpret_cast<const float2*>(prev)[reg_in_index<LOG2M>(t, i)];
  const float2* tw = s.tw;
  float2 w[Sh::WREG ? F::TWT : 1];
  if constexpr (Sh::WREG) {
    reg_twiddles<LOG2M, 1>(w, tw, t);
    if constexpr (NP > 2) reg_twiddles<LOG2M, 2>(w + F::tw_base(2), tw, t);
  }
  // tail (with partition 1's product) and partition 0 of this thread's bin
  // pairs (k, M - k), k < M / 2, with bin M / 2 beside bin 0: they do not
  // depend on the transform
  auto pair_reg = [](int p) { return p / (RL / 2) * RL + p % (RL / 2); };
  auto tail_of = [&](const float2* tl, const float2* hp, int k, int km, float2& a, float2& b) {
    a = tl[k];
    b = tl[km];
    if (p1) {
      a = (k == 0) ? c_mac_dc(a, xp[0], hp[M]) : c_mac(a, xp[k], hp[M + k]);
      b = c_mac(b, xp[km], hp[M + km]);
    }
  };
  float2 pt[Sh::PRE ? NPAIR : 1][2], ph[Sh::PRE ? NPAIR : 1][2], wp[Sh::PRE ? NPAIR : 1];
  if constexpr (Sh::PRE) {
#pragma unroll
    for (int p = 0; p < NPAIR; ++p) {
      const int k = reg_out_index<LOG2M>(t, pair_reg(p)), km = (k == 0) ? M / 2 : M - k;
      tail_of(t0, h0, k, km, pt[p][0], pt[p][1]);
      ph[p][0] = h0[k];
      ph[p][1] = h0[km];
      wp[p] = tw[k];
    }
  }
  float2* xs = Sh::PP ? bufs[1] : zb;  // free until after the next barrier
  if (x_v4) {
#pragma unroll
    for (int e = 0; e < NPAIR / 2; ++e)
      reinterpret_cast<float4*>(xs)[t + e * T] = make_float4(xr[2 * e].x, xr[2 * e].y, xr[2 * e + 1].x, xr[2 * e + 1].y);
  } else {
#pragma unroll
    for (int e = 0; e < NPAIR; ++e) xs[t + e * T] = xr[e];
  }
  sync();  // also: every thread has read its part of prev
#pragma unroll
  for (int e = 0; e < NPAIR / 2; ++e)
    reinterpret_cast<float4*>(prev)[t + e * T] = reinterpret_cast<const float4*>(xs)[t + e * T];
#pragma unroll
  for (int i = 0; i < E; ++i)
    if (i % R0 >= R0 / 2) v[i] = xs[reg_in_index<LOG2M>(t, i) - M / 2];

  reg_fft<LOG2M, false, Sh::WREG>(v, w, tw, bufs[0], bufs[1], t, sync);

  // the upper half of the bins through shared memory to the threads that hold
  // their partners, and the products' upper halves back the same way
  float2* F0 = s.fdl + ((size_t)c * s.P + cur) * M;
  const float inv_n = 1.0f / (float)(2 * M);
  float2* pb = bufs[(NP - 1) & 1];
#pragma unroll
  for (int i = 0; i < E; ++i)
    if (i % RL >= RL / 2) pb[F::pad(reg_out_index<LOG2M>(t, i))] = v[i];
  sync();
#pragma unroll
  for (int p = 0; p < NPAIR; ++p) {
    const int i = pair_reg(p);
    const int k = reg_out_index<LOG2M>(t, i), km = (k == 0) ? M / 2 : M - k;
    const float2 b = pb[F::pad(km)];
    float2 tk, tm, hk, hm, wk;
    if constexpr (Sh::PRE) {
      tk = pt[p][0]; tm = pt[p][1]; hk = ph[p][0]; hm = ph[p][1]; wk = wp[p];
    } else {
      tail_of(t0, h0, k, km, tk, tm);
      hk = h0[k]; hm = h0[km]; wk = tw[k];
    }
    float2 Xk, Xm, zk, zm;
    if (k == 0) {
      Xk = x_post_dc(v[i]);
      Xm = x_post_mid(b);
      zk = x_pre_dc(c_mac_dc(tk, Xk, hk), inv_n);
      zm = x_pre_mid(c_mac(tm, Xm, hm), inv_n);
    } else {
      x_post(v[i], b, wk, Xk, Xm);
      x_pre(c_mac(tk, Xk, hk), c_mac(tm, Xm, hm), wk, inv_n, zk, zm);
    }
    F0[k] = Xk;
    F0[km] = Xm;
    if constexpr (F::SYM) v[i] = zk;
    else pb[F::pad(k)] = zk;
    pb[F::pad(km)] = zm;
    if (swap) {
      float2 uk, um;
      tail_of(t1, h1, k, km, uk, um);
      if (k == 0) {
        zk = x_pre_dc(c_mac_dc(uk, Xk, h1[0]), inv_n);
        zm = x_pre_mid(c_mac(um, Xm, h1[km]), inv_n);
      } else {
        x_pre(c_mac(uk, Xk, h1[k]), c_mac(um, Xm, h1[km]), wk, inv_n, zk, zm);
      }
      zb[F::pad(k)] = zk;
      zb[F::pad(km)] = zm;
    }
  }
  sync();
  if constexpr (F::SYM) {
#pragma unroll
    for (int i = 0; i < E; ++i)
      if (i % R0 >= R0 / 2) v[i] = pb[F::pad(reg_in_index<LOG2M>(t, i))];
  } else {
    reg_load<LOG2M, 0>(v, pb, t);
  }
  if constexpr (!Sh::PP) sync();
  reg_fft<LOG2M, true, Sh::WREG>(v, w, tw, bufs[NP & 1], bufs[(NP + 1) & 1], t, sync);

  // overlap-save: samples [B, 2B) of the circular result are the output
  const float step = 1.0f / (float)M;
  if (swap) {
    float2 o[E / 2];
#pragma unroll
    for (int p = 0; p < NPAIR; ++p) o[p] = v[pair_reg(p) + RL / 2];
    reg_load<LOG2M, 0>(v, zb, t);
    if constexpr (!Sh::PP) sync();
    reg_fft<LOG2M, true, Sh::WREG>(v, w, tw, bufs[1], bufs[0], t, sync);
#pragma unroll
    for (int p = 0; p < NPAIR; ++p) {
      const int i = pair_reg(p) + RL / 2;
      v[i] = crossfade_pair(o[p], v[i], 2 * (reg_out_index<LOG2M>(t, i) - M / 2), step, M);
    }
  }
  if (!y) return;
  const bool y_vec = (reinterpret_cast<uintptr_t>(y) & 7) == 0;
#pragma unroll
  for (int p = 0; p < NPAIR; ++p) {
    const int i = pair_reg(p) + RL / 2, n = reg_out_index<LOG2M>(t, i) - M / 2;
    if (y_vec) {
      reinterpret_cast<float2*>(y)[n] = v[i];
    } else {
      y[2 * n] = v[i].x;
      y[2 * n + 1] = v[i].y;
    }
  }
  if (epi.active) mix_epilogue<M, T>(epi, c);
}

// Completion signal of a launch of `total` CTAs (HeadSignal): every CTA, running
// or not, once its output stores are visible to the host.
__device__ __forceinline__ void signal_heads(const HeadSignal& sig, unsigned total) {
  if (sig.seq == 0) return;
  if (sig.each) {
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence_system();  // behind the barrier: the whole CTA's stores
      *reinterpret_cast<volatile long long*>(sig.flag + 1 + blockIdx.x) = sig.seq;
    }
    return;
  }
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(sig.count, 1u) == total - 1) {
    *sig.count = 0u;
    __threadfence_system();
    *reinterpret_cast<volatile long long*>(sig.flag) = sig.seq;
  }
}

template <int LOG2M, class D>
__global__ void __launch_bounds__(RegFft<LOG2M>::T)
    head_kernel(DevState s, const __grid_constant__ D desc, int cur, int parity, MixEpi epi, HeadSignal sig) {
  // The tail launched behind this kernel (the next block's partitions >= 2)
  // shares no data with it and may start at once.
  griddep_launch_dependents();
  head_body<LOG2M>(s, desc, cur, parity, epi);
  signal_heads(sig, gridDim.x);
}

// One float4 = two packed bins. u == 0 holds the packed (DC, Nyquist) pair.
__device__ __forceinline__ float4 mac4(float4 acc, float4 f, float4 h, bool dc) {
  float2 lo = dc ? c_mac_dc(make_float2(acc.x, acc.y), make_float2(f.x, f.y), make_float2(h.x, h.y))
                 : c_mac(make_float2(acc.x, acc.y), make_float2(f.x, f.y), make_float2(h.x, h.y));
  float2 hi = c_mac(make_float2(acc.z, acc.w), make_float2(f.z, f.w), make_float2(h.z, h.w));
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}

template <int UX, int SY, int D, class DS>
__global__ void __launch_bounds__(UX* SY)
    tail_kernel(DevState s, const __grid_constant__ DS desc, int which, int cur, int trow) {
  const int c = blockIdx.y;
  const ChanCtl cc = desc.get_ctl(c);
  if (which == 0 ? !cc.run : !cc.swap) return;
  const int slot = (which == 0) ? (cc.swap ? cc.slot_new : cc.slot_cur) : cc.slot_new;
  const int U = s.B >> 1;  // float4 units per partition
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int u = blockIdx.x * UX + tx;
  const int P = s.P;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  const bool act = u < U && P > 2;
  const float4* Hc = reinterpret_cast<const float4*>(s.H + h_index(s, c, slot, 0)) + u;
  const float4* Fc = reinterpret_cast<const float4*>(s.fdl + (size_t)c * P * s.B) + u;
  const bool dc = (u == 0);
  if (act) {
    const int nparts = P - 2;  // partitions 2 .. P-1
    const int chunk = (nparts + SY - 1) / SY;
    const int i0 = 2 + ty * chunk;
    const int i1 = min(P, i0 + chunk);
    int i = i0;
    int fs = (cur + i - 1) % P;
    for (; i + D <= i1; i += D) {
      float4 h[D], f[D];
#pragma unroll
      for (int q = 0; q < D; ++q) {
        h[q] = __ldg(Hc + (size_t)(i + q) * U);
        f[q] = __ldg(Fc + (size_t)fs * U);
        fs = (fs + 1 == P) ? 0 : fs + 1;
      }
#pragma unroll
      for (int q = 0; q < D; ++q) acc = mac4(acc, f[q], h[q], dc);
    }
    for (; i < i1; ++i) {
      const float4 h = __ldg(Hc + (size_t)i * U);
      const float4 f = __ldg(Fc + (size_t)fs * U);
      fs = (fs + 1 == P) ? 0 : fs + 1;
      acc = mac4(acc, f, h, dc);
    }
  }
  if constexpr (SY > 1) {
    __shared__ float4 red[SY][UX];
    red[ty][tx] = acc;
    __syncthreads();
    if (ty != 0) return;
#pragma unroll
    for (int q = 1; q < SY; ++q) {
      const float4 r = red[q][tx];
      acc.x += r.x;
      acc.y += r.y;
      acc.z += r.z;
      acc.w += r.w;
    }
  }
  if (u < U) reinterpret_cast<float4*>(s.tail + ((size_t)c * 3 + trow) * s.B)[u] = acc;
}

// ---------------------------------------------------------------------------
// Several blocks in one call. With nb blocks in hand the sum
//   Y_b = sum_i X_{b - i} H_i,  b = 0 .. nb - 1
// reads each spectrum once per group of output blocks instead of once per
// block, so the call is bound by its transforms and its products and no longer
// by the IR spectra and the delay line (67 MB per block at 64 channels of 65536
// taps: 10.2 us a block in the one-block form, head and tail). Three launches:
//   run_forward_kernel  every new spectrum X_b, b < nb, into the workspace
//   run_mac_kernel      Y_b for every b, and the tail of block nb for the call
//                       after this one
//   run_inverse_kernel  the outputs, and the last P new spectra into the delay
//                       line
// The sums are formed in the order of tail_kernel and head_kernel (partitions
// 2 .. P-1 in the tiling's chunks, the chunks in order, then partition 1, then
// 0) and the transforms are the same register passes, so a call over several
// blocks gives the bits of the one-block calls.

// Threads of the transforms: as for the IR transforms, runs of consecutive blocks per group.
template <int LOG2M, class D>
__global__ void __launch_bounds__(RegGroups<LOG2M>::THREADS)
    run_forward_kernel(DevState s, const __grid_constant__ D desc, float2* __restrict__ X, int nb, int run) {
  using Sh = RegGroups<LOG2M>;
  using F = RegFft<LOG2M>;
  constexpr int M = F::M, T = F::T, E = F::E, G = Sh::G, R0 = F::R0, RL = F::RL, NPAIR = E / 2;
  extern __shared__ __align__(16) float2 sm[];
  auto sync = [] { group_sync<T, G>(); };
  const int grp = (int)threadIdx.x / T, t = (int)threadIdx.x % T;
  float2* buf0 = sm + (Sh::PP ? 2 : 1) * grp * F::PM;
  float2* buf1 = Sh::PP ? buf0 + F::PM : buf0;
  const int c = blockIdx.y;
  const float* x = desc.get_in(c);
  const float2* tw = s.tw;
  const int r0 = ((int)blockIdx.x * G + grp) * run, r1 = min(nb, r0 + run);
  if (r0 >= nb) return;
  float2 w[Sh::WREG ? F::TWT : 1];
  if constexpr (Sh::WREG) {
    reg_twiddles<LOG2M, 1>(w, tw, t);
    if constexpr (F::NP > 2) reg_twiddles<LOG2M, 2>(w + F::tw_base(2), tw, t);
  }
  const bool x8 = (reinterpret_cast<uintptr_t>(x) & 7) == 0;
  // samples of block r where pass 0 takes a frame's halves: the same thread
  // reads block r as the new half of frame r and the old half of frame r + 1
  auto load = [&](int r, float2 (&q)[NPAIR]) {
    const float* src = r < 0 ? s.prev + (size_t)c * M : x + (size_t)r * M;
#pragma unroll
    for (int p = 0; p < NPAIR; ++p) {
      const int n = reg_in_index<LOG2M>(t, p / (R0 / 2) * R0 + p % (R0 / 2));
      if (r >= 0 && !x) q[p] = make_float2(0.f, 0.f);
      else if (x8 || r < 0) q[p] = reinterpret_cast<const float2*>(src)[n];
      else q[p] = make_float2(src[2 * n], src[2 * n + 1]);
    }
  };
  float2 lo[NPAIR], hi[NPAIR];
  load(r0 - 1, lo);
  load(r0, hi);
  for (int r = r0; r < r1; ++r) {
    float2 v[E];
#pragma unroll
    for (int i = 0; i < E; ++i) {
      const int p = i / R0 * (R0 / 2) + i % (R0 / 2);
      v[i] = (i % R0 < R0 / 2) ? lo[p] : hi[p];
    }
#pragma unroll
    for (int p = 0; p < NPAIR; ++p) lo[p] = hi[p];
    if (r + 1 < r1) load(r + 1, hi);
    reg_fft<LOG2M, false, Sh::WREG>(v, w, tw, buf0, buf1, t, sync);
    float2* pb = (F::NP & 1) ? buf0 : buf1;
#pragma unroll
    for (int i = 0; i < E; ++i)
      if (i % RL >= RL / 2) pb[F::pad(reg_out_index<LOG2M>(t, i))] = v[i];
    sync();
    float2* Xr = X + ((size_t)c * nb + r) * M;
#pragma unroll
    for (int p = 0; p < NPAIR; ++p) {
      const int i = p / (RL / 2) * RL + p % (RL / 2);
      const int k = reg_out_index<LOG2M>(t, i), km = (k == 0) ? M / 2 : M - k;
      const float2 b = pb[F::pad(km)];
      float2 Xk, Xm;
      if (k == 0) {
        Xk = x_post_dc(v[i]);
        Xm = x_post_mid(b);
      } else {
        x_post(v[i], b, tw[k], Xk, Xm);
      }
      Xr[k] = Xk;
      Xr[km] = Xm;
    }
    if constexpr (!Sh::PP) {
      sync();
    } else if constexpr ((F::NP & 1) != 0) {
      float2* b = buf0;
      buf0 = buf1;
      buf1 = b;
    }
  }
}

template <int LOG2M, class D>
__global__ void __launch_bounds__(RegGroups<LOG2M>::THREADS)
    run_inverse_kernel(DevState s, const __grid_constant__ D desc, const float2* __restrict__ X,
                       const float2* __restrict__ Y, int nb, int run, int cur, HeadSignal sig) {
  using Sh = RegGroups<LOG2M>;
  using F = RegFft<LOG2M>;
  constexpr int M = F::M, T = F::T, E = F::E, G = Sh::G, RL = F::RL, NPAIR = E / 2;
  extern __shared__ __align__(16) float2 sm[];
  auto sync = [] { group_sync<T, G>(); };
  const int grp = (int)threadIdx.x / T, t = (int)threadIdx.x % T;
  float2* buf0 = sm + (Sh::PP ? 2 : 1) * grp * F::PM;
  float2* buf1 = Sh::PP ? buf0 + F::PM : buf0;
  const int c = blockIdx.y;
  float* y = desc.get_out(c);
  const bool y8 = (reinterpret_cast<uintptr_t>(y) & 7) == 0;
  const float2* tw = s.tw;
  const int r0 = ((int)blockIdx.x * G + grp) * run, r1 = min(nb, r0 + run);
  const float inv_n = 1.0f / (float)(2 * M);
  if (r0 < nb) {
    float2 w[Sh::WREG ? F::TWT : 1];
    if constexpr (Sh::WREG) {
      reg_twiddles<LOG2M, 1>(w, tw, t);
      if constexpr (F::NP > 2) reg_twiddles<LOG2M, 2>(w + F::tw_base(2), tw, t);
    }
    for (int r = r0; r < r1; ++r) {
      const float2* A = Y + ((size_t)c * nb + r) * M;
      if (r >= nb - s.P) {  // X_r into the delay line (older ones are already overwritten by newer)
        const float4* src = reinterpret_cast<const float4*>(X + ((size_t)c * nb + r) * M);
        int slot = (cur - 1 - r) % s.P;
        if (slot < 0) slot += s.P;
        float4* dst = reinterpret_cast<float4*>(s.fdl + ((size_t)c * s.P + slot) * M);
#pragma unroll
        for (int e = 0; e < NPAIR; ++e) dst[t + e * T] = src[t + e * T];
      }
      if (!y) continue;  // the same for every thread of the group: a channel's output is read or not
      float2 v[E];
#pragma unroll
      for (int p = 0; p < NPAIR; ++p) {
        const int i = p / (RL / 2) * RL + p % (RL / 2);
        const int k = reg_out_index<LOG2M>(t, i), km = (k == 0) ? M / 2 : M - k;
        const float2 a = A[k], b = A[km];
        float2 zk, zm;
        if (k == 0) {
          zk = x_pre_dc(a, inv_n);
          zm = x_pre_mid(b, inv_n);
        } else {
          x_pre(a, b, tw[k], inv_n, zk, zm);
        }
        if constexpr (F::SYM) v[i] = zk;
        else buf0[F::pad(k)] = zk;
        buf0[F::pad(km)] = zm;
      }
      sync();
      if constexpr (F::SYM) {
#pragma unroll
        for (int i = 0; i < E; ++i)
          if (i % F::R0 >= F::R0 / 2) v[i] = buf0[F::pad(reg_in_index<LOG2M>(t, i))];
      } else {
        reg_load<LOG2M, 0>(v, buf0, t);
      }
      if constexpr (!Sh::PP) sync();
      reg_fft<LOG2M, true, Sh::WREG>(v, w, tw, buf1, buf0, t, sync);
      float* yr = y + (size_t)r * M;
#pragma unroll
      for (int p = 0; p < NPAIR; ++p) {
        const int i = p / (RL / 2) * RL + p % (RL / 2) + RL / 2, n = reg_out_index<LOG2M>(t, i) - M / 2;
        if (y8) {
          reinterpret_cast<float2*>(yr)[n] = v[i];
        } else {
          yr[2 * n] = v[i].x;
          yr[2 * n + 1] = v[i].y;
        }
      }
      if constexpr (Sh::PP && (F::NP & 1) != 0) {
        float2* b = buf0;
        buf0 = buf1;
        buf1 = b;
      }
    }
  }
  signal_heads(sig, gridDim.x * gridDim.y);
}

// Output blocks of one run_mac_kernel CTA at most, bins per CTA, partition
// chunks in flight and spectra each thread has in flight. A thread keeps NB sums
// of one bin and the NB input spectra that a partition meets, so one partition
// and one spectrum are loaded for NB products. The products (six
// FP32 operations each; packed FP32 pairs issue at half the rate of two scalar
// operations and made every form slower) are what bounds the kernel.
constexpr int kRunBlocks = 8, kRunBins = 32, kRunRows = 8, kRunAhead = 4;

template <bool DC>
__device__ __forceinline__ float2 run_mac(float2 acc, float2 x, float2 h, bool dc) {
  const float2 a = c_mac(acc, x, h);
  if constexpr (!DC) return a;
  const float2 b = c_mac_dc(acc, x, h);
  return dc ? b : a;
}

// The spectra X_r of descending r of one bin: new blocks r >= 0 in the
// workspace, older ones in the delay line (slot (cur + i) mod P holds X_{-1-i}).
struct SpecWalk {
  const float2* p;
  const float2* fdl;
  ptrdiff_t step;
  int left, slot, B, P;
  __device__ __forceinline__ SpecWalk(const float2* X, const float2* fdl_, int r, int cur, int B_, int P_)
      : fdl(fdl_), B(B_), P(P_) {
    slot = cur;
    if (r >= 0) {
      p = X + (size_t)r * B;
      step = -(ptrdiff_t)B;
      left = r + 1;
    } else {
      slot = cur - 1 - r;
      if (slot >= P) slot -= P;
      line();
    }
  }
  __device__ __forceinline__ void line() {
    p = fdl + (size_t)slot * B;
    step = B;
    left = P - slot;
    slot = 0;  // where the line goes on after its end
  }
  __device__ __forceinline__ float2 next() {
    const float2 v = *p;
    p += step;
    if (--left == 0) line();
    return v;
  }
};

// The products of one bin for output blocks b0 .. b0 + NB - 1, partition by
// partition: the inputs a partition meets are a window over the spectra, one
// more of which enters with each partition. Rounds of NB partitions turn the
// window through the registers with compile-time positions; what is left of a
// span moves it by hand. kRunAhead partitions' loads are in flight (past the
// last partition they repeat its row, or go round the delay line, unused).
template <int NB, bool DC>
struct MacSpan {
  static constexpr int A = kRunAhead;
  static_assert(NB % A == 0, "the load queue turns with the window");
  SpecWalk walk;
  const float2* h;
  int hleft;  // partitions after the one h points to
  float2 win[NB];  // win[m] = X_{b0 + NB - 1 - i - m}, i the next partition (m = NB - 1 enters with it)
  float2 hq[A], xq[A];
  float2 acc[NB];

  // starts at partition i0 of a row of P: X_r for r >= nb do not exist; the
  // outputs that would read them are not stored
  __device__ __forceinline__ MacSpan(const float2* H, const float2* fdl, const float2* X, int B, int P, int cur, int nb,
                                     int b0, int i0)
      : walk(X, fdl, min(nb - 1, b0 + NB - 1 - i0), cur, B, P), h(H + (size_t)i0 * B), hleft(P - 1 - i0) {
    const int skip = max(0, b0 + NB - 1 - i0 - (nb - 1));
#pragma unroll
    for (int m = 0; m < NB - 1; ++m) {
      win[m] = make_float2(0.f, 0.f);
      if (m >= skip) win[m] = walk.next();
    }
#pragma unroll
    for (int a = 0; a < A; ++a) fetch(a);
    clear();
  }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int b = 0; b < NB; ++b) acc[b] = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ void fetch(int a) {
    hq[a] = __ldg(h);
    xq[a] = walk.next();
    h += hleft > 0 ? walk.B : 0;
    --hleft;
  }
  // n more partitions into the sums
  __device__ __forceinline__ void run(int n, bool dc) {
    for (; n >= NB; n -= NB) {
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        const float2 hv = hq[u % A];
        win[(NB - 1 + u) % NB] = xq[u % A];
        fetch(u % A);
#pragma unroll
        for (int b = 0; b < NB; ++b) acc[b] = run_mac<DC>(acc[b], win[(NB - 1 - b + u) % NB], hv, dc);
      }
    }
#pragma unroll 1
    for (; n > 0; --n) {
      const float2 hv = hq[0];
      win[NB - 1] = xq[0];
#pragma unroll
      for (int a = 0; a + 1 < A; ++a) {
        hq[a] = hq[a + 1];
        xq[a] = xq[a + 1];
      }
      fetch(A - 1);
#pragma unroll
      for (int b = 0; b < NB; ++b) acc[b] = run_mac<DC>(acc[b], win[NB - 1 - b], hv, dc);
      const float2 first = win[0];
#pragma unroll
      for (int m = 0; m + 1 < NB; ++m) win[m] = win[m + 1];
      win[NB - 1] = first;
    }
  }
};

template <int NB, bool DC, class D>
__device__ __forceinline__ void run_mac_body(const DevState& s, const D& desc, const float2* __restrict__ X,
                                             float2* __restrict__ Y, int nb, int per, int sy, int cur, int trow,
                                             float2 (*red)[NB][kRunBins]) {
  constexpr int NO = (NB + kRunRows - 1) / kRunRows;  // outputs a row finishes
  const int c = blockIdx.y, tx = threadIdx.x, ty = threadIdx.y;
  const int u = blockIdx.x * kRunBins + tx;
  const int B = s.B, P = s.P;
  const int b0 = blockIdx.z * per, b1 = min(nb + 1, b0 + per);  // output nb: the next call's first tail
  const bool dc = (u == 0);
  const ChanCtl cc = desc.get_ctl(c);
  const float2* H = s.H + h_index(s, c, cc.slot_cur, 0) + u;
  const float2* fdl = s.fdl + (size_t)c * P * B + u;
  const float2* Xc = X + (size_t)c * nb * B + u;
  if (blockIdx.z == 0 && ty == 0) {
    // the last block's samples are the next call's history
    const float* x = desc.get_in(c);
    s.prev[(size_t)c * B + u] = x ? x[(size_t)(nb - 1) * B + u] : 0.f;
  }
  float2 tot[NO];
#pragma unroll
  for (int o = 0; o < NO; ++o) tot[o] = make_float2(0.f, 0.f);
  const int nparts = max(0, P - 2), chunk = (nparts + sy - 1) / sy;
  if (nparts > 0) {
    for (int q0 = 0; q0 < sy; q0 += kRunRows) {
      const int i0 = 2 + (q0 + ty) * chunk, i1 = min(P, i0 + chunk);
      if (q0) __syncthreads();
      if (i0 < i1) {
        MacSpan<NB, DC> span(H, fdl, Xc, B, P, cur, nb, b0, i0);
        span.run(i1 - i0, dc);
#pragma unroll
        for (int b = 0; b < NB; ++b) red[ty][b][tx] = span.acc[b];
      } else {
#pragma unroll
        for (int b = 0; b < NB; ++b) red[ty][b][tx] = make_float2(0.f, 0.f);
      }
      __syncthreads();
#pragma unroll
      for (int o = 0; o < NO; ++o) {
        const int b = ty + o * kRunRows;
        if (b < NB) {
          float2 a = red[0][b][tx];
          if (q0) a = make_float2(__fadd_rn(tot[o].x, a.x), __fadd_rn(tot[o].y, a.y));
#pragma unroll
          for (int q = 1; q < kRunRows; ++q) {
            const float2 r = red[q][b][tx];
            a = make_float2(__fadd_rn(a.x, r.x), __fadd_rn(a.y, r.y));
          }
          tot[o] = a;
        }
      }
    }
  }
#pragma unroll
  for (int o = 0; o < NO; ++o) {
    const int b = b0 + ty + o * kRunRows;
    if (ty + o * kRunRows >= NB || b >= b1) continue;
    if (b == nb) {
      if (nparts > 0) s.tail[((size_t)c * 3 + trow) * B + u] = tot[o];
      continue;
    }
    float2 a = tot[o];
    if (P > 1) {
      const float2 x = b > 0 ? Xc[(size_t)(b - 1) * B] : fdl[(size_t)cur * B];
      a = dc ? c_mac_dc(a, x, H[B]) : c_mac(a, x, H[B]);
    }
    const float2 x = Xc[(size_t)b * B];
    Y[((size_t)c * nb + b) * B + u] = dc ? c_mac_dc(a, x, H[0]) : c_mac(a, x, H[0]);
  }
}

// The same sums for calls with enough work to fill the GPU: one warp takes all
// partitions of NB output blocks of 64 bins (two a thread), and the warps of a
// CTA are the output groups of the same bins, which share the rows they read.
// Rows reach shared memory by asynchronous copies of 16 bytes a thread, stages
// of kLineStage partitions, kLineDepth of them ahead: IR rows in a ring by
// partition, input rows in a ring by q = top - r, X_top the newest spectrum the
// CTA meets, so that group g's row for partition i is q = (G - 1 - g) NB + NB - 3
// + i. The inner loop is one copy of code for every bin, stage and chunk: the
// kernel runs for some twenty stages, and with the loop doubled for the packed
// bin 0 and for chunk ends it waited for instructions. At 64 channels of 128
// partitions of 512 and 32 blocks a launch takes 79 us alone: 512 CTAs of six warps
// are 0.86 of a wave at four per SM, and their dependent FP32 operations and the
// barriers between stages keep the issue slots 65% busy. (The width of six outputs
// spills 64 bytes a thread, 128 with device tables, at the 80 registers that allows.)
constexpr int kLineStage = 8, kLineDepth = 2, kLineGroups = 6, kLineBins = 64, kLineXRows = 64, kLineHRows = 32;

// acc + x h for two bins; (h0, nh0, g0, k0): of the first bin, h.x, -h.y and
// h.y, h.x, or for the packed bin 0 h.x, 0 and 0, h.y
__device__ __forceinline__ float4 line_mac(float4 acc, float4 x, float4 h, float nh0, float g0, float k0) {
  return make_float4(__fadd_rn(__fmaf_rn(x.x, h.x, __fmul_rn(x.y, nh0)), acc.x),
                     __fadd_rn(__fmaf_rn(x.x, g0, __fmul_rn(x.y, k0)), acc.y),
                     __fadd_rn(__fmaf_rn(x.z, h.z, -__fmul_rn(x.w, h.w)), acc.z),
                     __fadd_rn(__fmaf_rn(x.z, h.w, __fmul_rn(x.w, h.z)), acc.w));
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) {
  return make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z), __fadd_rn(a.w, b.w));
}

template <int NB, class D>
__global__ void __launch_bounds__(kLineGroups * 32, 4)
    run_mac_line_kernel(DevState s, const __grid_constant__ D desc, const float2* __restrict__ Xw,
                        float2* __restrict__ Y, int nb, int span, int sy, int cur, int trow) {
  // rows in use (the groups' offsets, a window behind, a stage) and in flight
  static_assert(kLineGroups * NB + (kLineDepth + 1) * kLineStage <= kLineXRows + 1, "input row ring");
  static_assert((kLineDepth + 1) * kLineStage <= kLineHRows, "IR row ring");
  __shared__ __align__(16) float4 xring[kLineXRows][32];
  __shared__ __align__(16) float4 hring[kLineHRows][32];
  const int c = blockIdx.y, lane = threadIdx.x & 31, grp = threadIdx.x >> 5, G = blockDim.x >> 5;
  const int B = s.B, P = s.P, ub = blockIdx.x * kLineBins, u0 = ub + 2 * lane;
  const int bs = blockIdx.z * span, be = min(nb + 1, bs + span);  // this CTA's outputs
  const int b0 = bs + grp * NB;
  const bool dc = u0 == 0;
  const ChanCtl cc = desc.get_ctl(c);
  const float2* H = s.H + h_index(s, c, cc.slot_cur, 0) + ub;
  const float2* fdl = s.fdl + (size_t)c * P * B + ub;
  const float2* X = Xw + (size_t)c * nb * B + ub;
  if (bs == 0 && grp == 0) {
    // the last block's samples are the next call's history
    const float* x = desc.get_in(c);
    float* prev = s.prev + (size_t)c * B + u0;
    prev[0] = x ? x[(size_t)(nb - 1) * B + u0] : 0.f;
    prev[1] = x ? x[(size_t)(nb - 1) * B + u0 + 1] : 0.f;
  }
  const int nparts = max(0, P - 2), chunk = (nparts + sy - 1) / sy;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 tot[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) tot[b] = zero;
  auto mac = [&](float4& acc, float4 x, float4 h) {
    acc = line_mac(acc, x, h, dc ? 0.f : -h.y, dc ? 0.f : h.y, dc ? h.y : h.x);
  };
  if (nparts > 0) {
    const int top = bs + G * NB - 3;
    auto copy16 = [](float4* dst, const float2* src) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                       static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
    };
    auto x_row = [&](int r) -> const float2* {
      r = min(r, nb - 1);  // newer ones are read by outputs that are not stored
      if (r >= 0) return X + (size_t)r * B;
      int slot = cur - 1 - max(r, -P);
      if (slot >= P) slot -= P;
      return fdl + (size_t)slot * B;
    };
    // partitions i0 .. i0 + kLineStage - 1 and the input rows that enter group
    // 0's window with them (past the last partition: its row again)
    auto issue = [&](int i0) {
      for (int v = threadIdx.x; v < kLineStage * 32; v += blockDim.x) {
        const int i = i0 + (v >> 5), at = v & 31;
        copy16(&hring[i & (kLineHRows - 1)][at], H + (size_t)min(i, P - 1) * B + 2 * at);
        copy16(&xring[(top - bs + i) & (kLineXRows - 1)][at], x_row(bs - i) + 2 * at);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int v = threadIdx.x; v < (G * NB - 1) * 32; v += blockDim.x) {  // the first windows
      const int q = v >> 5, at = v & 31;
      copy16(&xring[q & (kLineXRows - 1)][at], x_row(top - q) + 2 * at);
    }
#pragma unroll 1
    for (int d = 0; d < kLineDepth; ++d) issue(2 + d * kLineStage);
    float4 acc[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) acc[b] = zero;
    const int q0 = (G - 1 - grp) * NB + NB - 3;
    int flush = 2 + chunk;  // partition before which the running chunk ends
    int i = 2;
#pragma unroll 1
    for (int i0 = 2; i0 < P; i0 += kLineStage) {
      // a copy group per stage, in order: all but the newest one have landed
      asm volatile("cp.async.wait_group %0;" ::"n"(kLineDepth - 1) : "memory");
      __syncthreads();  // and everyone is done with the stage before this one
      issue(i0 + kLineDepth * kLineStage);
      const int i1 = min(P, i0 + kLineStage);
#pragma unroll 1
      while (i < i1) {
        const int n = min(i1, flush) - i;
        const int q = q0 + i, hs = i & (kLineHRows - 1);
        float4 win[NB];
#pragma unroll
        for (int m = 0; m < NB - 1; ++m) win[m] = xring[(q - (NB - 1) + m) & (kLineXRows - 1)][lane];
#pragma unroll
        for (int u = 0; u < kLineStage; ++u) {
          if (u >= n) break;
          const float4 h = hring[(hs + u) & (kLineHRows - 1)][lane];
          win[(NB - 1 + u) % NB] = xring[(q + u) & (kLineXRows - 1)][lane];
          const float nh0 = dc ? 0.f : -h.y, g0 = dc ? 0.f : h.y, k0 = dc ? h.y : h.x;
#pragma unroll
          for (int b = 0; b < NB; ++b) acc[b] = line_mac(acc[b], win[(NB - 1 - b + u) % NB], h, nh0, g0, k0);
        }
        i += n;
        if (i == flush || i == P) {
          flush += chunk;
#pragma unroll
          for (int b = 0; b < NB; ++b) {
            tot[b] = add4(tot[b], acc[b]);
            acc[b] = zero;
          }
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
#pragma unroll
  for (int j = 0; j < NB; ++j) {
    const int b = b0 + j;
    if (b >= be) continue;
    float4 a = tot[j];
    if (b == nb) {  // the next call's first tail
      if (nparts > 0) *reinterpret_cast<float4*>(s.tail + ((size_t)c * 3 + trow) * B + u0) = a;
      continue;
    }
    const float4* Hl = reinterpret_cast<const float4*>(H) + lane;
    if (P > 1) {
      const float2* xp = b > 0 ? X + (size_t)(b - 1) * B : fdl + (size_t)cur * B;
      mac(a, reinterpret_cast<const float4*>(xp)[lane], Hl[B / 2]);
    }
    mac(a, reinterpret_cast<const float4*>(X + (size_t)b * B)[lane], Hl[0]);
    *reinterpret_cast<float4*>(Y + ((size_t)c * nb + b) * B + u0) = a;
  }
}

template <int NB, class D>
__global__ void __launch_bounds__(kRunBins* kRunRows)
    run_mac_kernel(DevState s, const __grid_constant__ D desc, const float2* __restrict__ X, float2* __restrict__ Y,
                   int nb, int per, int sy, int cur, int trow) {
  __shared__ float2 red[kRunRows][NB][kRunBins];  // the chunks' sums
  if (blockIdx.x == 0) run_mac_body<NB, true>(s, desc, X, Y, nb, per, sy, cur, trow, red);
  else run_mac_body<NB, false>(s, desc, X, Y, nb, per, sy, cur, trow, red);
}

// ---------------------------------------------------------------------------
// Tail MAC with cp.async.bulk staging. One CTA per (channel, BR-bin slice):
// thread 0 streams, for each chunk of RS partitions, the IR-spectrum and
// delay-line row segments of the slice (BR x 8 bytes each, 16-byte aligned)
// into stage (chunk mod NS) of a shared-memory ring and arms that stage's
// mbarrier with the byte count; all BR/2 threads wait on the barrier, multiply
// and accumulate their two bins from shared memory, then release the stage to
// the next chunk. Up to NS x RS x BR x 16 bytes are in flight per CTA without
// holding them in registers. Waits are bounded: on timeout the kernel records
// kErrBulkWaitTimeout, waits (bounded) for its copies in flight and returns.
// Every copy lands in this CTA's own shared memory and reads this GPU's own memory.

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int limit) {
  for (int it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

template <int BR, int RS, int NS, class DS>
__global__ void __launch_bounds__(BR / 2)
    tail_bulk_kernel(DevState s, const __grid_constant__ DS desc, int which, int cur, int trow) {
  constexpr int U = BR / 2;                     // threads = float4 units of the slice
  constexpr uint32_t kRowBytes = BR * sizeof(float2);
  extern __shared__ __align__(128) unsigned char bulk_smem[];
  float4* hbuf = reinterpret_cast<float4*>(bulk_smem);             // [NS][RS][U]
  float4* fbuf = hbuf + NS * RS * U;                                // [NS][RS][U]
  uint64_t* bars = reinterpret_cast<uint64_t*>(fbuf + NS * RS * U);  // [NS]
  const int c = blockIdx.y;
  const ChanCtl cc = desc.get_ctl(c);
  if (which == 0 ? !cc.run : !cc.swap) return;
  const int slot = (which == 0) ? (cc.swap ? cc.slot_new : cc.slot_cur) : cc.slot_new;
  const int P = s.P;
  const int bin0 = blockIdx.x * BR;
  const int tid = threadIdx.x;
  const int nparts = P - 2;  // partitions 2 .. P-1
  const int nchunks = (nparts + RS - 1) / RS;
  const float2* Hrow = s.H + h_index(s, c, slot, 0) + bin0;  // + i * B for partition i
  const float2* Frow = s.fdl + (size_t)c * P * s.B + bin0;    // + slot * B

  auto issue = [&](int q) {  // chunk q -> stage q % NS (thread 0 only)
    const int st = q % NS;
    const int i0 = 2 + q * RS;
    const int rows = min(RS, P - i0);
    const uint32_t bar = smem_addr(&bars[st]);
    mbar_expect_tx(bar, 2u * rows * kRowBytes);
    for (int r = 0; r < rows; ++r) {
      const int i = i0 + r;
      const int fs = (cur + i - 1) % P;
      bulk_g2s(smem_addr(hbuf + (st * RS + r) * U), Hrow + (size_t)i * s.B, kRowBytes, bar);
      bulk_g2s(smem_addr(fbuf + (st * RS + r) * U), Frow + (size_t)fs * s.B, kRowBytes, bar);
    }
  };

  if (tid == 0) {
    for (int st = 0; st < NS; ++st) mbar_init(smem_addr(&bars[st]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (tid == 0)
    for (int q = 0; q < NS && q < nchunks; ++q) issue(q);

  const bool dc = (bin0 == 0 && tid == 0);
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  bool ok = true;
  int q = 0;
  for (; q < nchunks; ++q) {
    const int st = q % NS;
    const uint32_t parity = (uint32_t)(q / NS) & 1u;
    const bool landed = mbar_wait(smem_addr(&bars[st]), parity, s.wait_limit);
    if (__syncthreads_or(!landed)) {  // CTA-uniform decision
      ok = false;
      break;
    }
    const int rows = min(RS, P - (2 + q * RS));
    for (int r = 0; r < rows; ++r)
      acc = mac4(acc, fbuf[(st * RS + r) * U + tid], hbuf[(st * RS + r) * U + tid], dc);
    __syncthreads();  // every thread is done reading stage st
    if (tid == 0 && q + NS < nchunks) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      issue(q + NS);
    }
  }
  if (!ok) {
    // record the failure, then let copies already issued land before exiting
    if (tid == 0) {
      atomicExch(s.err, kErrBulkWaitTimeout);
      for (int r = q; r < nchunks && r < q + NS; ++r)
        mbar_wait(smem_addr(&bars[r % NS]), (uint32_t)(r / NS) & 1u, kBulkWaitLimit);
    }
    __syncthreads();
    return;
  }
  reinterpret_cast<float4*>(s.tail + ((size_t)c * 3 + trow) * s.B + bin0)[tid] = acc;
}

template <int BR, int RS, int NS>
constexpr int bulk_smem_bytes() {
  return 2 * NS * RS * BR * (int)sizeof(float2) + NS * 8;
}

template <int LOG2M, class D>
cudaError_t set_run_attrs() {
  cudaError_t e = cudaFuncSetAttribute(run_forward_kernel<LOG2M, D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       RegGroups<LOG2M>::SMEM);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(run_inverse_kernel<LOG2M, D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              RegGroups<LOG2M>::SMEM);
}

template <int LOG2M>
cudaError_t set_attrs() {
  constexpr int smem = HeadShape<LOG2M>::SMEM;
  cudaError_t e =
      cudaFuncSetAttribute(head_kernel<LOG2M, DevDesc>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(head_kernel<LOG2M, ParDesc>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(head_kernel<LOG2M, StgDesc>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(ir_spectrum_kernel<LOG2M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              RegGroups<LOG2M>::SMEM);
}

template <int LOG2M>
cudaError_t set_attrs_once() {
  static OncePerDevice once;
  return once.run([] { return set_attrs<LOG2M>(); });
}

// Partitions of an IR update that one group of threads takes in turn: enough to
// pay for loading the twiddles, few enough that every SM has several CTAs.
constexpr int kIrPartsPerGroup = 4;

template <int LOG2M>
cudaError_t launch_ir_t(const DevState& s, const IrRows& ir, const int* chans, int nch, const ChanCtl* ctl,
                        cudaStream_t st) {
  using R = RegGroups<LOG2M>;
  const long long groups = ((long long)s.P * nch + R::G - 1) / R::G;  // CTAs at one partition per group
  const int iters = (int)std::max<long long>(1, std::min<long long>(kIrPartsPerGroup, groups / (kSms * 2)));
  const int gx = (s.P + R::G * iters - 1) / (R::G * iters);
  ir_spectrum_kernel<LOG2M><<<dim3(gx, nch), R::THREADS, R::SMEM, st>>>(s, ir, chans, ctl);
  return cudaGetLastError();
}

template <int LOG2M>
cudaError_t launch_head_t(const DevState& s, const BlockRef& d, int cur, int parity, cudaStream_t st,
                          const MixEpi& epi, const HeadSignal& sig) {
  constexpr int T = RegFft<LOG2M>::T;
  constexpr size_t smem = HeadShape<LOG2M>::SMEM;
  const int cv = pair_carveout(LOG2M);
  if (d.stage)
    return launch_k(head_kernel<LOG2M, StgDesc>, dim3(s.C), dim3(T), smem, st, false, cv, s, StgDesc{*d.stage},
                    cur, parity, epi, sig);
  if (d.param)
    return launch_k(head_kernel<LOG2M, ParDesc>, dim3(s.C), dim3(T), smem, st, false, cv, s, ParDesc{*d.param},
                    cur, parity, epi, sig);
  return launch_k(head_kernel<LOG2M, DevDesc>, dim3(s.C), dim3(T), smem, st, false, cv, s,
                  DevDesc{d.ctl, d.in, d.out}, cur, parity, epi, sig);
}

// Consecutive blocks one group of threads transforms in turn: enough that
// twiddles and (for caller rows on the host bus) samples are read once, few
// enough that every SM has work.
constexpr int kRunMax = 8;

// Warps from which run_mac_line_kernel takes the sums. Its CTAs go through all
// partitions in series: a call of 12 blocks of 512 with 65536 taps takes 34 us with
// run_mac_kernel and 61 with it at one channel, 58 and 74 at 32 channels (512
// warps), 90 and 90 at 64 (1024 warps).
constexpr int kRunLineWarps = kSms * 6;

template <int LOG2M>
cudaError_t launch_run_t(const DevState& s, const BlockRef& d, const RunShape& r, cudaStream_t st,
                         const HeadSignal& sig) {
  using Sh = RegGroups<LOG2M>;
  const int run = (int)std::max<long long>(1, std::min<long long>(kRunMax, (long long)s.C * r.nb / ((long long)Sh::G * kSms * 2)));
  const dim3 gf((r.nb + Sh::G * run - 1) / (Sh::G * run), s.C);
  const int groups = (r.nb + 1 + kRunBlocks - 1) / kRunBlocks, per = (r.nb + 1 + groups - 1) / groups;
  const dim3 gm(s.B / kRunBins, s.C, groups), bm(kRunBins, kRunRows);
  auto go = [&](const auto& desc) {
    using D = std::decay_t<decltype(desc)>;
    static OncePerDevice once;
    cudaError_t e = once.run([] { return set_run_attrs<LOG2M, D>(); });
    if (e != cudaSuccess) return e;
    e = launch_k(run_forward_kernel<LOG2M, D>, gf, dim3(Sh::THREADS), Sh::SMEM, st, false, -1, s, desc, r.X,
                             r.nb, run);
    if (e != cudaSuccess) return e;
    if (s.B >= kLineBins && (long long)s.B / kLineBins * s.C * groups >= kRunLineWarps) {
      // outputs (and the next call's first tail) over CTAs of at most
      // kLineGroups groups of NB
      const int n = r.nb + 1, NB = n <= 4 ? 4 : 6;
      const int supers = (n + kLineGroups * NB - 1) / (kLineGroups * NB), span = ((n + supers - 1) / supers + NB - 1) / NB * NB;
      const dim3 gl(s.B / kLineBins, s.C, (n + span - 1) / span);
      auto line = [&](auto kernel) {
        return launch_k(kernel, gl, dim3(32 * span / NB), 0, st, false, -1, s, desc, r.X, r.Y, r.nb, span, r.sy, r.cur,
                        r.trow);
      };
      e = NB == 4 ? line(run_mac_line_kernel<4, D>) : line(run_mac_line_kernel<6, D>);
      if (e != cudaSuccess) return e;
      return launch_k(run_inverse_kernel<LOG2M, D>, gf, dim3(Sh::THREADS), Sh::SMEM, st, false, -1, s, desc, r.X, r.Y,
                      r.nb, run, r.cur, sig);
    }
    auto mac = [&](auto kernel) {
      return launch_k(kernel, gm, bm, 0, st, false, -1, s, desc, r.X, r.Y, r.nb, per, r.sy, r.cur, r.trow);
    };
    e = per <= 4 ? mac(run_mac_kernel<4, D>) : mac(run_mac_kernel<kRunBlocks, D>);
    if (e != cudaSuccess) return e;
    return launch_k(run_inverse_kernel<LOG2M, D>, gf, dim3(Sh::THREADS), Sh::SMEM, st, false, -1, s, desc, r.X, r.Y,
                    r.nb, run, r.cur, sig);
  };
  if (d.stage) return go(StgDesc{*d.stage});
  if (d.param) return go(ParDesc{*d.param});
  return go(DevDesc{d.ctl, d.in, d.out});
}

#define TANB_DISPATCH_LOG2(L2, FN, ...)                          \
  switch (L2) {                                                  \
    case 5: return FN<5>(__VA_ARGS__);                           \
    case 6: return FN<6>(__VA_ARGS__);                           \
    case 7: return FN<7>(__VA_ARGS__);                           \
    case 8: return FN<8>(__VA_ARGS__);                           \
    case 9: return FN<9>(__VA_ARGS__);                           \
    case 10: return FN<10>(__VA_ARGS__);                         \
    case 11: return FN<11>(__VA_ARGS__);                         \
    case 12: return FN<12>(__VA_ARGS__);                         \
    case 13: return FN<13>(__VA_ARGS__);                         \
    default: return cudaErrorInvalidValue;                       \
  }

template <int UX, int SY, int D>
cudaError_t launch_tail_t(const DevState& s, const BlockRef& d, int which, int cur, int trow, cudaStream_t st,
                          bool pdl) {
  const int U = s.B >> 1;
  dim3 grid((U + UX - 1) / UX, s.C);
  dim3 block(UX, SY);
  if (const CtlParam* cp = d.ctl_param())
    return launch_k(tail_kernel<UX, SY, D, CtlDesc>, grid, block, 0, st, pdl, pair_carveout(s.log2B), s,
                    CtlDesc{*cp}, which, cur, trow);
  return launch_k(tail_kernel<UX, SY, D, DevDesc>, grid, block, 0, st, pdl, pair_carveout(s.log2B), s,
                  DevDesc{d.ctl, d.in, d.out}, which,
                  cur, trow);
}

template <int BR, int RS, int NS>
cudaError_t launch_bulk_t(const DevState& s, const BlockRef& d, int which, int cur, int trow, cudaStream_t st,
                          bool pdl) {
  if (s.B % BR != 0) return cudaErrorInvalidValue;
  constexpr int smem = bulk_smem_bytes<BR, RS, NS>();
  static OncePerDevice once;
  const cudaError_t attr = once.run([] {
    cudaError_t e = cudaFuncSetAttribute(tail_bulk_kernel<BR, RS, NS, DevDesc>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(tail_bulk_kernel<BR, RS, NS, CtlDesc>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                smem);
  });
  if (attr != cudaSuccess) return attr;
  dim3 grid(s.B / BR, s.C);
  if (const CtlParam* cp = d.ctl_param())
    return launch_k(tail_bulk_kernel<BR, RS, NS, CtlDesc>, grid, dim3(BR / 2), smem, st, pdl, pair_carveout(s.log2B), s, CtlDesc{*cp},
                    which, cur, trow);
  return launch_k(tail_bulk_kernel<BR, RS, NS, DevDesc>, grid, dim3(BR / 2), smem, st, pdl, pair_carveout(s.log2B), s,
                  DevDesc{d.ctl, d.in, d.out}, which, cur, trow);
}

using TailLauncher = cudaError_t (*)(const DevState&, const BlockRef&, int, int, int, cudaStream_t, bool);
struct TailEntry {
  MacTiling t;
  TailLauncher fn;
};
// The tilings the autotuner chooses among.
const TailEntry kTail[] = {
    {{32, 8, 4}, launch_tail_t<32, 8, 4>},   {{16, 16, 4}, launch_tail_t<16, 16, 4>},
    {{32, 8, 8}, launch_tail_t<32, 8, 8>},   {{32, 16, 4}, launch_tail_t<32, 16, 4>},
    {{32, 16, 8}, launch_tail_t<32, 16, 8>}, {{64, 4, 4}, launch_tail_t<64, 4, 4>},
    {{64, 8, 4}, launch_tail_t<64, 8, 4>},   {{64, 8, 8}, launch_tail_t<64, 8, 8>},
    {{128, 2, 8}, launch_tail_t<128, 2, 8>}, {{32, 32, 4}, launch_tail_t<32, 32, 4>},
    {{16, 32, 8}, launch_tail_t<16, 32, 8>}, {{64, 16, 2}, launch_tail_t<64, 16, 2>},
    // cp.async.bulk pipelines: {BR/2, stages, rows per stage, kind 1}
    {{32, 4, 8, 1}, launch_bulk_t<64, 8, 4>},   {{64, 4, 8, 1}, launch_bulk_t<128, 8, 4>},
    {{64, 6, 4, 1}, launch_bulk_t<128, 4, 6>},  {{128, 4, 4, 1}, launch_bulk_t<256, 4, 4>},
    {{64, 8, 8, 1}, launch_bulk_t<128, 8, 8>},  {{128, 3, 8, 1}, launch_bulk_t<256, 8, 3>},
};
constexpr int kTailCount = sizeof(kTail) / sizeof(kTail[0]);

}  // namespace

cudaError_t prepare_kernels(int log2B) { TANB_DISPATCH_LOG2(log2B, set_attrs_once); }

cudaError_t launch_ir_spectrum(const DevState& s, const IrRows& ir, const int* chans, int nch,
                               const ChanCtl* ctl, cudaStream_t st) {
  if (nch <= 0) return cudaSuccess;
  TANB_DISPATCH_LOG2(s.log2B, launch_ir_t, s, ir, chans, nch, ctl, st);
}

cudaError_t launch_head(const DevState& s, const BlockRef& d, int cur, int parity, cudaStream_t st,
                        const MixEpi& epi, const HeadSignal& sig) {
  TANB_DISPATCH_LOG2(s.log2B, launch_head_t, s, d, cur, parity, st, epi, sig);
}

cudaError_t launch_tail(const DevState& s, const BlockRef& d, int which, int cur, int trow, MacTiling t,
                        cudaStream_t st, bool pdl) {
  if (s.P <= 2) return cudaSuccess;
  for (int i = 0; i < kTailCount; ++i)
    if (kTail[i].t.ux == t.ux && kTail[i].t.sy == t.sy && kTail[i].t.depth == t.depth &&
        kTail[i].t.kind == t.kind)
      return kTail[i].fn(s, d, which, cur, trow, st, pdl);
  return cudaErrorInvalidValue;
}

cudaError_t launch_run(const DevState& s, const BlockRef& d, const RunShape& r, cudaStream_t st,
                       const HeadSignal& sig) {
  TANB_DISPATCH_LOG2(s.log2B, launch_run_t, s, d, r, st, sig);
}

int mac_tiling_count() { return kTailCount; }

MacTiling mac_tiling(int index) { return kTail[index].t; }

void make_twiddles(int N, float2* out) {
  const int q4 = N / 4;
  for (int j = 0; j < N; ++j) {
    const int q = j / q4, r = j % q4;
    const double th = 2.0 * M_PI * (double)r / (double)N;
    const double c = std::cos(th), sn = std::sin(th);
    double cc, ss;  // cos and sin of 2 pi j / N
    switch (q) {
      case 0: cc = c; ss = sn; break;
      case 1: cc = -sn; ss = c; break;
      case 2: cc = -c; ss = -sn; break;
      default: cc = sn; ss = -c; break;
    }
    out[j] = make_float2((float)cc, (float)(-ss));
  }
}

void make_plan_twiddles(int log2M, float2* out) {
  const int M = 1 << log2M;
  std::vector<float2> w(2 * M);
  make_twiddles(2 * M, w.data());
  for (int i = 0; i < 2 * M; ++i) out[i] = w[plan_twiddle_index(log2M, i)];
}

}  // namespace tanb
