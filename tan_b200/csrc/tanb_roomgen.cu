// GPU-resident IR producer: the left / right impulse responses of a shoebox room
// written straight into device memory, for tanb_convolution_update_response_td_device
// (the GPU path of TrueAudioVR::generateRoomResponse with GENROOM_USE_GPU_MEM,
// samples/src/TrueAudioVR/TrueAudioVR.cpp:659-786; kernels
// Kernels/GenerateRoomResponse.cl:206-321 and Kernels/Fill.cl).
//
// Per image source (index i_x in [-n_W, n_W] along the width, etc., over the grid
// the reference launches: local size 4, so the last index exists only when 2 n_W
// is not a multiple of 4) and ear: an image at
// distance d lands at sample 1 + (int)(d / 340 * rate) with gain
// damp^walls x distance gain; early images (before the HRTF cutoff) add the
// head filter lowPass + hf * highPass (hf from the angle to the ear vector),
// late ones a single tap. Each contribution is truncated to a 2^-26 fixed
// point value, as the reference, and summed with 64-bit integer atomics, so
// the sum is exact and independent of thread order; a second kernel converts
// to float and clears the accumulator. Both kernels take both ears, and the
// powers of the walls' damping and the image coordinates, which depend on one
// index each, come from tables in shared memory (with the powers multiplied out
// for every image and one launch per ear, 2.3 million images took 2 x 47 us). Differences from the reference: damp^k
// by repeated multiplication (native_powr is implementation-defined), sqrt
// correctly rounded, 64-bit sums converted as signed (the reference's int32
// sums can wrap and Fill.cl converts them as unsigned). Every product and sum
// is an explicit round-to-nearest operation, so the results are reproducible.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>

#include "../../include/tanb.h"
#include "tanb_internal.h"

namespace tanb {
namespace {

struct RoomArgs {
  float W, H, L;
  float dLeft, dRight, dTop, dBottom, dFront, dBack;
  float sx, sy, sz;
  float hx[2], hy[2], hz[2];                // left, right
  float evx[2], evy[2], evz[2], earV[2];
  float maxGain, dMin, maxD2;               // maxD2: squared distance past which no image reaches the response
  int rate, length, hrtfLength, filterLength;
  int numRefX, numRefY, numRefZ;  // 2 n per axis
  int cx, cy, cz;                 // grid extent per axis (indices 0 .. c-1)
  float lp[64], hp[64];
};

__device__ __forceinline__ float pow_int(float b, int k) {
  float r = 1.0f;
  for (int i = 0; i < k; ++i) r = __fmul_rn(r, b);
  return r;
}

__device__ __forceinline__ float image_pos(int idx, float size, float s) {
  const float a = (idx % 2 == 0) ? (float)idx : (float)(idx + 1);
  const float b = (idx % 2 == 0) ? 1.0f : -1.0f;
  return __fadd_rn(__fmul_rn(a, size), __fmul_rn(b, s));
}

// One image at offset (dx, dy, dz) from ear e's head position with the walls'
// product `amp`.
__device__ __forceinline__ void room_image(const RoomArgs& a, int e, float amp, float dx, float dy, float dz, float d2,
                                           unsigned long long* __restrict__ acc) {
  const float kF2I = 67108864.0f;
  const float d = __fsqrt_rn(d2);
  const int fi = 1 + __float2int_rz(__fmul_rn(__fdiv_rn(d, 340.0f), (float)a.rate));
  if (fi >= a.length) return;
  const float dr = (d <= a.dMin) ? a.maxGain : __fdiv_rn(__fmul_rn(a.maxGain, a.dMin), d);
  const float g = __fmul_rn(__fmul_rn(kF2I, amp), dr);
  if (fi < a.hrtfLength) {
    const float dp = __fadd_rn(__fadd_rn(__fmul_rn(a.evx[e], dx), __fmul_rn(a.evy[e], dy)), __fmul_rn(a.evz[e], dz));
    const float cosA = __fdiv_rn(dp, __fmul_rn(a.earV[e], d));
    const float hf = __fdiv_rn(__fadd_rn(cosA, 1.0f), 2.0f);
    const int len = min(a.filterLength, a.length - fi);
    for (int i = 0; i < len; ++i) {
      const int v = __float2int_rz(__fmul_rn(g, __fadd_rn(a.lp[i], __fmul_rn(hf, a.hp[i]))));
      atomicAdd(acc + fi + i, (unsigned long long)(long long)v);
    }
  } else {
    atomicAdd(acc + fi, (unsigned long long)(long long)__float2int_rz(g));
  }
}

// Reflections off the two walls of an axis for index i (GenerateRoomResponse.cl:261-276).
__device__ __forceinline__ int refl_near(int i) { return i > 0 ? i / 2 : abs(i - 1) / 2; }
__device__ __forceinline__ int refl_far(int i) { return i > 0 ? (i + 1) / 2 : abs(i) / 2; }

// One axis's table entry: offsets from each ear and the two walls' powers.
struct __align__(16) RoomAxis {
  float d0, d1;  // image coordinate minus the left / right ear's
  float p, q;    // damp_far ^ k_far, damp_near ^ k_near
};

// Images of both ears: a warp per row along the longest axis (FAST: 0 x, 1 y,
// 2 z), rows from a grid-stride loop. `acc` + ear * stride: the ears' sums.
template <int FAST>
__global__ void __launch_bounds__(256) room_images_kernel(const __grid_constant__ RoomArgs a,
                                                          unsigned long long* __restrict__ acc, size_t stride) {
  extern __shared__ RoomAxis tab[];
  RoomAxis* tx = tab;
  RoomAxis* ty = tab + a.cx;
  RoomAxis* tz = ty + a.cy;
  float* pw = reinterpret_cast<float*>(tz + a.cz);  // [3 axes][far, near][max power + 1]
  const int np = max(a.numRefX, max(a.numRefY, a.numRefZ)) / 2 + 2;
  if (threadIdx.x < 6) {
    const float b = threadIdx.x == 0 ? a.dRight : threadIdx.x == 1 ? a.dLeft : threadIdx.x == 2 ? a.dTop
                    : threadIdx.x == 3 ? a.dBottom : threadIdx.x == 4 ? a.dFront : a.dBack;
    float r = 1.0f;
    for (int k = 0; k < np; ++k) {
      pw[threadIdx.x * np + k] = r;
      r = __fmul_rn(r, b);
    }
  }
  __syncthreads();
  for (int v = threadIdx.x; v < a.cx + a.cy + a.cz; v += blockDim.x) {
    const int ax = v < a.cx ? 0 : v < a.cx + a.cy ? 1 : 2;
    const int i = ax == 0 ? v - a.numRefX / 2 : ax == 1 ? v - a.cx - a.numRefY / 2 : v - a.cx - a.cy - a.numRefZ / 2;
    const float r = image_pos(i, ax == 0 ? a.W : ax == 1 ? a.H : a.L, ax == 0 ? a.sx : ax == 1 ? a.sy : a.sz);
    RoomAxis e;
    e.d0 = __fsub_rn(r, ax == 0 ? a.hx[0] : ax == 1 ? a.hy[0] : a.hz[0]);
    e.d1 = __fsub_rn(r, ax == 0 ? a.hx[1] : ax == 1 ? a.hy[1] : a.hz[1]);
    e.p = pw[2 * ax * np + refl_far(i)];
    e.q = pw[(2 * ax + 1) * np + refl_near(i)];
    tab[v] = e;
  }
  __syncthreads();
  const int cf = FAST == 0 ? a.cx : FAST == 1 ? a.cy : a.cz;    // along the row
  const int cu = FAST == 0 ? a.cy : a.cx, cv = FAST == 2 ? a.cy : a.cz;
  const RoomAxis* tf = FAST == 0 ? tx : FAST == 1 ? ty : tz;
  const RoomAxis* tu = FAST == 0 ? ty : tx;
  const RoomAxis* tv = FAST == 2 ? ty : tz;
  const int lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
  const long long rows = (long long)cu * cv;
  for (long long row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); row < rows; row += warps) {
    const RoomAxis u = tu[(int)(row % cu)], v = tv[(int)(row / cu)];
    // rows out of reach of both ears (maxD2 has a margin for the rounding)
    if (fmaf(u.d0, u.d0, v.d0 * v.d0) > a.maxD2 && fmaf(u.d1, u.d1, v.d1 * v.d1) > a.maxD2) continue;
    for (int f = lane; f < cf; f += 32) {
      const RoomAxis w = tf[f];
      const RoomAxis x = FAST == 0 ? w : u, y = FAST == 1 ? w : FAST == 0 ? u : v, z = FAST == 2 ? w : v;
      // far and near walls of x, y, z in the reference's order
      float amp = __fmul_rn(x.p, x.q);
      amp = __fmul_rn(amp, y.p);
      amp = __fmul_rn(amp, y.q);
      amp = __fmul_rn(amp, z.p);
      amp = __fmul_rn(amp, z.q);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float dx = e ? x.d1 : x.d0, dy = e ? y.d1 : y.d0, dz = e ? z.d1 : z.d0;
        const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
        if (d2 <= a.maxD2) room_image(a, e, amp, dx, dy, dz, d2, acc + e * stride);
      }
    }
  }
}

// The same with every image from its indices alone, for grids whose tables do
// not fit in shared memory.
__global__ void room_images_any_kernel(const __grid_constant__ RoomArgs a, unsigned long long* __restrict__ acc,
                                       size_t stride, long long images) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < images;
       t += (long long)gridDim.x * blockDim.x) {
    const int ix = (int)(t % a.cx) - a.numRefX / 2, iy = (int)((t / a.cx) % a.cy) - a.numRefY / 2,
              iz = (int)(t / ((long long)a.cx * a.cy)) - a.numRefZ / 2;
    const float rx = image_pos(ix, a.W, a.sx), ry = image_pos(iy, a.H, a.sy), rz = image_pos(iz, a.L, a.sz);
    float amp = pow_int(a.dRight, refl_far(ix));
    amp = __fmul_rn(amp, pow_int(a.dLeft, refl_near(ix)));
    amp = __fmul_rn(amp, pow_int(a.dTop, refl_far(iy)));
    amp = __fmul_rn(amp, pow_int(a.dBottom, refl_near(iy)));
    amp = __fmul_rn(amp, pow_int(a.dFront, refl_far(iz)));
    amp = __fmul_rn(amp, pow_int(a.dBack, refl_near(iz)));
    for (int e = 0; e < 2; ++e) {
      const float dx = __fsub_rn(rx, a.hx[e]), dy = __fsub_rn(ry, a.hy[e]), dz = __fsub_rn(rz, a.hz[e]);
      const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
      if (d2 <= a.maxD2) room_image(a, e, amp, dx, dy, dz, d2, acc + e * stride);
    }
  }
}

// Sums to float, cleared for the next call: ear ear0 + blockIdx.y.
__global__ void room_fill_kernel(unsigned long long* __restrict__ acc, size_t stride, float* left, float* right,
                                 int length, int ear0) {
  const int ear = ear0 + blockIdx.y;
  unsigned long long* s = acc + ear * stride;
  float* out = ear ? right : left;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < length; i += gridDim.x * blockDim.x) {
    out[i] = __fdiv_rn(__ll2float_rn((long long)s[i]), 67108864.0f);
    s[i] = 0ull;
  }
}

// Tables of a launch at most (fits beside four CTAs per SM, below the 48 KB of
// unconfigured dynamic shared memory).
constexpr size_t kRoomTableBytes = 40u << 10;

int32_t rfail(int32_t code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  set_last_error(buf);
  return code;
}

}  // namespace
}  // namespace tanb

struct tanb_room_generator {
  tanb_context* ctx = nullptr;
  std::mutex mu;
  cudaStream_t stream = nullptr;
  int max_length = 0;
  unsigned long long* acc = nullptr;  // [2][max_length], zero between calls
  cudaEvent_t done = nullptr;         // end of the last call, on whichever stream it ran
  long long images_last = 0;
};

extern "C" {

int32_t tanb_room_generator_create(tanb_context* ctx, int32_t max_length, tanb_room_generator** out) {
  if (!ctx || !out) return tanb::rfail(TANB_INVALID_POINTER, "null argument");
  *out = nullptr;
  if (max_length <= 0) return tanb::rfail(TANB_INVALID_ARG, "max_length must be > 0");
  tanb_room_generator* g = new tanb_room_generator();
  g->ctx = ctx;
  g->max_length = max_length;
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&g->done, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaMalloc(&g->acc, 2 * (size_t)max_length * sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMemsetAsync(g->acc, 0, 2 * (size_t)max_length * sizeof(unsigned long long), g->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
  if (e != cudaSuccess) {
    if (g->acc) cudaFree(g->acc);
    if (g->done) cudaEventDestroy(g->done);
    if (g->stream) cudaStreamDestroy(g->stream);
    delete g;
    cudaGetLastError();
    return tanb::rfail(e == cudaErrorMemoryAllocation ? TANB_OUT_OF_MEMORY : TANB_FAIL, "room generator: %s",
                       cudaGetErrorString(e));
  }
  *out = g;
  return TANB_OK;
}

int32_t tanb_room_generator_release(tanb_room_generator* g) {
  if (!g) return TANB_OK;
  {
    std::lock_guard<std::mutex> lock(g->mu);
    cudaSetDevice(g->ctx->device);
    cudaEventSynchronize(g->done);
    cudaStreamSynchronize(g->stream);
    cudaFree(g->acc);
    cudaEventDestroy(g->done);
    cudaStreamDestroy(g->stream);
  }
  delete g;
  return TANB_OK;
}

int32_t tanb_room_response(tanb_room_generator* g, const tanb_room* room, const tanb_source* source,
                           const tanb_listener* ears, int32_t sample_rate, int32_t length, float* left, float* right,
                           uint32_t flags, int32_t max_bounces, void* stream) {
  if (!g || !room || !source || !ears || !left || !right) return tanb::rfail(TANB_INVALID_POINTER, "null argument");
  if (length <= 0 || length > g->max_length)
    return tanb::rfail(TANB_INVALID_ARG, "length %d not in [1, %d]", length, g->max_length);
  if (sample_rate <= 0) return tanb::rfail(TANB_INVALID_ARG, "sample_rate must be > 0");
  if (ears->filter_length < 0 || ears->filter_length > 64)
    return tanb::rfail(TANB_INVALID_ARG, "filter_length must be in [0, 64]");
  if ((flags & TANB_GENROOM_LIMIT_BOUNCES) && max_bounces <= 0)
    return tanb::rfail(TANB_INVALID_ARG, "max_bounces must be > 0 with TANB_GENROOM_LIMIT_BOUNCES");
  std::lock_guard<std::mutex> lock(g->mu);
  cudaError_t e = cudaSetDevice(g->ctx->device);
  if (e != cudaSuccess) return tanb::rfail(TANB_FAIL, "%s", cudaGetErrorString(e));
  cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : g->stream;

  // host setup, TrueAudioVR.cpp:663-731
  tanb::RoomArgs a{};
  a.W = room->width;
  a.H = room->height;
  a.L = room->length;
  a.dLeft = room->damp_left;
  a.dRight = room->damp_right;
  a.dTop = room->damp_top;
  a.dBottom = room->damp_bottom;
  a.dFront = room->damp_front;
  a.dBack = room->damp_back;
  a.sx = std::min(std::max(source->x, 0.0f), a.W);
  a.sy = std::min(std::max(source->y, 0.0f), a.H);
  a.sz = std::min(std::max(source->z, 0.0f), a.L);
  const float es = ears->ear_spacing;
  float ev[4][3] = {{es / 2, 0.0f, 0.0f}, {-es / 2, 0.0f, 0.0f}, {es / 2, 0.0f, -(es / 2)}, {-es / 2, 0.0f, -es / 2}};
  const float pi = (float)3.141592653589793;
  const float sY = std::sin(ears->yaw * pi / 180), cY = std::cos(ears->yaw * pi / 180);
  const float sP = std::sin(ears->pitch * pi / 180), cP = std::cos(ears->pitch * pi / 180);
  const float sR = std::sin(ears->roll * pi / 180), cR = std::cos(ears->roll * pi / 180);
  const float m[3][3] = {{cR * cY - sR * sP * sY, -sR * cP, cR * sY + sR * sP * cY},
                         {sR * cY + cR * sP * sY, cR * cP, sR * sY - cR * sP * cY},
                         {-cP * sY, sP, cP * cY}};
  for (auto& v : ev) {
    const float x = v[0], y = v[1], z = v[2];
    v[0] = x * m[0][0] + y * m[0][1] + z * m[0][2];
    v[1] = x * m[1][0] + y * m[1][1] + z * m[1][2];
    v[2] = x * m[2][0] + y * m[2][1] + z * m[2][2];
  }
  const int nSW = (int)((a.W / 340.0f) * sample_rate), nSH = (int)((a.H / 340.0f) * sample_rate),
            nSL = (int)((a.L / 340.0f) * sample_rate);
  if (nSW <= 0 || nSH <= 0 || nSL <= 0)
    return tanb::rfail(TANB_INVALID_ARG, "room smaller than one sample of sound travel");
  int nW = 1 + length / nSW, nH = 1 + length / nSH, nL = 1 + length / nSL;
  if (flags & TANB_GENROOM_LIMIT_BOUNCES) {
    nW = std::min(nW, max_bounces);
    nH = std::min(nH, max_bounces);
    nL = std::min(nL, max_bounces);
  }
  a.numRefX = 2 * nW;
  a.numRefY = 2 * nH;
  a.numRefZ = 2 * nL;
  // the reference's NDRange: 2n rounded up to the local size 4, ids above 2n return
  auto extent = [](int n2) { return std::min((n2 % 4) ? n2 + 4 - n2 % 4 : n2, n2 + 1); };
  a.cx = extent(a.numRefX);
  a.cy = extent(a.numRefY);
  a.cz = extent(a.numRefZ);
  a.rate = sample_rate;
  a.length = length;
  a.hrtfLength = 2 * (nSW + nSH + nSL);
  a.filterLength = ears->filter_length;
  a.maxGain = 2.0f;
  a.dMin = 2 * es;
  std::memcpy(a.lp, ears->low_pass, sizeof(a.lp));
  std::memcpy(a.hp, ears->high_pass, sizeof(a.hp));
  const long long images = (long long)a.cx * a.cy * a.cz;
  g->images_last = images;
  for (int ch = 0; ch < 2; ++ch) {
    a.hx[ch] = ears->head_x + ev[ch][0];
    a.hy[ch] = ears->head_y + ev[ch][1];
    a.hz[ch] = ears->head_z + ev[ch][2];
    a.evx[ch] = ev[2 + ch][0];
    a.evy[ch] = ev[2 + ch][1];
    a.evz[ch] = ev[2 + ch][2];
    a.earV[ch] = std::sqrt(a.evx[ch] * a.evx[ch] + a.evy[ch] * a.evy[ch] + a.evz[ch] * a.evz[ch]);
  }
  // An image at or past sample `length` contributes nothing; the kernels' single
  // precision distances are within a few 2^-24 of the exact ones, so that no image
  // past this squared distance can land before it.
  const double reach = (double)length / sample_rate * 340.0;
  a.maxD2 = (float)(reach * reach * (1.0 + 1e-4));
  // calls share the accumulator: each starts after the previous one ended
  e = cudaStreamWaitEvent(st, g->done, 0);
  if (e != cudaSuccess) return tanb::rfail(TANB_FAIL, "%s", cudaGetErrorString(e));
  const int np = std::max(a.numRefX, std::max(a.numRefY, a.numRefZ)) / 2 + 2;
  const size_t smem = (size_t)((long long)a.cx + a.cy + a.cz) * sizeof(tanb::RoomAxis) + 6 * (size_t)np * sizeof(float);
  if (smem <= tanb::kRoomTableBytes) {
    const int fast = a.cx >= a.cy && a.cx >= a.cz ? 0 : a.cy >= a.cz ? 1 : 2;
    const long long rows = images / (fast == 0 ? a.cx : fast == 1 ? a.cy : a.cz);
    const unsigned blocks = (unsigned)std::max<long long>(1, std::min<long long>((rows + 7) / 8, tanb::kSms * 4));
    auto kernel = fast == 0 ? tanb::room_images_kernel<0> : fast == 1 ? tanb::room_images_kernel<1>
                                                                      : tanb::room_images_kernel<2>;
    kernel<<<blocks, 256, smem, st>>>(a, g->acc, (size_t)g->max_length);
  } else {
    const unsigned blocks = (unsigned)std::max<long long>(1, std::min<long long>((images + 255) / 256, 16LL * tanb::kSms));
    tanb::room_images_any_kernel<<<blocks, 256, 0, st>>>(a, g->acc, (size_t)g->max_length, images);
  }
  const unsigned fill = (unsigned)std::min(1024, (length + 255) / 256);
  if (left + length <= right || right + length <= left) {
    tanb::room_fill_kernel<<<dim3(fill, 2), 256, 0, st>>>(g->acc, (size_t)g->max_length, left, right, length, 0);
  } else {  // overlapping rows: the right ear is written last
    for (int ear = 0; ear < 2; ++ear)
      tanb::room_fill_kernel<<<fill, 256, 0, st>>>(g->acc, (size_t)g->max_length, left, right, length, ear);
  }
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaEventRecord(g->done, st);
  if (e != cudaSuccess) return tanb::rfail(TANB_FAIL, "room response launch: %s", cudaGetErrorString(e));
  return TANB_OK;
}

int64_t tanb_room_images(tanb_room_generator* g) { return g ? g->images_last : 0; }

int32_t tanb_room_generator_synchronize(tanb_room_generator* g) {
  if (!g) return tanb::rfail(TANB_INVALID_POINTER, "null generator");
  std::lock_guard<std::mutex> lock(g->mu);
  cudaError_t e = cudaSetDevice(g->ctx->device);
  if (e == cudaSuccess) e = cudaEventSynchronize(g->done);
  if (e != cudaSuccess) return tanb::rfail(TANB_FAIL, "%s", cudaGetErrorString(e));
  return TANB_OK;
}

void* tanb_room_generator_stream(tanb_room_generator* g) { return g ? (void*)g->stream : nullptr; }

}  // extern "C"
