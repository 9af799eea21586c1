// fa_kernels.cu -- sm_100a kernels of the warper path.
//
//   sobel_kernel    Sobel3d (FrameAligner/Sobel3d.cpp:8-85), bit-exact float arithmetic
//   hessian_*       computeSteepestDecentImages + computeHessian (FrameWarper.cpp:296-395)
//   eval_kernel     fused warpImageInterpolated + computeErrorImage + computeJacobian
//                   (FrameWarper.cpp:4-69,147-176): one HBM pass per frame evaluation
//   reduce_kernel   deterministic tile -> frame reduction of f and J^T e
//   warp_kernel     warpImageInterpolated output image
//
// Layout: volumes {nz, ny, nx}, x fastest. A tile is `tile_rows` consecutive image rows; the host
// picks tile_rows so that a tile meets at most two storage ranges (three control points).
#include <algorithm>

#include "fa_device.cuh"

namespace fa {

namespace {
std::atomic<unsigned> g_smem_epoch[kSmemDevices];
}
unsigned smem_epoch(int device) {
  return device >= 0 && device < kSmemDevices ? g_smem_epoch[device].load(std::memory_order_acquire) : 0u;
}
void smem_new_context(int device) {
  if (device < 0 || device >= kSmemDevices) return;
  if (++g_smem_epoch[device] == 0u) ++g_smem_epoch[device];
}

// ------------------------------------------------------------------ Sobel3d ----------------------

// One separable pass (Sobel3d.cpp:8-58) at a position of an axis from its neighbours: interior
// f0*lo + f1*mid + f2*hi; first of the axis e1a*mid + e1b*hi; last e2a*mid + e2b*lo. Float products and
// sums are rounded one by one (no FMA), as in the reference build. EDGE false: interior for certain.
struct AxisPos {
  bool first, last;
};
template <bool EDGE>
__device__ __forceinline__ float pass3(AxisPos q, float lo, float mid, float hi, float f0, float f1, float f2, float e1a,
                                       float e1b, float e2a, float e2b) {
  float r = __fadd_rn(__fadd_rn(__fmul_rn(f0, lo), __fmul_rn(f1, mid)), __fmul_rn(f2, hi));
  if (EDGE) {
    if (q.first)
      r = __fadd_rn(__fmul_rn(e1a, mid), __fmul_rn(e1b, hi));
    else if (q.last)
      r = __fadd_rn(__fmul_rn(e2a, mid), __fmul_rn(e2b, lo));
  }
  return r;
}
template <bool EDGE>
__device__ __forceinline__ float smooth3(AxisPos q, float lo, float mid, float hi) {
  return pass3<EDGE>(q, lo, mid, hi, 1.0f / 4.0f, 2.0f / 4.0f, 1.0f / 4.0f, 2.0f / 3.0f, 2.0f / 3.0f, 2.0f / 3.0f, 2.0f / 3.0f);
}
template <bool EDGE>
__device__ __forceinline__ float diff3(AxisPos q, float lo, float mid, float hi) {
  return pass3<EDGE>(q, lo, mid, hi, -0.5f, 0.0f, 0.5f, -0.5f, 0.5f, 0.5f, -0.5f);
}

// Sobel3d (Sobel3d.cpp:60-85), gx = Dx(Sz(Sy(m))), gy = Dy(Sz(Sx(m))), gz = Dz(Sy(Sx(m))) (:73-84), bit
// for bit: every value is formed by pass3 with its global position, so the edge rules apply at the
// volume's faces and every product and sum is rounded in the reference's order. A thread marches along
// z at one (x, y): of each plane it reads the 3 x 3 neighbourhood (nine loads, the cache serves eight) and
// keeps Sx of the three rows, Sy of the three columns and Sy(Sx) for three planes, from which the plane in
// the middle follows. With QUAD (nx a multiple of 4, so that a group of four voxels is four lanes) the
// BF16 groups of RefDev::q16 are written in the same pass: four lanes exchange so that each writes one
// quantity of the group.
// HBM-bound in principle (4 B in, 12 or 20 B out per voxel: 15 us for 512 x 512 x 16 at the copy rate);
// with the groups 40 us there, by instruction issue (131 + 39 us before: passes through shared memory with
// a division per element and step, then a conversion of its own; the edge rules cost another 30 us
// where no column of a CTA is at a face, so those CTAs take a march without them).
constexpr int kSobX = 32, kSobY = 8;

// The march of one CTA; EDGE: some of its columns are at a face along x or y.
template <bool QUAD, bool EDGE>
__device__ __forceinline__ void sobel_march(const float* __restrict__ m, int nz, int ny, int nx, int zc,
                                            float* __restrict__ gx, float* __restrict__ gy, float* __restrict__ gz,
                                            __nv_bfloat16* __restrict__ q16) {
  const int x = blockIdx.x * kSobX + threadIdx.x, y = blockIdx.y * kSobY + threadIdx.y;
  const int z0 = blockIdx.z * zc, z1 = min(z0 + zc, nz);
  if (y >= ny) return;  // whole warps: a warp is one row
  const bool in = x < nx;
  const int xc = min(x, nx - 1);
  const int xs[3] = {max(xc - 1, 0), xc, min(xc + 1, nx - 1)};
  const int ys[3] = {max(y - 1, 0), y, min(y + 1, ny - 1)};
  const AxisPos px{xc == 0, xc == nx - 1}, py{y == 0, y == ny - 1};  // a clamped neighbour is never used
  const int plane = ny * nx;  // fewer than 2^31 voxels
  float A[3][3], A2[3][3], B[3];  // [plane][row]: Sx(m); [plane][column]: Sy(m); [plane]: Sy(Sx(m))
  float mid[3];                   // the reference itself
  auto load = [&](int z, float* a, float* a2, float& b, float& v) {
    const float* p = m + min(max(z, 0), nz - 1) * plane;
    float w[3][3];
#pragma unroll
    for (int j = 0; j < 3; j++)
#pragma unroll
      for (int i = 0; i < 3; i++) w[j][i] = __ldg(p + ys[j] * nx + xs[i]);
#pragma unroll
    for (int j = 0; j < 3; j++) a[j] = smooth3<EDGE>(px, w[j][0], w[j][1], w[j][2]);
#pragma unroll
    for (int i = 0; i < 3; i++) a2[i] = smooth3<EDGE>(py, w[0][i], w[1][i], w[2][i]);
    b = smooth3<EDGE>(py, a[0], a[1], a[2]);
    v = w[1][1];
  };
  load(z0 - 1, A[0], A2[0], B[0], mid[0]);
  load(z0, A[1], A2[1], B[1], mid[1]);
#pragma unroll 1
  for (int z = z0; z < z1; z++) {
    load(z + 1, A[2], A2[2], B[2], mid[2]);
    float c[3], b2[3], g[3];
    if (nz > 1 && z > 0 && z < nz - 1) {
      const AxisPos pz{false, false};
#pragma unroll
      for (int i = 0; i < 3; i++) {
        c[i] = smooth3<false>(pz, A[0][i], A[1][i], A[2][i]);
        b2[i] = smooth3<false>(pz, A2[0][i], A2[1][i], A2[2][i]);
      }
      g[2] = diff3<false>(pz, B[0], B[1], B[2]);
    } else {  // a single plane is copied by the z passes
      const AxisPos pz{z == 0, z == nz - 1};
#pragma unroll
      for (int i = 0; i < 3; i++) {
        c[i] = nz == 1 ? A[1][i] : smooth3<true>(pz, A[0][i], A[1][i], A[2][i]);
        b2[i] = nz == 1 ? A2[1][i] : smooth3<true>(pz, A2[0][i], A2[1][i], A2[2][i]);
      }
      g[2] = nz == 1 ? B[1] : diff3<true>(pz, B[0], B[1], B[2]);
    }
    g[0] = diff3<EDGE>(px, b2[0], b2[1], b2[2]);
    g[1] = diff3<EDGE>(py, c[0], c[1], c[2]);
    const int p = z * plane + y * nx + x;
    if (in) {
      gx[p] = g[0];
      gy[p] = g[1];
      gz[p] = g[2];
    }
    if (QUAD) {
      // four lanes hold a group of four voxels, four quantities each; lane j has to hold quantity j of the
      // four: a 4 x 4 transpose in two exchanges
      const int j = threadIdx.x & 3;
      float q[4] = {mid[1], g[0], g[1], g[2]};
      const bool odd = j & 1, high = j & 2;
      const float s0 = __shfl_xor_sync(0xffffffffu, odd ? q[0] : q[1], 1), s1 = __shfl_xor_sync(0xffffffffu, odd ? q[2] : q[3], 1);
      if (odd) {
        q[0] = s0;
        q[2] = s1;
      } else {
        q[1] = s0;
        q[3] = s1;
      }
      const float t0 = __shfl_xor_sync(0xffffffffu, high ? q[0] : q[2], 2), t1 = __shfl_xor_sync(0xffffffffu, high ? q[1] : q[3], 2);
      if (high) {
        q[0] = t0;
        q[1] = t1;
      } else {
        q[2] = t0;
        q[3] = t1;
      }
      const __nv_bfloat162 lo = __floats2bfloat162_rn(q[0], q[1]), hi = __floats2bfloat162_rn(q[2], q[3]);
      if (in)
        *reinterpret_cast<uint2*>(q16 + (long long)(p >> 2) * 16 + j * 4) =
            make_uint2(*reinterpret_cast<const unsigned*>(&lo), *reinterpret_cast<const unsigned*>(&hi));
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
      A[0][i] = A[1][i];
      A[1][i] = A[2][i];
      A2[0][i] = A2[1][i];
      A2[1][i] = A2[2][i];
    }
    B[0] = B[1];
    B[1] = B[2];
    mid[1] = mid[2];
  }
}

template <bool QUAD>
__global__ void __launch_bounds__(kSobX * kSobY) sobel_kernel(const float* __restrict__ m, int nz, int ny, int nx,
                                                             int zc, float* __restrict__ gx, float* __restrict__ gy,
                                                             float* __restrict__ gz, __nv_bfloat16* __restrict__ q16) {
  const bool edge = blockIdx.x == 0 || blockIdx.y == 0 || (int)(blockIdx.x + 1) * kSobX >= nx ||
                    (int)(blockIdx.y + 1) * kSobY >= ny;
  if (edge)
    sobel_march<QUAD, true>(m, nz, ny, nx, zc, gx, gy, gz, q16);
  else
    sobel_march<QUAD, false>(m, nz, ny, nx, zc, gx, gy, gz, q16);
}

cudaError_t launch_sobel(const float* m, int nz, int ny, int nx, float* gx, float* gy, float* gz, __nv_bfloat16* q16,
                         cudaStream_t s) {
  // planes per CTA: the march pays two extra planes per chunk, a short one fills the GPU
  const long long cols = (long long)((nx + kSobX - 1) / kSobX) * ((ny + kSobY - 1) / kSobY);
  int zc = nz;
  while (zc > 4 && cols * ((nz + zc - 1) / zc) < 148 * 8) zc = (zc + 1) / 2;
  const dim3 grid((nx + kSobX - 1) / kSobX, (ny + kSobY - 1) / kSobY, (nz + zc - 1) / zc), block(kSobX, kSobY);
  if (grid.y > 65535 || grid.z > 65535) return cudaErrorInvalidValue;
  if (q16 != nullptr && nx % 4 == 0) {
    sobel_kernel<true><<<grid, block, 0, s>>>(m, nz, ny, nx, zc, gx, gy, gz, q16);
    return cudaGetLastError();
  }
  sobel_kernel<false><<<grid, block, 0, s>>>(m, nz, ny, nx, zc, gx, gy, gz, nullptr);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && q16 != nullptr) e = launch_to_quad16(m, gx, gy, gz, (long long)nz * ny * nx, q16, s);
  return e;
}

// ------------------------------------------------------------------ conversions ------------------

__global__ void to_quad16_kernel(const float* __restrict__ ref, const float* __restrict__ gx,
                                 const float* __restrict__ gy, const float* __restrict__ gz, long long n,
                                 __nv_bfloat16* __restrict__ q16) {
  const long long groups = (n + 3) / 4;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < groups * 16;
       i += (long long)gridDim.x * blockDim.x) {
    const long long g = i >> 4;
    const int k = (int)(i >> 2) & 3, j = (int)i & 3;
    const long long p = 4 * g + j;
    const float* src = k == 0 ? ref : (k == 1 ? gx : (k == 2 ? gy : gz));
    q16[i] = __float2bfloat16_rn(p < n ? src[p] : 0.0f);
  }
}

cudaError_t launch_to_quad16(const float* ref, const float* gx, const float* gy, const float* gz, long long n,
                             __nv_bfloat16* q16, cudaStream_t s) {
  const long long total = (n + 3) / 4 * 16;
  int blocks = (int)((total + 255) / 256);
  if (blocks > 148 * 32) blocks = 148 * 32;
  if (blocks < 1) blocks = 1;
  to_quad16_kernel<<<blocks, 256, 0, s>>>(ref, gx, gy, gz, n, q16);
  return cudaGetLastError();
}

__device__ __forceinline__ float load_any(const void* in, int t, long long i) {
  switch (t) {
    case FA_F32: return static_cast<const float*>(in)[i];
    case FA_F16: return __half2float(static_cast<const __half*>(in)[i]);
    case FA_BF16: return __bfloat162float(static_cast<const __nv_bfloat16*>(in)[i]);
    default: return (float)static_cast<const uint16_t*>(in)[i];
  }
}

// Raw frame (any dtype) -> warper storage with FrameWarpAligner's +1 offset
// (FrameWarpAligner.cpp:142), converted to float first as the reference does (convertTo CV_32F).
__global__ void offset_convert_kernel(const void* __restrict__ in, int in_t, void* __restrict__ out, int out_t,
                                      long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    float v = load_any(in, in_t, i) + 1.0f;
    if (out_t == FA_F16)
      static_cast<__half*>(out)[i] = __float2half_rn(v);
    else
      static_cast<float*>(out)[i] = v;
  }
}

cudaError_t launch_offset_convert(const void* in, fa_dtype in_type, void* out, fa_dtype out_type, long long n,
                                  cudaStream_t s) {
  int blocks = (int)((n + 255) / 256);
  if (blocks > 148 * 32) blocks = 148 * 32;
  if (blocks < 1) blocks = 1;
  offset_convert_kernel<<<blocks, 256, 0, s>>>(in, (int)in_type, out, (int)out_type, n);
  return cudaGetLastError();
}

// Raw or converted values into a frame slot's interior (row pitch fpitch, plane stride fplane, out
// pointing at voxel (0,0,0)); add_one applies FrameWarpAligner's +1 (FrameWarpAligner.cpp:142).
__global__ void to_slot_kernel(const void* __restrict__ in, int in_t, void* __restrict__ out, int out_kind, int ny,
                               int nx, int n_rows, int fpitch, long long fplane, int add_one) {
  for (int row = blockIdx.x; row < n_rows; row += gridDim.x) {
    const int y = row % ny, z = row / ny;
    const long long ib = (long long)row * nx;
    const long long ob = (long long)z * fplane + (long long)y * fpitch;
    for (int x = threadIdx.x; x < nx; x += blockDim.x) {
      if (out_kind == kFrameRawU16) {
        // count + 1, saturated (a raw count of 65535 is stored as 65535)
        const unsigned c = static_cast<const unsigned short*>(in)[ib + x] + (add_one ? 1u : 0u);
        static_cast<unsigned short*>(out)[ob + x] = (unsigned short)(c > 65535u ? 65535u : c);
      } else {
        const float v = load_any(in, in_t, ib + x) + (add_one ? 1.0f : 0.0f);
        if (out_kind == kFrameF16)
          static_cast<__half*>(out)[ob + x] = __float2half_rn(v);
        else
          static_cast<float*>(out)[ob + x] = v;
      }
    }
  }
}

// The same conversion 8 elements per thread with 16-byte loads and stores (rows of a multiple of 8
// elements, 16-byte aligned rows on both sides): dense FP32 or uint16 in, slot storage IN_U16 ->
// raw counts (saturated + 1) or FP16 / FP32 values.
template <bool IN_U16, int OUT_KIND>
__global__ void __launch_bounds__(256) to_slot_vec_kernel(const void* __restrict__ in, void* __restrict__ out,
                                                          int nx8, int ny, long long n_chunks, int fpitch,
                                                          long long fplane, int add_one) {
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n_chunks;
       c += (long long)gridDim.x * blockDim.x) {
    const long long row = c / nx8;
    const int xc = (int)(c - row * nx8);
    const int y = (int)(row % ny);
    const long long z = row / ny;
    const long long ib = c * 8;  // rows are dense: row * nx + 8 * xc
    const long long ob = z * fplane + (long long)y * fpitch + 8 * xc;
    if (OUT_KIND == kFrameRawU16) {
      // count + 1, saturated (a raw count of 65535 is stored as 65535)
      uint4 q = *reinterpret_cast<const uint4*>(static_cast<const unsigned short*>(in) + ib);
      unsigned w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const unsigned lo = min((w[i] & 0xffffu) + (unsigned)add_one, 65535u);
        const unsigned hi = min((w[i] >> 16) + (unsigned)add_one, 65535u);
        w[i] = lo | (hi << 16);
      }
      *reinterpret_cast<uint4*>(static_cast<unsigned short*>(out) + ob) = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
      float v[8];
      if (IN_U16) {
        const uint4 q = *reinterpret_cast<const uint4*>(static_cast<const unsigned short*>(in) + ib);
        const unsigned w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
          v[2 * i] = (float)(w[i] & 0xffffu);
          v[2 * i + 1] = (float)(w[i] >> 16);
        }
      } else {
        const float4 a = *reinterpret_cast<const float4*>(static_cast<const float*>(in) + ib);
        const float4 b = *reinterpret_cast<const float4*>(static_cast<const float*>(in) + ib + 4);
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
      }
#pragma unroll
      for (int i = 0; i < 8; i++) v[i] = v[i] + (add_one ? 1.0f : 0.0f);
      if (OUT_KIND == kFrameF16) {
        __half2 h[4];
#pragma unroll
        for (int i = 0; i < 4; i++) h[i] = __halves2half2(__float2half_rn(v[2 * i]), __float2half_rn(v[2 * i + 1]));
        *reinterpret_cast<uint4*>(static_cast<__half*>(out) + ob) = *reinterpret_cast<const uint4*>(h);
      } else {
        float* o = static_cast<float*>(out) + ob;
        *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(o + 4) = make_float4(v[4], v[5], v[6], v[7]);
      }
    }
  }
}

cudaError_t launch_to_slot(const void* in, fa_dtype in_type, void* out, int out_kind, int nz, int ny, int nx,
                           int fpitch, long long fplane, bool add_one, cudaStream_t s) {
  const int n_rows = nz * ny;
  const size_t out_esz = out_kind == kFrameF32 ? 4 : 2;
  const bool vec = nx % 8 == 0 && (in_type == FA_U16 || in_type == FA_F32) &&
                   (out_kind != kFrameRawU16 || in_type == FA_U16) && reinterpret_cast<uintptr_t>(in) % 16 == 0 &&
                   reinterpret_cast<uintptr_t>(out) % 16 == 0 && (fpitch * out_esz) % 16 == 0 &&
                   (fplane * (long long)out_esz) % 16 == 0;
  if (vec) {
    const long long n_chunks = (long long)n_rows * (nx / 8);
    const int blocks = (int)std::min<long long>((n_chunks + 255) / 256, 148 * 8);
    const int a1 = add_one ? 1 : 0;
    if (in_type == FA_U16) {
      if (out_kind == kFrameRawU16)
        to_slot_vec_kernel<true, kFrameRawU16><<<blocks, 256, 0, s>>>(in, out, nx / 8, ny, n_chunks, fpitch, fplane, a1);
      else if (out_kind == kFrameF16)
        to_slot_vec_kernel<true, kFrameF16><<<blocks, 256, 0, s>>>(in, out, nx / 8, ny, n_chunks, fpitch, fplane, a1);
      else
        to_slot_vec_kernel<true, kFrameF32><<<blocks, 256, 0, s>>>(in, out, nx / 8, ny, n_chunks, fpitch, fplane, a1);
    } else {
      if (out_kind == kFrameF16)
        to_slot_vec_kernel<false, kFrameF16><<<blocks, 256, 0, s>>>(in, out, nx / 8, ny, n_chunks, fpitch, fplane, a1);
      else
        to_slot_vec_kernel<false, kFrameF32><<<blocks, 256, 0, s>>>(in, out, nx / 8, ny, n_chunks, fpitch, fplane, a1);
    }
    return cudaGetLastError();
  }
  int blocks = n_rows < 148 * 16 ? n_rows : 148 * 16;
  to_slot_kernel<<<blocks, 256, 0, s>>>(in, (int)in_type, out, out_kind, ny, nx, n_rows, fpitch, fplane, add_one ? 1 : 0);
  return cudaGetLastError();
}

// downsample (AbstractFrameAligner.cpp:37-56): output (z, y/b, x/b) = float sum of its b x b block,
// accumulated in the reference's loop order (y, then x).
__global__ void downsample_kernel(const void* __restrict__ in, int in_t, int nz, int ny, int nx, int b,
                                  float* __restrict__ out) {
  const int nh = (ny + b - 1) / b, nw = (nx + b - 1) / b;
  const long long n = (long long)nz * nh * nw;
  for (long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x; o < n; o += (long long)gridDim.x * blockDim.x) {
    const int ox = (int)(o % nw);
    const long long r = o / nw;
    const int oy = (int)(r % nh);
    const int z = (int)(r / nh);
    float acc = 0.0f;
    for (int y = oy * b; y < min(ny, oy * b + b); y++)
      for (int x = ox * b; x < min(nx, ox * b + b); x++)
        acc = __fadd_rn(acc, load_any(in, in_t, ((long long)z * ny + y) * nx + x));
    out[o] = acc;
  }
}

cudaError_t launch_downsample(const void* in, fa_dtype in_type, int nz, int ny, int nx, int b, float* out,
                              cudaStream_t s) {
  long long n = (long long)nz * ((ny + b - 1) / b) * ((nx + b - 1) / b);
  int blocks = (int)((n + 255) / 256);
  if (blocks > 148 * 32) blocks = 148 * 32;
  if (blocks < 1) blocks = 1;
  downsample_kernel<<<blocks, 256, 0, s>>>(in, (int)in_type, nz, ny, nx, b, out);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ fused evaluation -------------

// RUNS: the form for few tiles, where what a lane's voxels cost is the latency of their loads.
template <int NDIM, typename FT, typename RT, bool RUNS>
__global__ void __launch_bounds__(kEvalThreads) eval_kernel(const Job* __restrict__ jobs) {
  const Job& job = jobs[blockIdx.y];
  if (job.state != nullptr && (job.state->phase == kPhaseDone || job.state->phase == kPhaseWaitWarm)) return;
  const RefDev& R = job.R;
  const int tile = blockIdx.x;
  if (tile >= R.n_tiles) return;
  const int nx = R.nx, ny = R.ny, nz = R.nz;
  const int row_begin = tile * R.tile_rows;
  const int row_end = min(row_begin + R.tile_rows, R.n_rows);
  const int c0 = R.tile_c0[tile];
  const int cw = max(c0 - 1, 0);
  const bool bidir = R.bidir != 0;
  const float dq = R.dq;

  __shared__ float4 sD[kWin * kDParamF4];
  __shared__ float sred[kEvalWarps][1 + 3 * NDIM];
  for (int i = threadIdx.x; i < kWin * kDParamF4; i += blockDim.x) {
    const int k = cw + i / kDParamF4;
    sD[i] = (k < R.nD) ? job.dparams[k * kDParamF4 + i % kDParamF4] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();

  const FT* __restrict__ fr = static_cast<const FT*>(job.frame);
  // reference / gradient value k (0: reference, 1..3: gx, gy, gz) of voxel p
  auto refgrad = [&](int k, long long p) -> float {
    if constexpr (sizeof(RT) == 4) {
      const float* planes[4] = {R.ref32, R.gx32, R.gy32, R.gz32};
      return __ldg(planes[k] + p);
    } else {
      return __bfloat162float(__ldg(R.q16 + (p >> 2) * 16 + k * 4 + (p & 3)));
    }
  };

  float af = 0.0f;
  float ag[3][NDIM];
#pragma unroll
  for (int s = 0; s < 3; s++)
#pragma unroll
    for (int k = 0; k < NDIM; k++) ag[s][k] = 0.0f;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // One voxel of the general form: any interval, range and position.
  const bool padded = job.fpad != 0;
  auto general = [&](const RowDesc& rd, bool flip, int x, long long p) {
    const VoxelModel vm = voxel_model(rd, x, nx, flip, bidir, dq);
    // the host geometry guarantees c0-1 <= di <= c0+2; the clamp only keeps the shared-memory
    // window in bounds
    const int wi = min(max(vm.di - cw, 0), kWin - 2);
    const float v = sample<NDIM, FT>(fr, job.fplane, job.fpitch, sD + wi * kDParamF4, vm.f, x, rd.y, rd.z, nx, ny, nz);
    const float t = refgrad(0, p);
    // include iff the interpolated value is positive: CPU rule px == 0 -> -1, then wimg >= 0
    // (FrameWarper.cpp:67, 16-25)
    const float e = (v > 0.0f) ? v - t : 0.0f;
    af = fmaf(e, e, af);
    if (!vm.last) {
      const float e1 = e * vm.f;           // weight of control r+1: Df
      const float e0 = e * (1.0f - vm.f);  // weight of control r:   1 - Df
      float gk[NDIM];
#pragma unroll
      for (int k = 0; k < NDIM; k++) gk[k] = refgrad(k + 1, p);
      if (vm.r == c0) {
#pragma unroll
        for (int k = 0; k < NDIM; k++) {
          ag[0][k] = fmaf(gk[k], e0, ag[0][k]);
          ag[1][k] = fmaf(gk[k], e1, ag[1][k]);
        }
      } else {
#pragma unroll
        for (int k = 0; k < NDIM; k++) {
          ag[1][k] = fmaf(gk[k], e0, ag[1][k]);
          ag[2][k] = fmaf(gk[k], e1, ag[2][k]);
        }
      }
    }
  };
  if (!RUNS) {
    for (int row = row_begin + warp; row < row_end; row += kEvalWarps) {
      const RowDesc rd = R.rows[row];
      const bool flip = bidir && (rd.y & 1);
      for (int x = lane; x < nx; x += 32) general(rd, flip, x, (long long)row * nx + x);
    }
  }
  // Most of a row has one interval, one range and one integer offset of the sample position: a run. Its
  // parameters and tap rows stay in registers, and kTogether steps of 32 voxels have their loads in flight
  // together; a step that leaves the run (by a vote on every voxel's own values) takes the general form
  // and starts the next one. The values are the general form's, bit for bit.
  constexpr int kTogether = 4;
  for (int row = row_begin + warp; RUNS && row < row_end; row += kEvalWarps) {
    const RowDesc rd = R.rows[row];
    const bool flip = bidir && (rd.y & 1);
    const long long rowoff = (long long)row * nx;
    int di = -1, r = 0, y_first = 0, z_first = 0, ox = 0;
    float3 fl = make_float3(0.f, 0.f, 0.f);
    float4 ph, dd;
    bool run = false;
    auto start = [&](int x) {  // the run that voxel x (the same for every lane) is in
      const VoxelModel vm = voxel_model(rd, x, nx, flip, bidir, dq);
      di = vm.di;
      r = vm.r;
      const float4* P = sD + min(max(di - cw, 0), kWin - 2) * kDParamF4;
      const float4 n = P[0];
      ph = P[1];
      dd = P[2];
      fl.x = floorf(fmaf(vm.f, dd.x, ph.x));
      fl.y = floorf(fmaf(vm.f, dd.y, ph.y));
      fl.z = NDIM == 3 ? floorf(fmaf(vm.f, dd.z, ph.z)) : 0.0f;
      ox = (int)n.x + (int)fl.x;
      y_first = min(max(rd.y + (int)n.y + (int)fl.y, -kHaloY), ny + kHaloY - 2);
      z_first = NDIM == 3 ? min(max(rd.z + (int)n.z + (int)fl.z, -kHaloZ), nz + kHaloZ - 2) : 0;
      // the taps x + ox, x + ox + 1 of every voxel of the row inside the halo
      run = padded && ox >= -kHaloX && ox <= kHaloX - 1;
    };
    start(0);
    for (int xb = 0; xb < nx; xb += 32 * kTogether) {
      float f[kTogether], w[kTogether][NDIM];
      bool same = run;
#pragma unroll
      for (int u = 0; u < kTogether; u++) {
        const int x = min(xb + 32 * u + lane, nx - 1);
        const VoxelModel vm = voxel_model(rd, x, nx, flip, bidir, dq);
        f[u] = vm.f;
        const float tx = fmaf(vm.f, dd.x, ph.x), ty = fmaf(vm.f, dd.y, ph.y);
        w[u][0] = tx - fl.x;
        w[u][1] = ty - fl.y;
        same = same && vm.di == di && vm.r == r && !vm.last && floorf(tx) == fl.x && floorf(ty) == fl.y;
        if (NDIM == 3) {
          const float tz = fmaf(vm.f, dd.z, ph.z);
          w[u][NDIM - 1] = tz - fl.z;
          same = same && floorf(tz) == fl.z;
        }
      }
      if (!__all_sync(0xffffffffu, same)) {
#pragma unroll 1
        for (int u = 0; u < kTogether; u++) {
          const int x = xb + 32 * u + lane;
          if (x < nx) general(rd, flip, x, rowoff + x);
        }
        __syncwarp();
        start(min(xb + 32 * kTogether, nx - 1));
        continue;
      }
      float v[kTogether][NDIM == 3 ? 8 : 4], t[kTogether], gk[kTogether][NDIM];
#pragma unroll
      for (int u = 0; u < kTogether; u++) {
        const int x = min(xb + 32 * u + lane, nx - 1);
        const FT* p = fr + ((long long)z_first * job.fplane + (long long)y_first * job.fpitch + (x + ox));
        v[u][0] = ldf(p);
        v[u][1] = ldf(p + 1);
        v[u][2] = ldf(p + job.fpitch);
        v[u][3] = ldf(p + job.fpitch + 1);
        if (NDIM == 3) {
          const FT* q = p + job.fplane;
          v[u][NDIM == 3 ? 4 : 0] = ldf(q);
          v[u][NDIM == 3 ? 5 : 0] = ldf(q + 1);
          v[u][NDIM == 3 ? 6 : 0] = ldf(q + job.fpitch);
          v[u][NDIM == 3 ? 7 : 0] = ldf(q + job.fpitch + 1);
        }
        t[u] = refgrad(0, rowoff + x);
#pragma unroll
        for (int k = 0; k < NDIM; k++) gk[u][k] = refgrad(k + 1, rowoff + x);
      }
#pragma unroll
      for (int u = 0; u < kTogether; u++) {
        const float c00 = fmaf(w[u][0], v[u][1] - v[u][0], v[u][0]);
        const float c01 = fmaf(w[u][0], v[u][3] - v[u][2], v[u][2]);
        float val = fmaf(w[u][1], c01 - c00, c00);
        if (NDIM == 3) {
          const float* h = v[u] + (NDIM == 3 ? 4 : 0);
          const float c10 = fmaf(w[u][0], h[1] - h[0], h[0]);
          const float c11 = fmaf(w[u][0], h[3] - h[2], h[2]);
          const float c1 = fmaf(w[u][1], c11 - c10, c10);
          val = fmaf(w[u][NDIM - 1], c1 - val, val);
        }
        if (xb + 32 * u + lane < nx) {
          const float e = (val > 0.0f) ? val - t[u] : 0.0f;
          af = fmaf(e, e, af);
          const float e1 = e * f[u];
          const float e0 = e * (1.0f - f[u]);
          if (r == c0) {
#pragma unroll
            for (int k = 0; k < NDIM; k++) {
              ag[0][k] = fmaf(gk[u][k], e0, ag[0][k]);
              ag[1][k] = fmaf(gk[u][k], e1, ag[1][k]);
            }
          } else {
#pragma unroll
            for (int k = 0; k < NDIM; k++) {
              ag[1][k] = fmaf(gk[u][k], e0, ag[1][k]);
              ag[2][k] = fmaf(gk[u][k], e1, ag[2][k]);
            }
          }
        }
      }
    }
  }

  // FP32 butterfly across the warp, FP64 across warps (fixed order).
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    af += __shfl_xor_sync(0xffffffffu, af, o);
#pragma unroll
    for (int s = 0; s < 3; s++)
#pragma unroll
      for (int k = 0; k < NDIM; k++) ag[s][k] += __shfl_xor_sync(0xffffffffu, ag[s][k], o);
  }
  if (lane == 0) {
    sred[warp][0] = af;
#pragma unroll
    for (int s = 0; s < 3; s++)
#pragma unroll
      for (int k = 0; k < NDIM; k++) sred[warp][1 + s * NDIM + k] = ag[s][k];
  }
  __syncthreads();
  double* out = job.partials + (long long)tile * kPartialDoubles;
  if (threadIdx.x < 1 + 3 * NDIM) {
    double acc = 0.0;
    for (int w = 0; w < kEvalWarps; w++) acc += (double)sred[w][threadIdx.x];
    const int i = threadIdx.x;
    if (i == 0) {
      out[0] = acc;
    } else {
      const int s = (i - 1) / NDIM, k = (i - 1) % NDIM;
      out[2 + s * 3 + k] = acc;
    }
  } else if (threadIdx.x == 1 + 3 * NDIM) {
    out[1] = (double)c0;
    if (NDIM == 2) out[2 + 0 * 3 + 2] = out[2 + 1 * 3 + 2] = out[2 + 2 * 3 + 2] = 0.0;
  }
}

cudaError_t launch_eval4(const Job* jobs_dev, int n_jobs, int max_tiles, int n_dim, int frame_kind, bool ref_bf16,
                         int mb, cudaStream_t s);

cudaError_t launch_eval(const Job* jobs_dev, int n_jobs, int max_tiles, int n_dim, int frame_kind, bool ref_bf16,
                        cudaStream_t s, bool rows_multiple_of_4, int mb) {
  // One tile per CTA either way. Up to two tiles per SM a tile's latency counts: 168 tiles of 423 x 301 x 5
  // (FP32) 23.8 us in the general form, 16.1 in runs; beyond, the run form's registers halve the resident
  // warps: 4 FP32 frames of 511 x 511 x 16 168 us against 250 (8 mixed ones 302 against 288).
  constexpr long long kScalarFew = 296;
  if (rows_multiple_of_4) return launch_eval4(jobs_dev, n_jobs, max_tiles, n_dim, frame_kind, ref_bf16, mb, s);
  const dim3 grid(max_tiles, n_jobs);
  return dispatch_cfg(n_dim, frame_kind, ref_bf16, [&](auto c) {
    using C = decltype(c);
    if ((long long)max_tiles * n_jobs <= kScalarFew)
      eval_kernel<C::nd, typename C::F, typename C::R, true><<<grid, kEvalThreads, 0, s>>>(jobs_dev);
    else
      eval_kernel<C::nd, typename C::F, typename C::R, false><<<grid, kEvalThreads, 0, s>>>(jobs_dev);
    return cudaGetLastError();
  });
}

// ------------------------------------------------------------------ reductions -------------------

__global__ void __launch_bounds__(kSolveThreads) reduce_kernel(const Job* __restrict__ job) {
  const RefDev& R = job->R;
  __shared__ double s_f;
  cudaGridDependencySynchronize();  // the pass's partial sums
  reduce_partials(R, job->partials, &s_f, job->result + 1);
  if (threadIdx.x == 0) job->result[0] = s_f;
}

// reduce_partials for frames of many tiles, spread over CTAs: CTA c < nD of a frame takes control point c (its
// tiles' sums are brought into shared memory by all threads and added in tile order by one thread per
// component), CTA nD takes f. One CTA for everything waited for its own loads: 74 us of a step for
// 1024 x 1024 x 64 (16384 tiles, 512 to 768 of them per control point). f goes to *f_out, g to g_out.
constexpr int kWideThreads = 128, kWideStage = 512;
static_assert(kWideThreads == kReduceRuns, "f runs");
__device__ __forceinline__ void wide_reduce(const RefDev& R, const double* __restrict__ parts, double* f_out,
                                            double* g_out, double* stage) {
  const int tid = threadIdx.x;
  if ((int)blockIdx.x == R.nD) {
    double acc = 0.0;
    for (int t = tid; t < R.n_tiles; t += kReduceRuns * kReduceDepth) {
      double v[kReduceDepth];
#pragma unroll
      for (int u = 0; u < kReduceDepth; u++) {
        const int tt = t + u * kReduceRuns;
        v[u] = tt < R.n_tiles ? parts[(long long)tt * kPartialDoubles] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < kReduceDepth; u++) acc += v[u];
    }
    stage[tid] = acc;
    __syncthreads();
    if (tid < 32) {  // the tree of reduce_partials
      double a = (stage[tid] + stage[tid + 64]) + (stage[tid + 32] + stage[tid + 96]);
#pragma unroll
      for (int w = 16; w > 0; w >>= 1) a += __shfl_down_sync(0xffffffffu, a, w);
      if (tid == 0) *f_out = a;
    }
    __syncthreads();
    return;
  }
  const int c = blockIdx.x, nd = R.n_dim;
  const int4 tr = R.ctrl_tiles[c];
  double a = 0.0;
  for (int t0 = tr.x; t0 < tr.w; t0 += kWideStage) {
    const int n = min(kWideStage, tr.w - t0);
    __syncthreads();
    for (int i = tid; i < n; i += kWideThreads) {
      const int t = t0 + i, s = t < tr.y ? 2 : (t < tr.z ? 1 : 0);
      const double* p = parts + (long long)t * kPartialDoubles + 2 + s * 3;
      for (int k = 0; k < 3; k++) stage[k * kWideStage + i] = p[k];
    }
    __syncthreads();
    if (tid < nd) {
#pragma unroll 8
      for (int i = 0; i < n; i++) a += stage[tid * kWideStage + i];
    }
  }
  if (tid < nd) g_out[c * nd + tid] = a;
  __syncthreads();
}

// The frames of a step: f to work[0] (and of the paired start's rigid point to work[1]), g to gt (and p).
__global__ void __launch_bounds__(kWideThreads) wide_reduce_kernel(const Job* __restrict__ jobs,
                                                                   const int* __restrict__ active,
                                                                   const int* __restrict__ n_active, int bare) {
  __shared__ double stage[3 * kWideStage];
  if (active != nullptr && (int)blockIdx.y >= *n_active) return;
  const Job& job = jobs[active != nullptr ? active[blockIdx.y] : blockIdx.y];
  const RefDev& R = job.R;
  if ((int)blockIdx.x > R.nD || (R.n_tiles <= kWideTiles && !bare)) return;
  if (bare) {
    wide_reduce(R, job.partials, job.result, job.result + 1, stage);
    return;
  }
  const int phase = job.state->phase;
  if (phase == kPhaseDone || phase == kPhaseWaitWarm) return;
  wide_reduce(R, job.partials, job.work, job.gt, stage);
  if (phase == kPhaseStartPair) wide_reduce(R, job.partials2, job.work + 1, job.p, stage);
}

bool wide_reduction(int n_tiles) { return n_tiles > kWideTiles; }

cudaError_t launch_wide_reduce(const Job* jobs_dev, int n_jobs, int max_nD, cudaStream_t s, const int* active,
                               const int* n_active) {
  wide_reduce_kernel<<<dim3(max_nD + 1, n_jobs), kWideThreads, 0, s>>>(jobs_dev, active, n_active, 0);
  return cudaGetLastError();
}

cudaError_t launch_reduce(const Job* job_dev, int n_tiles, int nD, cudaStream_t s, bool overlap) {
  // A bare evaluation's reduction is a launch of its own either way: 1024 tiles (512 x 512 x 16) 65 us a call
  // with one CTA, 59 with many; a step's would be one launch more (271 -> 299 us a solve there).
  constexpr int kBareWideTiles = 768;
  return launch_reduce_form(job_dev, n_tiles > kBareWideTiles, nD, s, overlap);
}

cudaError_t launch_reduce_form(const Job* job_dev, bool wide, int nD, cudaStream_t s, bool overlap) {
  if (wide) {
    wide_reduce_kernel<<<dim3(nD + 1, 1), kWideThreads, 0, s>>>(job_dev, nullptr, nullptr, 1);
    return cudaGetLastError();
  }
  return launch_overlapped(reduce_kernel, dim3(1), dim3(kSolveThreads), 0, s, overlap, job_dev);
}

// ------------------------------------------------------------------ warped image -----------------

template <int NDIM, typename FT>
__global__ void __launch_bounds__(256) warp_kernel(const RefDev* __restrict__ Rp, const FT* __restrict__ fr,
                                                   long long fplane, int fpitch, const float4* __restrict__ dparams,
                                                   float invalid_value, float* __restrict__ out) {
  const RefDev& R = *Rp;
  const int nx = R.nx, ny = R.ny, nz = R.nz;
  extern __shared__ float4 sAll[];
  for (int i = threadIdx.x; i < R.nD * kDParamF4; i += blockDim.x) sAll[i] = dparams[i];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  for (int row = blockIdx.x * nwarps + warp; row < R.n_rows; row += gridDim.x * nwarps) {
    const RowDesc rd = R.rows[row];
    const int z = row / ny;
    const int y = row - z * ny;
    const bool flip = R.bidir && (y & 1);
    for (int x = lane; x < nx; x += 32) {
      const VoxelModel vm = voxel_model(rd, x, nx, flip, R.bidir != 0, R.dq);
      const int di = min(max(vm.di, 0), R.nD - 2);
      float v = sample<NDIM, FT>(fr, fplane, fpitch, sAll + di * kDParamF4, vm.f, x, y, z, nx, ny, nz);
      if (v == 0.0f) v = invalid_value;
      out[(long long)row * nx + x] = v;
    }
  }
}

constexpr size_t kMostSmem = 227 * 1024;  // all a CTA can have: 4842 control points

cudaError_t launch_warp(const RefDev* ref_dev, const RefDev& R, const void* frame, long long fplane, int fpitch,
                        int frame_kind, const float4* dparams, float invalid_value, float* out, cudaStream_t s) {
  int blocks = (R.n_rows + 7) / 8;
  if (blocks > 148 * 8) blocks = 148 * 8;
  const size_t smem = (size_t)R.nD * kDParamF4 * sizeof(float4);
  return dispatch_cfg(R.n_dim, frame_kind, false, [&](auto c) {
    using C = decltype(c);
    constexpr auto kern = warp_kernel<C::nd, typename C::F>;
    const cudaError_t e = allow_smem<kern>(smem, kMostSmem);
    if (e != cudaSuccess) return e;
    kern<<<blocks, 256, smem, s>>>(ref_dev, static_cast<const typename C::F*>(frame), fplane, fpitch, dparams,
                                   invalid_value, out);
    return cudaGetLastError();
  });
}

// ------------------------------------------------------------------ Hessian ----------------------

// Per tile and per storage-range slot s (range c0 + s): the 21 (3-D) or 10 (2-D) sums
//   A = sum v0 v0^T (upper), B = sum v1 v1^T (upper), C = sum v1 v0^T
// with v0 = float(grad * float(1 - Df)), v1 = float(grad * Df) and Df exact
// (FrameWarper.cpp:258-259, 319-342), over the voxels of the range that are not its last.
constexpr int kHessTerms = 21;

// The block tree of one CTA's 256 values of a term: run t takes run t + w, w = 128, 64, ..., 1, by one warp.
__device__ __forceinline__ double tree256(const double* v, int lane) {
  double a = ((v[lane] + v[lane + 128]) + (v[lane + 64] + v[lane + 192])) +
             ((v[lane + 32] + v[lane + 160]) + (v[lane + 96] + v[lane + 224]));
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) a += __shfl_down_sync(0xffffffffu, a, w);
  return a;
}

// What bounded it were the reductions, 21 block trees of eight barriers each, and the second slot's pass
// over tiles that have only one range: the trees are now one warp's each after one barrier (the same
// order), and an empty slot is written as zeros. 512 x 512 x 16: 134 -> 63 us, now the FP64 division and
// the 21 conversions and sums of every voxel.
template <int NDIM>
__global__ void __launch_bounds__(256) hessian_tile_kernel(const RefDev* __restrict__ Rp, double pd, double ild,
                                                           double ifd, double stack, double* __restrict__ parts) {
  const RefDev& R = *Rp;
  const int tile = blockIdx.x;
  const int slot = blockIdx.y;
  const int nx = R.nx;
  const int row_begin = tile * R.tile_rows;
  const int row_end = min(row_begin + R.tile_rows, R.n_rows);
  const int c0 = R.tile_c0[tile];
  const double nDm1 = (double)(R.nD - 1);
  constexpr int NU = NDIM * (NDIM + 1) / 2;
  constexpr int kTerms = 2 * NU + NDIM * NDIM;
  double* out = parts + ((long long)tile * 2 + slot) * kHessTerms;
  if (slot == 1) {  // the ranges do not decrease: the tile has a second one if its last row reaches it
    const RowDesc rl = R.rows[row_end - 1];
    const int last = R.bidir ? rl.r0 + (rl.xr < nx ? 1 : 0) : rl.di0 + (rl.xdi < nx ? 1 : 0);
    if (last == c0) {
      if (threadIdx.x < kTerms) out[threadIdx.x] = 0.0;
      return;
    }
  }
  double acc[kTerms];
#pragma unroll
  for (int i = 0; i < kTerms; i++) acc[i] = 0.0;
  for (int row = row_begin; row < row_end; row++) {
    const RowDesc rd = R.rows[row];
    const int z = rd.z, y = rd.y;
    const bool flip = R.bidir && (y & 1);
    for (int x = threadIdx.x; x < nx; x += blockDim.x) {
      const int r = R.bidir ? rd.r0 + (x >= rd.xr ? 1 : 0) : rd.di0 + (x >= rd.xdi ? 1 : 0);
      if (r - c0 != slot || x == rd.xlast) continue;
      const int xs = flip ? nx - 1 - x : x;
      // t = z*interframe + y*interline + x*pixel; q = t / stack * (nD - 1) (FrameWarper.cpp:258-259)
      const double t = __dadd_rn(__dadd_rn(__dmul_rn((double)z, ifd), __dmul_rn((double)y, ild)), __dmul_rn((double)xs, pd));
      const double q = __dmul_rn(__ddiv_rn(t, stack), nDm1);
      const float df = (float)(q - floor(q));
      const float w0 = __fsub_rn(1.0f, df);
      const long long p = (long long)row * nx + x;
      float g[NDIM];
      g[0] = R.gx32[p];
      g[1] = R.gy32[p];
      if (NDIM == 3) g[NDIM - 1] = R.gz32[p];
      float v0[NDIM], v1[NDIM];
#pragma unroll
      for (int k = 0; k < NDIM; k++) {
        v0[k] = __fmul_rn(g[k], w0);
        v1[k] = __fmul_rn(g[k], df);
      }
      int u = 0;
#pragma unroll
      for (int a = 0; a < NDIM; a++)
#pragma unroll
        for (int b = a; b < NDIM; b++, u++) {
          acc[u] += (double)__fmul_rn(v0[a], v0[b]);
          acc[NU + u] += (double)__fmul_rn(v1[a], v1[b]);
        }
#pragma unroll
      for (int a = 0; a < NDIM; a++)
#pragma unroll
        for (int b = 0; b < NDIM; b++) acc[2 * NU + a * NDIM + b] += (double)__fmul_rn(v1[a], v0[b]);
    }
  }
  __shared__ double sacc[kTerms][256];
#pragma unroll
  for (int i = 0; i < kTerms; i++) sacc[i][threadIdx.x] = acc[i];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = warp; i < kTerms; i += 8) {
    const double a = tree256(sacc[i], lane);
    if (lane == 0) out[i] = a;
  }
}

// Hd[c] = sum_t A(t, c - c0_t) + B(t, c - 1 - c0_t);  Hl[c] = sum_t C(t, c - 1 - c0_t), one thread per entry,
// each in tile order (first the range c, then c - 1: at most one of a tile's two slots is either) with
// the loads of eight tiles in flight (one thread per control point: 138 us for 32 of them, now 14).
template <int NDIM>
__global__ void __launch_bounds__(64) hessian_reduce_kernel(const RefDev* __restrict__ Rp,
                                                            const double* __restrict__ parts, double* __restrict__ Hd,
                                                            double* __restrict__ Hl) {
  const RefDev& R = *Rp;
  constexpr int NU = NDIM * (NDIM + 1) / 2, NN = NDIM * NDIM;
  const int c = blockIdx.x;
  const int4 tr = R.ctrl_tiles[c];
  if (threadIdx.x >= NU + NN) return;
  const bool diag = threadIdx.x < NU;
  const int i = diag ? threadIdx.x : threadIdx.x - NU;
  double h = 0.0;
  // tiles that start at range c - 2 hold range c - 1 in slot 1; at c - 1, range c - 1 in slot 0 and range c in
  // slot 1; at c, range c in slot 0
  constexpr int kDepth = 8;
  for (int t = tr.x; t < tr.w; t += kDepth) {
    double v[kDepth][2];
#pragma unroll
    for (int u = 0; u < kDepth; u++) {
      const int tt = min(t + u, tr.w - 1);
      const double* p0 = parts + (long long)tt * 2 * kHessTerms;
      const double* p1 = p0 + kHessTerms;
      if (diag) {
        v[u][0] = tt < tr.y ? 0.0 : (tt < tr.z ? p0[NU + i] : p0[i]);
        v[u][1] = tt < tr.y ? p1[NU + i] : (tt < tr.z ? p1[i] : 0.0);
      } else {
        v[u][0] = tt >= tr.y && tt < tr.z ? p0[2 * NU + i] : 0.0;
        v[u][1] = tt < tr.y ? p1[2 * NU + i] : 0.0;
      }
    }
#pragma unroll
    for (int u = 0; u < kDepth; u++)
      if (t + u < tr.w) {
        h += v[u][0];
        h += v[u][1];
      }
  }
  if (diag) {
    int a = 0, b = i;
    while (b >= NDIM - a) {  // entry i of the upper triangle, row by row
      b -= NDIM - a;
      a++;
    }
    b += a;
    Hd[c * NN + a * NDIM + b] = h;
    Hd[c * NN + b * NDIM + a] = h;
  } else {
    Hl[c * NN + i] = h;
  }
}

cudaError_t launch_hessian(const RefDev* ref_dev, const RefDev& R, const double* scan4, double* tile_parts, double* Hd,
                           double* Hl, cudaStream_t s) {
  dim3 grid(R.n_tiles, 2);
  if (R.n_dim == 3) {
    hessian_tile_kernel<3><<<grid, 256, 0, s>>>(ref_dev, scan4[0], scan4[1], scan4[2], scan4[3], tile_parts);
    hessian_reduce_kernel<3><<<R.nD, 64, 0, s>>>(ref_dev, tile_parts, Hd, Hl);
  } else {
    hessian_tile_kernel<2><<<grid, 256, 0, s>>>(ref_dev, scan4[0], scan4[1], scan4[2], scan4[3], tile_parts);
    hessian_reduce_kernel<2><<<R.nD, 64, 0, s>>>(ref_dev, tile_parts, Hd, Hl);
  }
  return cudaGetLastError();
}

// ------------------------------------------------------------------ batched-solve bookkeeping ----

// The first list of a solve or of a server's graph launch (later ones come from the solve steps).
__global__ void __launch_bounds__(256) compact_kernel(const Job* __restrict__ jobs, ActiveOut out) {
  if (threadIdx.x == 0 && out.rounds != nullptr) *out.rounds = 0;
  compact_block(jobs, out);
}

cudaError_t launch_compact(const Job* jobs_dev, const ActiveOut& out, cudaStream_t s) {
  compact_kernel<<<1, 256, 0, s>>>(jobs_dev, out);
  return cudaGetLastError();
}

// Zero start of a batched solve (the host-side init of the single-frame driver, on the device).
__global__ void activate_kernel(const Job* __restrict__ jobs, const Activation* __restrict__ recs, int* busy) {
  const Activation r = recs[blockIdx.x];
  const Job& j = jobs[r.job];
  const RefDev& R = j.R;
  for (int i = threadIdx.x; i < R.P; i += blockDim.x) {
    j.x[i] = 0.0;
    j.g[i] = 0.0;
    j.p[i] = 0.0;
    j.gt[i] = 0.0;
  }
  for (int i = threadIdx.x; i < R.nD * kDParamF4; i += blockDim.x) j.dparams[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  double rigid[3];
  bool nonzero = false;
  for (int c = 0; c < 3; c++) {
    rigid[c] = (c < R.n_dim) ? r.rigid[c] : 0.0;
    nonzero = nonzero || rigid[c] != 0.0;
  }
  const bool pair = r.pair != 0 && nonzero;
  if (pair) write_const_dparams(j.dparams2, R.nD, R.n_dim, rigid, threadIdx.x, blockDim.x);
  if (threadIdx.x == 0) {
    FrameState S{};
    S.phase = pair ? kPhaseStartPair : kPhaseStartZero;
    S.max_iter = r.max_iter > 0 ? r.max_iter : 100;
    S.warm = r.warm;
    S.warm_seq = r.warm_seq;
    S.warm_need = r.warm_need;
    S.seq = r.seq;
    S.use_warm = (r.use_warm != 0 && r.warm != nullptr && r.warm_seq != nullptr) ? 1 : 0;
    for (int c = 0; c < 3; c++) S.rigid[c] = r.rigid[c];
    if (R.n_dim == 2) S.rigid[2] = 0.0;
    *j.state = S;
    busy[r.job] = 1;
  }
}

// Start of the aligner's batched solve straight from the phase-correlation peaks in device memory, so
// that the host need not read them first: job i takes peak i (flat index of the correlation surface
// of a cnz x cny x cnx volume), unravels and wraps it like unravel_shift (VolumePhaseCorrelator.cpp:
// 94-103), scales x and y by the binning (FrameWarpAligner.cpp:186-188) and sets the zero start, or the
// paired start when `pair` and the shift is not zero.
__global__ void activate_peaks_kernel(const Job* __restrict__ jobs, const long long* __restrict__ peaks, int cnx,
                                      int cny, int cnz, int binning, int max_iter, int pair) {
  const Job& j = jobs[blockIdx.x];
  const RefDev& R = j.R;
  const long long idx = peaks[blockIdx.x];
  long long x = idx % cnx, y = (idx / cnx) % cny, z = idx / ((long long)cnx * cny);
  if (x > cnx / 2) x -= cnx;
  if (y > cny / 2) y -= cny;
  if (z > cnz / 2) z -= cnz;
  double rigid[3] = {(double)x * binning, (double)y * binning, R.n_dim == 3 ? (double)z : 0.0};
  bool nonzero = false;
  for (int c = 0; c < R.n_dim; c++) nonzero = nonzero || rigid[c] != 0.0;
  const bool paired = pair != 0 && nonzero;
  for (int i = threadIdx.x; i < R.P; i += blockDim.x) {
    j.x[i] = 0.0;
    j.g[i] = 0.0;
    j.p[i] = 0.0;
    j.gt[i] = 0.0;
  }
  for (int i = threadIdx.x; i < R.nD * kDParamF4; i += blockDim.x) j.dparams[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (paired) write_const_dparams(j.dparams2, R.nD, R.n_dim, rigid, threadIdx.x, blockDim.x);
  if (threadIdx.x == 0) {
    FrameState S{};
    S.phase = paired ? kPhaseStartPair : kPhaseStartZero;
    S.max_iter = max_iter > 0 ? max_iter : 100;
    for (int c = 0; c < 3; c++) S.rigid[c] = rigid[c];
    *j.state = S;
  }
}

cudaError_t launch_activate_peaks(const Job* jobs_dev, int n, const long long* peaks, int cnx, int cny, int cnz,
                                  int binning, int max_iter, bool pair, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  activate_peaks_kernel<<<n, 128, 0, s>>>(jobs_dev, peaks, cnx, cny, cnz, binning, max_iter, pair ? 1 : 0);
  return cudaGetLastError();
}

// The zero start of one frame's own solve (kPhaseStartZero, then the rigid shift if it is not zero).
struct RigidShift {
  double v[3];
};
__global__ void start_kernel(const Job* __restrict__ job, RigidShift rigid, int max_iter) {
  const Job& j = *job;
  const RefDev& R = j.R;
  for (int i = threadIdx.x; i < R.P; i += blockDim.x) {
    j.x[i] = 0.0;
    j.g[i] = 0.0;
    j.p[i] = 0.0;
    j.gt[i] = 0.0;
  }
  for (int i = threadIdx.x; i < R.nD * kDParamF4; i += blockDim.x) j.dparams[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (threadIdx.x == 0) {
    FrameState S{};
    S.phase = kPhaseStartZero;
    S.max_iter = max_iter;
    for (int c = 0; c < 3; c++) S.rigid[c] = c < R.n_dim ? rigid.v[c] : 0.0;
    *j.state = S;
  }
}

cudaError_t launch_start(const Job* job_dev, const double* rigid, int max_iter, cudaStream_t s) {
  RigidShift r{{0.0, 0.0, 0.0}};
  for (int c = 0; c < 3 && rigid; c++) r.v[c] = rigid[c];
  start_kernel<<<1, 128, 0, s>>>(job_dev, r, max_iter);
  return cudaGetLastError();
}

cudaError_t launch_activate(const Job* jobs_dev, const Activation* recs, int n, int* busy, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  activate_kernel<<<n, 128, 0, s>>>(jobs_dev, recs, busy);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ smoothStack ------------------

// FrameWarpAligner::smoothStack (FrameWarpAligner.cpp:46-64): per plane, cv::GaussianBlur with sigma
// along x and 1 along y, BORDER_REFLECT_101, float arithmetic (products and sums rounded one by one):
// a row pass summing taps in kernel order, then a column pass in the symmetric form.
__device__ __forceinline__ int reflect101(int p, int n) {
  if (n == 1) return 0;
  while (p < 0 || p >= n) {
    if (p < 0) p = -p;
    if (p >= n) p = 2 * n - 2 - p;
  }
  return p;
}

__global__ void smooth_rows_kernel(const void* __restrict__ in, int in_t, int ny, int nx, long long n,
                                   const float* __restrict__ k, int nk, float* __restrict__ out) {
  const int r = nk / 2;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % nx);
    const long long row = i - x;
    float s = __fmul_rn(k[0], load_any(in, in_t, row + reflect101(x - r, nx)));
    for (int t = 1; t < nk; t++) s = __fadd_rn(s, __fmul_rn(k[t], load_any(in, in_t, row + reflect101(x + t - r, nx))));
    out[i] = s;
  }
}

__global__ void smooth_cols_kernel(const float* __restrict__ in, int ny, int nx, long long n,
                                   const float* __restrict__ k, int nk, float* __restrict__ out) {
  const int r = nk / 2;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % nx);
    const long long py = i / nx;
    const int y = (int)(py % ny);
    const long long plane = (py - y) * nx;
    float s = __fmul_rn(k[r], in[i]);
    for (int t = 1; t <= r; t++) {
      const float a = in[plane + (long long)reflect101(y - t, ny) * nx + x];
      const float b = in[plane + (long long)reflect101(y + t, ny) * nx + x];
      s = __fadd_rn(s, __fmul_rn(k[r + t], __fadd_rn(a, b)));
    }
    out[i] = s;
  }
}

cudaError_t launch_smooth(const void* in, fa_dtype in_type, int nz, int ny, int nx, const float* kx, int nkx,
                          const float* ky, int nky, float* tmp, float* out, cudaStream_t s) {
  const long long n = (long long)nz * ny * nx;
  long long blocks = (n + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  smooth_rows_kernel<<<(int)blocks, 256, 0, s>>>(in, (int)in_type, ny, nx, n, kx, nkx, tmp);
  smooth_cols_kernel<<<(int)blocks, 256, 0, s>>>(tmp, ny, nx, n, ky, nky, out);
  return cudaGetLastError();
}

}  // namespace fa
