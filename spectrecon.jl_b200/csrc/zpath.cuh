// zpath.cuh -- the fused SPECT projector pair on z-fastest layouts (sm_100a),
// for the common case: cached attenuation, separable (rank-1) PSF planes.
//
// Layouts (float32, z fastest; nzp = nz rounded up to 16; every entry with
// z >= nz is zero):
//   IZ    [L][L][nzp]        image on the zero-padded rotation grid
//                            (L = nx + 2 pad, pad = ceil(1 + nx sqrt2/2 - nx/2),
//                            src/plan-rotate.jl:56): voxel (x, y, z) at
//                            ((y + pad) L + x + pad) nzp + z.  The ring is
//                            zero, so bilinear taps need no bounds tests.
//   ATT   [view][y][x][nzp]  attenuation exp(-dy (sum_{j<y} mu_j + mu_y/2)) on
//                            the view's rotated grid (src/project.jl:103-113)
//   T     [slot][y][x][nzp]  adjoint planes att .* conv_adj(view) of a group
//   views [slot][nz][nx]     the reference's views[nx, nz, nview], unchanged
//
// k_zfwd   project! (src/project.jl:77-135): the blocks share one flat walk
//          over the planes (slot, y) of a group; per plane a block gathers the
//          rotated image (imrotate!, src/rotatez.jl:331-362) column by column
//          from IZ, times the attenuation, straight into the z pass's pair
//          lines; then the z pass and the x pass of the replicate-boundary
//          convolution that fft_conv! computes (src/fft_convolve.jl:33-55).
//          A plane's x outputs are summed in registers and added to the
//          block's partial view of the slot (the depth sum,
//          src/project.jl:127-130); k_reduce_parts sums the partials in block
//          order.  The rotated volume never leaves the SM.
// k_zadj   backproject! (src/backproject.jl:69-124), convolution half, on row
//          tiles of a view: per plane the z pass and the x pass of
//          fft_conv_adj! (src/fft_convolve.jl:82-130), times the attenuation,
//          stored as T.
// The forward of planes too large for k_zfwd's shared memory is in zstrip.cuh
// (same layouts and passes, over plane tiles).
// k_zrot_adj  imrotate_adj! (src/rotatez.jl:390-416) and the view sum
//          (src/backproject.jl:146-153): output-stationary gather.  Every image
//          column sums, over the views in order, the weights of the
//          rotated-grid points whose footprint covers it, listed once per
//          column and slot in shared memory: the exact transpose of the
//          forward sampling, without atomics.  The EM update
//          (src/ml-os-em.jl:111-126) is its epilogue.
// ONE: the three shears of :one as eight taps of IZ (one_line).
//
// Convolution passes.  fft_conv! equals the replicate-boundary convolution
// out[i] = sum_{m<p} w[m] in[clamp(i - h + m)] with the reversed factor w
// (the plan factors each PSF plane as a[d] b[e]).  Here two input lines sit
// interleaved and zero-padded in shared memory, one element f2 = (line a,
// line b), and a task of W = 8 or 16 consecutive outputs of both runs packed
// FMAs (fma.rn.f32x2): half the issue slots of a line at a time, which is what
// bounds these loops next to their index and shared-memory work (63.4 against
// 48.9 TFLOP/s beside one integer operation per two FMAs).  Data start at an offset
// D0 = h rounded up to 4 and the weights are shifted right by D0 - h, so the
// window is read in 16-byte-aligned pieces; the clamped
// boundary is added as tail terms: the edge value times EL[i] =
// sum_{m < h - i} w[m] (i < h) or ER[n-1-i] = sum_{m > h + n-1-i} w[m]
// (i > n-1-h).  The adjoint passes are the zero-padded correlations with the
// factors themselves plus the folded padding at the two ends (cL_k, cR_k:
// sums of the factor beyond k), as the reference's padding adjoint does.
// The plan zeroes the outer taps of each factor whose summed magnitude per
// side is within 2^-27 of the factor's (below Float32 resolution; a narrow
// Gaussian plane keeps a few of its p taps) and cuts the rows to the widest
// support that is left; every table, tails and folds included, comes from
// those factors, and per plane and pass a range gives the 4-tap blocks that
// hold the kept taps: only those are run.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "bulk_copy.cuh"
#include "zpath_api.h"

namespace spect {

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
// four floats as two packed pairs; ldp_cs: read once (the image that the
// gather reads again and again stays in L2 instead)
__device__ __forceinline__ ulonglong2 ldp(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }
__device__ __forceinline__ ulonglong2 ldp_cs(const float* p) { return __ldcs(reinterpret_cast<const ulonglong2*>(p)); }
// q = t / n for 0 <= t < 2^20, 1 <= n <= 4096, with r = 1/n rounded to float:
// (t + 1/2) / n is at least 1/(2n) from an integer, far above the rounding
// error of (t + 1/2) * r, so truncation gives the exact quotient
__device__ __forceinline__ int zdiv(int t, float r) { return (int)(((float)t + 0.5f) * r); }

// ------------------------------------------------------------------------
// Pair passes: one task runs W consecutive outputs of TWO lines whose values
// are interleaved in shared memory (element i = (a[i], b[i])), so every FMA
// is a packed FFMA2 (two lines a lane) and an output pair needs no register
// moves.  The FP32 pipe takes an FFMA2 every other cycle, which leaves every
// second issue slot to the loads and address arithmetic (measured: with one
// integer operation per two FMAs a chain of FFMA2 keeps 63 TFLOP/s where
// FFMA falls to 49).  Weights are stored twice ((w, w)); taps run in blocks of
// 4, m in [4 b4, 4 b4 + 4 n4) (n4 <= 18), in ascending order for every output:
// the same result for every W, and for either lane as for a single line.
using f2 = unsigned long long;  // two packed floats in one 64-bit register (pair)
__device__ __forceinline__ f2 pack2(float a, float b) {
  f2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float2 unpack2(f2 d) {
  float2 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(d));
  return v;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

template <int W>
__device__ __forceinline__ void zpass2(const f2* __restrict__ w, int b4, int n4, const f2* line, f2 (&o)[W]) {
  const ulonglong2* w4 = reinterpret_cast<const ulonglong2*>(w + 4 * b4);
  const ulonglong2* l4 = reinterpret_cast<const ulonglong2*>(line + 4 * b4);
  f2 e[W + 4 * 18];
#pragma unroll
  for (int i = 0; i < W / 2; ++i) {
    const ulonglong2 q = l4[i];
    e[2 * i] = q.x;
    e[2 * i + 1] = q.y;
  }
#pragma unroll
  for (int k = 0; k < 18; ++k) {
    if (k >= n4) break;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const ulonglong2 q = l4[2 * k + W / 2 + i];
      e[4 * k + W + 2 * i] = q.x;
      e[4 * k + W + 2 * i + 1] = q.y;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const ulonglong2 q = w4[2 * k + h];
#pragma unroll
      for (int j = 0; j < W; ++j) o[j] = fma2(q.x, e[4 * k + 2 * h + j], o[j]);
#pragma unroll
      for (int j = 0; j < W; ++j) o[j] = fma2(q.y, e[4 * k + 2 * h + 1 + j], o[j]);
    }
  }
}

// sum_{k < n} c[k] v[step k] of a pair of lines: four partial sums over k mod
// 4, added as (s0 + s1) + (s2 + s3), so a round waits for one load latency
__device__ __forceinline__ f2 zfold2(const float* c, const f2* v, int step, int n) {
  f2 s[4] = {0, 0, 0, 0};
  int k = 0;
  for (; k + 4 <= n; k += 4)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] = fma2(pack2(c[k + j], c[k + j]), v[step * (k + j)], s[j]);
#pragma unroll
  for (int j = 0; j < 3; ++j)
    if (k + j < n) s[j] = fma2(pack2(c[k + j], c[k + j]), v[step * (k + j)], s[j]);
  return add2(add2(s[0], s[1]), add2(s[2], s[3]));
}

// the outputs (2 m, 2 m + 1) of a task over the pair (a, b) of lines, as two
// elements (line pairs of the other direction): (o[2m].a, o[2m+1].a),
// (o[2m].b, o[2m+1].b)
__device__ __forceinline__ float4 zturn(f2 p, f2 q) {
  const float2 u = unpack2(p), v = unpack2(q);
  return make_float4(u.x, v.x, u.y, v.y);
}

// four z of a rotated, attenuated column as two packed pairs: the four taps at
// p, p + nzp, p + Lz, p + Lz + nzp with the doubled weights w4[0] = (w00 w00
// w10 w10), w4[1] = (w01 w01 w11 w11), times the attenuation at att
__device__ __forceinline__ void zsample4(const float* p, int nzp, size_t Lz, const float4* w4, const float* att, f2& lo,
                                         f2& hi) {
  const ulonglong2 t0 = ldp(p), t1 = ldp(p + nzp), t2 = ldp(p + Lz), t3 = ldp(p + Lz + nzp);
  const ulonglong2 at = ldp_cs(att);
  const ulonglong2 wa = reinterpret_cast<const ulonglong2*>(w4)[0], wb = reinterpret_cast<const ulonglong2*>(w4)[1];
  lo = mul2(fma2(wb.y, t3.x, fma2(wb.x, t2.x, fma2(wa.y, t1.x, mul2(wa.x, t0.x)))), at.x);
  hi = mul2(fma2(wb.y, t3.y, fma2(wb.x, t2.y, fma2(wa.y, t1.y, mul2(wa.x, t0.y)))), at.y);
}

// the clamped boundary of a forward task's outputs i0 .. i0 + W - 1 of a line
// of n elements with edge values e0, e1: + EL[i] e0 (i < h), + ER[n-1-i] e1
template <int W>
__device__ __forceinline__ void zclamp(f2 (&o)[W], const float* EL, const float* ER, int h, int i0, int n, f2 e0, f2 e1) {
  if (i0 < h) {
#pragma unroll
    for (int k = 0; k < W; ++k)
      if (i0 + k < h) o[k] = fma2(pack2(EL[i0 + k], EL[i0 + k]), e0, o[k]);
  }
  if (i0 + W > n - h) {
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const int kk = n - 1 - i0 - k;
      if (kk >= 0 && kk < h) o[k] = fma2(pack2(ER[kk], ER[kk]), e1, o[k]);
    }
  }
}

// a task's outputs (rows z, z + 1, columns x0 ..) into a partial view [nz][nx]
template <int X>
__device__ __forceinline__ void zstore_part(float* part, const f2 (&acc)[X], int nx, int nz, int z, int x0) {
  float* q = part + (size_t)z * nx + x0;
  const bool two = z + 1 < nz;
  if (nx % 4 == 0) {
#pragma unroll
    for (int k = 0; k < X; k += 4)
      if (x0 + k < nx) {
        const float4 u = zturn(acc[k], acc[k + 1]), w = zturn(acc[k + 2], acc[k + 3]);
        st4(q + k, make_float4(u.x, u.y, w.x, w.y));
        if (two) st4(q + nx + k, make_float4(u.z, u.w, w.z, w.w));
      }
  } else {
#pragma unroll
    for (int k = 0; k < X; ++k)
      if (x0 + k < nx) {
        const float2 u = unpack2(acc[k]);
        q[k] = u.x;
        if (two) q[nx + k] = u.y;
      }
  }
}

// programmatic dependent launch: wait until the kernels before this one in the
// stream have completed, then let the next one's blocks start where room is
// (they wait here in turn).  What a kernel does before it touches nothing
// that an earlier kernel writes or reads: its own shared memory, the plan's
// constant tables, the view list.  Data that such kernels exchange is read by
// plain loads: a pointer marked __restrict__ or a read-only load could be
// moved above the wait.
__device__ __forceinline__ void grid_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// fetch the 128-byte line of p into L2
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// fetch `bytes` (a multiple of 16, p 16-byte aligned) into L2
__device__ __forceinline__ void prefetch_l2_bulk(const void* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// 16-byte asynchronous copy global -> shared of the calling thread, and the
// wait for all of its copies
__device__ __forceinline__ void cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ------------------------------------------------------------------------
// Layout changes between the caller's image [z][y][x] and IZ.
// k_to_iz: IZ interior (and its z padding) from img; grid (ceil(nx/32),
// ny, ceil(nzp/32)), block (32, 8).
__global__ void __launch_bounds__(256) k_to_iz(ZGeom g, const float* img, float* iz) {
  __shared__ float tile[32][33];
  const int x0 = blockIdx.x * 32, y = blockIdx.y, z0 = blockIdx.z * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
  grid_wait();
  for (int k = ty; k < 32; k += 8) {  // tile[z][x], coalesced over x
    const int z = z0 + k, x = x0 + tx;
    tile[k][tx] = (z < g.nz && x < g.nx) ? img[((size_t)z * g.ny + y) * g.nx + x] : 0.f;
  }
  __syncthreads();
  for (int k = ty; k < 32; k += 8) {  // IZ column x, coalesced over z
    const int x = x0 + k, z = z0 + tx;
    if (x < g.nx && z < g.nzp) iz[((size_t)(y + g.pad) * g.L + x + g.pad) * g.nzp + z] = tile[tx][k];
  }
}

// k_from_iz: dst (caller layout) from the IZ interior.  mode 0: dst = v;
// 1: dst = v, zeros -> +Inf (EM sensitivity, src/ml-os-em.jl:111-114);
// 2: dst = dst * (v / asum) (EM update, asum in the caller layout).
__global__ void __launch_bounds__(256) k_from_iz(ZGeom g, const float* iz, float* dst, const float* asum,
                                                 int mode) {
  __shared__ float tile[32][33];
  const int x0 = blockIdx.x * 32, y = blockIdx.y, z0 = blockIdx.z * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
  grid_wait();
  for (int k = ty; k < 32; k += 8) {  // tile[x][z], coalesced over z
    const int x = x0 + k, z = z0 + tx;
    tile[k][tx] = (x < g.nx && z < g.nz) ? iz[((size_t)(y + g.pad) * g.L + x + g.pad) * g.nzp + z] : 0.f;
  }
  __syncthreads();
  for (int k = ty; k < 32; k += 8) {  // caller row (z, y), coalesced over x
    const int z = z0 + k, x = x0 + tx;
    if (z < g.nz && x < g.nx) {
      const size_t o = ((size_t)z * g.ny + y) * g.nx + x;
      float v = tile[tx][k];
      if (mode == 1 && v == 0.f) v = __int_as_float(0x7f800000);
      if (mode == 2) v = dst[o] * (v / asum[o]);
      dst[o] = v;
    }
  }
}

// k_t_to_z: adjoint planes of the direct split kernel ([plane][nz][nx], plane =
// slot * ny + y) into the z-fastest T layout ([plane][nx][nzp], zeros for
// z >= nz) that k_zrot_adj reads, multiplied by the attenuation when the
// convolution has not applied it (att non-null, the same product as the
// reference's a_y .* conv_adj); grid (ceil(nx/32), planes, ceil(nzp/32)),
// block (32, 8).
__global__ void __launch_bounds__(256) k_t_to_z(ZGeom g, const float* __restrict__ src, float* __restrict__ dst,
                                                const float* __restrict__ att, const int* __restrict__ vidx) {
  __shared__ float tile[32][33];
  const int x0 = blockIdx.x * 32, pl = blockIdx.y, z0 = blockIdx.z * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const float* s = src + (size_t)pl * g.nz * g.nx;
  float* d = dst + (size_t)pl * g.nx * g.nzp;
  // att (split layout [view][y][z][x]) given: the planes are not premultiplied yet
  const float* av = att ? att + ((size_t)vidx[pl / g.ny] * g.ny + pl % g.ny) * g.nz * g.nx : nullptr;
  for (int k = ty; k < 32; k += 8) {  // tile[z][x], coalesced over x
    const int z = z0 + k, x = x0 + tx;
    const size_t o = (size_t)z * g.nx + x;
    tile[k][tx] = (z < g.nz && x < g.nx) ? (av ? __fmul_rn(av[o], s[o]) : s[o]) : 0.f;
  }
  __syncthreads();
  for (int k = ty; k < 32; k += 8) {  // column x, coalesced over z
    const int x = x0 + k, z = z0 + tx;
    if (x < g.nx && z < g.nzp) d[(size_t)x * g.nzp + z] = tile[tx][k];
  }
}

// ------------------------------------------------------------------------
// Geometry of rotated-grid point (x, y) of a view, with the forward
// sampling's products and sums in the same order and rounding
// (RotPos::pos): the IZ offset of its lower-left tap and the four bilinear
// weights (w00, w10, w01, w11); theta == 0 copies (the reference's forward
// shortcut).  Every sample of the cropped grid lies inside the padded grid;
// a point outside it (impossible for finite angles) contributes nothing.
__device__ __forceinline__ void zgeo(const ZGeom& g, float cs, float sn, bool ident, int x, int y, float4& w,
                                     int& off) {
  int j1 = x, j2 = y;
  w = make_float4(1.f, 0.f, 0.f, 0.f);
  if (!ident) {
    const float di = __fsub_rn((float)x, g.c0), dj = __fsub_rn((float)y, g.c0);
    const float s1 = __fadd_rn(g.c0, __fsub_rn(__fmul_rn(cs, di), __fmul_rn(sn, dj)));
    const float s2 = __fadd_rn(g.c0, __fadd_rn(__fmul_rn(sn, di), __fmul_rn(cs, dj)));
    const float f1 = floorf(s1), f2 = floorf(s2);
    const float t1 = __fsub_rn(s1, f1), t2 = __fsub_rn(s2, f2);
    const float u1 = __fsub_rn(1.0f, t1), u2 = __fsub_rn(1.0f, t2);
    j1 = (int)f1;
    j2 = (int)f2;
    w = make_float4(__fmul_rn(u1, u2), __fmul_rn(t1, u2), __fmul_rn(u1, t2), __fmul_rn(t1, t2));
    if (j1 < -g.pad || j1 > g.nx + g.pad - 2 || j2 < -g.pad || j2 > g.nx + g.pad - 2) {
      j1 = j2 = 0;
      w = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  off = ((j2 + g.pad) * g.L + j1 + g.pad) * g.nzp;
}

// The three shears of imrotate! :one (src/rotatez.jl:240-322) as one gather.
// A line's shear is out(q) = lo in(q + off) + (1 - lo) in(q + off + 1)
// (linearinterp!, src/rotatez.jl:21-51: positions in Float64), so an output
// point of the cropped grid is the sum of 2 x 2 x 2 taps of the padded image.
// The index clamps of linearinterp! never reach such a point with a nonzero
// value: its own x shear stays inside the padded grid, and a clamped y or
// first x shear reads the grid's zero ring.  Weights are products in Float64,
// rounded once.
// Measured, 96x96x48, 15 of 90 views, 21 taps, forward and adjoint: 1437 us of
// kernels with the line-by-line passes (k_rot1_fwd, k_rot1_adj, the convolution
// and attenuation kernels around them), 100 us here.
struct OneLine {
  double lo;
  int off;
};
__device__ __forceinline__ OneLine one_line(int i, double t, int L) {  // 0-based line i
  const double s = (i + 1 - (L + 1) / 2.0) * t + 1;
  const double c = ceil(s);
  return OneLine{c - s, s <= 1 ? (int)c - 2 : (int)floor(s) - 1};
}
// taps of rotated-grid point (x, y): off[k], off[k] + delta with the weights
// w[2 k], w[2 k + 1]; delta = one_delta(view): the next element along the
// first shear's lines, in IZ, after rot_f90! by m
__device__ __forceinline__ int one_delta(const ZGeom& g, int m) {
  return m == 0 ? g.nzp : m == 1 ? -g.L * g.nzp : m == 2 ? -g.nzp : g.L * g.nzp;
}
__device__ __forceinline__ void one_geo(const ZGeom& g, const Rot1View& V, int x, int y, float (&w)[8], int (&off)[4]) {
  const int L = g.L, a = g.pad + x, b = g.pad + y, m = V.mode == 0 ? 0 : V.m;
  auto pos = [&](int p, int q) {  // IZ column of element (p, q) after rot_f90! by m
    const int u = m == 0 ? p : m == 1 ? q : m == 2 ? L - 1 - p : L - 1 - q;
    const int v = m == 0 ? q : m == 1 ? L - 1 - p : m == 2 ? L - 1 - q : p;
    return (v * L + u) * g.nzp;
  };
  const int ring = (L + 1) * g.nzp;  // column (1, 1): zero, and its neighbours too (pad >= 2)
#pragma unroll
  for (int k = 0; k < 8; ++k) w[k] = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k) off[k] = ring;
  if (V.mode != 2) {
    off[0] = pos(a, b);
    w[0] = 1.f;
    return;
  }
  const OneLine l3 = one_line(b, V.tn, L);
#pragma unroll
  for (int e3 = 0; e3 < 2; ++e3) {
    const int a1 = a + l3.off + e3;
    if (a1 < 0 || a1 >= L) continue;
    const OneLine l2 = one_line(a1, V.sn, L);
#pragma unroll
    for (int e2 = 0; e2 < 2; ++e2) {
      const int b1 = b + l2.off + e2;
      if (b1 < 0 || b1 >= L) continue;
      const OneLine l1 = one_line(b1, V.tn, L);
      const int a0 = a1 + l1.off;
      if (a0 < 0 || a0 > L - 2) continue;
      const double w32 = (e3 ? 1.0 - l3.lo : l3.lo) * (e2 ? 1.0 - l2.lo : l2.lo);
      off[2 * e3 + e2] = pos(a0, b1);
      w[4 * e3 + 2 * e2] = (float)(w32 * l1.lo);
      w[4 * e3 + 2 * e2 + 1] = (float)(w32 * (1.0 - l1.lo));
    }
  }
}

// the transpose of one_geo: hit(x, y, w) for the rotated-grid points that read
// image column (j1, j2) with a weight that is not zero
template <class F>
__device__ __forceinline__ void one_hits(const ZGeom& g, const Rot1View& V, int j1, int j2, F hit) {
  const int L = g.L, p = g.pad + j1, q = g.pad + j2, m = V.mode == 0 ? 0 : V.m, nx = g.nx, pad = g.pad;
  const int A = m == 0 ? p : m == 1 ? L - 1 - q : m == 2 ? L - 1 - p : q;  // rot_f90! by m
  const int B = m == 0 ? q : m == 1 ? p : m == 2 ? L - 1 - q : L - 1 - p;
  if (V.mode != 2) {
    if (A >= pad && A < pad + nx && B >= pad && B < pad + nx) hit(A - pad, B - pad, 1.f);
    return;
  }
  const OneLine l1 = one_line(B, V.tn, L);
#pragma unroll
  for (int e1 = 0; e1 < 2; ++e1) {
    const int a1 = A - l1.off - e1;
    if (a1 < 0 || a1 >= L) continue;
    const OneLine l2 = one_line(a1, V.sn, L);
#pragma unroll
    for (int e2 = 0; e2 < 2; ++e2) {
      const int b = B - l2.off - e2;
      if (b < pad || b >= pad + nx) continue;
      const OneLine l3 = one_line(b, V.tn, L);
#pragma unroll
      for (int e3 = 0; e3 < 2; ++e3) {
        const int a = a1 - l3.off - e3;
        if (a < pad || a >= pad + nx) continue;
        const float w = (float)((e1 ? 1.0 - l1.lo : l1.lo) * (e2 ? 1.0 - l2.lo : l2.lo) * (e3 ? 1.0 - l3.lo : l3.lo));
        if (w != 0.f) hit(a - pad, b - pad, w);
      }
    }
  }
}

// Attenuation cache in the ATT layout: block (column x, view v), one thread
// per z (nzp threads); each walks y and scans the rotated mu-map (bilinear
// sample of the IZ-laid-out mu-map with bilinear()'s fmul/fadd order), as
// k_atten_build does.
template <bool ONE>
__global__ void __launch_bounds__(256) k_zatten(ZGeom g, const float* __restrict__ muz,
                                               const float4* __restrict__ rot, const Rot1View* __restrict__ r1, float dy,
                                               float* __restrict__ att) {
  const int x = blockIdx.x, v = blockIdx.y, z = threadIdx.x;
  if (z >= g.nzp) return;
  const float mdy = -dy;
  float prefix = 0.f;
  const size_t Lz = (size_t)g.L * g.nzp;
  for (int y = 0; y < g.ny; ++y) {
    float m;
    if constexpr (ONE) {
      float w[8];
      int off[4];
      const Rot1View V = r1[v];
      const int d = one_delta(g, V.mode == 0 ? 0 : V.m);
      one_geo(g, V, x, y, w, off);
      m = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float* p = muz + off[k] + z;
        m = fmaf(w[2 * k], p[0], m);
        m = fmaf(w[2 * k + 1], p[d], m);
      }
    } else {
      const float4 r = rot[v];
      float4 w;
      int off;
      zgeo(g, r.x, r.y, r.z != 0.f, x, y, w, off);
      const float* p = muz + off + z;
      m = __fmul_rn(w.x, p[0]);
      m = __fadd_rn(m, __fmul_rn(w.y, p[g.nzp]));
      m = __fadd_rn(m, __fmul_rn(w.z, p[Lz]));
      m = __fadd_rn(m, __fmul_rn(w.w, p[Lz + g.nzp]));
    }
    const float e = __fadd_rn(prefix, __fmul_rn(0.5f, m));
    att[(((size_t)v * g.ny + y) * g.nx + x) * g.nzp + z] = z < g.nz ? expf(__fmul_rn(e, mdy)) : 0.f;
    prefix = __fadd_rn(prefix, m);
  }
}

// ------------------------------------------------------------------------
// k_zrot_fwd: the rotated image planes P[plane][nz][nx] (plane = slot * ny + y)
// of the split kernels from the z-fastest volume: products and sums of the
// slice kernel (bilinear, spect_kernels.cuh), so the planes are the same bits.
// A thread takes four z of a column: its taps are four
// 16-byte loads next to its neighbours', where the slice kernel reads four
// scattered floats of shared memory an output and works out each output's
// weights; here 32 columns' weights serve all z.  The tile turns the columns
// into rows.  Bound: issue slots (70 % taken) and the write of P.  Measured
// for 15 views of 128x128x80 (79 MB): 39 us and 6 us for k_to_iz, the slice
// kernel 78 us (43 us with every thread working out its own weights).
// grid (planes, ceil(nx/32)), 256 threads, shared memory 33 * zround(nz, 4) floats.
__global__ void __launch_bounds__(256) k_zrot_fwd(ZGeom g, const float* iz, const float4* __restrict__ rot,
                                                  const int* __restrict__ vidx, float* __restrict__ P) {
  extern __shared__ float4 smem4[];
  float* const tile = reinterpret_cast<float*>(smem4);  // [z][33]
  __shared__ float4 geoW[32];                           // a column's weights and the offset of its first tap
  __shared__ int geoO[32];
  const int x0 = blockIdx.y * 32, pl = blockIdx.x, slot = pl / g.ny, y = pl - slot * g.ny;
  const int n4 = (g.nz + 3) / 4, nxb = min(32, g.nx - x0), nzp = g.nzp;
  const size_t Lz = (size_t)g.L * nzp;
  const float4 r = rot[vidx[slot]];
  const bool ident = r.z != 0.f;
  if (threadIdx.x < nxb) {
    float4 w;
    int off;
    zgeo(g, r.x, r.y, ident, x0 + threadIdx.x, y, w, off);
    geoW[threadIdx.x] = w;
    geoO[threadIdx.x] = off;
  }
  __syncthreads();
  grid_wait();
  const int dx = 256 / n4, dz = 256 - dx * n4;
  int x = threadIdx.x / n4, z4 = threadIdx.x - x * n4;
  while (x < nxb) {
    const float* p = iz + geoO[x] + 4 * z4;
    float4 v = ld4(p);
    if (!ident) {
      const float4 b = ld4(p + nzp), c = ld4(p + Lz), d = ld4(p + Lz + nzp), w = geoW[x];
      auto mix = [&](float a, float b, float c, float d) {
        return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(w.x, a), __fmul_rn(w.y, b)), __fmul_rn(w.z, c)),
                         __fmul_rn(w.w, d));
      };
      v = make_float4(mix(v.x, b.x, c.x, d.x), mix(v.y, b.y, c.y, d.y), mix(v.z, b.z, c.z, d.z),
                      mix(v.w, b.w, c.w, d.w));
    }
    float* t = tile + 4 * z4 * 33 + x;
    t[0] = v.x;
    t[33] = v.y;
    t[66] = v.z;
    t[99] = v.w;
    x += dx;
    z4 += dz;
    if (z4 >= n4) {
      z4 -= n4;
      ++x;
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  float* o = P + (size_t)pl * g.nz * g.nx + x0 + lane;
  if (lane < nxb)
    for (int z = threadIdx.x >> 5; z < g.nz; z += 8) o[(size_t)z * g.nx] = tile[z * 33 + lane];
}

// ------------------------------------------------------------------------
// Walk over the depth planes of a group: plane q = (slot, j) of the slot-major
// list of n = nv ny is depth y = j ystep mod ny of the slot's view (ystep
// coprime to ny and near 0.618 ny: a short range of j holds narrow and wide
// PSF planes alike), and block b of a grid of G owns planes [b n / G,
// (b + 1) n / G).  The forward sums a block's planes of one slot into one
// partial view, number b + slot (different for every pair that occurs).
// k_reduce_parts adds a slot's partials in block order (+ the EM ratio
// y / (A x + bg), src/ml-os-em.jl:38,119).
__device__ __forceinline__ int zblock_of(long long q, int n, int G) { return (int)(((q + 1) * G - 1) / n); }

// four view elements a thread where nxz % 4 == 0 (V = 4), else one
template <int V>
__global__ void __launch_bounds__(256) k_reduce_parts(const float* part, int nv, int ny, int G, int nxz, float* out,
                                                      const float* y, const float* bg,
                                                      const __grid_constant__ ViewList list) {
  const int* const vidx = list.ptr();
  const int per = nxz / V, n = nv * ny;
  grid_wait();
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nv * per; k += gridDim.x * blockDim.x) {
    const int slot = k / per, e = V * (k - slot * per);
    const int b0 = zblock_of((long long)slot * ny, n, G), b1 = zblock_of((long long)(slot + 1) * ny - 1, n, G);
    const float* p = part + (size_t)(b0 + slot) * nxz + e;
    float s[V];
#pragma unroll
    for (int i = 0; i < V; ++i) s[i] = 0.f;
#pragma unroll 8
    for (int b = b0; b <= b1; ++b, p += nxz) {
      if constexpr (V == 4) {
        const float4 q = ld4(p);
        s[0] += q.x;
        s[1] += q.y;
        s[2] += q.z;
        s[3] += q.w;
      } else {
        s[0] += p[0];
      }
    }
    const size_t src = y ? (size_t)vidx[slot] * nxz + e : 0, dst = (size_t)slot * nxz + e;
#pragma unroll
    for (int i = 0; i < V; ++i) out[dst + i] = y ? y[src + i] / (s[i] + bg[src + i]) : s[i];
  }
}

// ------------------------------------------------------------------------
// k_zfwd<NT>: forward.  Per plane: the rotated, attenuated image columns 2 xp,
// 2 xp + 1 as pair lines ZB (gather), the z pass -> rows 2 zp, 2 zp + 1 as
// pair lines XB, the x pass accumulated in registers over the block's planes
// of the view (NT tasks of X outputs a thread).  Two barriers a plane:
// phase A runs the z pass of plane p and the sample geometry of plane p + 1,
// phase B the x pass of plane p and the gather of plane p + 1; its table is
// copied and its attenuation prefetched into L2 during phase A.  Small planes
// take a few warps a block and several blocks an SM, so that one's barriers
// and gather latency pass behind another's FMAs; tasks of 8 outputs keep a
// thread at 96 registers, x outputs included (16 spilled them).
// Bound: the shared-memory/L1 pipe (63 % busy at 128x128x80, 37 taps) and the
// gather's L2 latency between the barriers; FFMA2 is 37 % of the
// instructions.  Measured there: 15 views 78.3 us, 120 views 573 us; 64x64x40,
// 19 taps, 60 views 38 us; 128x128x1, 80 views 45 us (one line a lane, chunks
// of 15 planes on one block an SM: 107.7, 695, 107, 229 us).
// ONE: the :one rotation (eight taps a column, one_geo).
// Shared memory: [2 tables][geoW nx x (w00 w00 w10 w10 | w01 w01 w11 w11)]
// [geoO nx int][ZB nxp * vst][XB (nz + 1) / 2 * bst] (lines: float2).
template <int NT, bool ONE>
__global__ void __launch_bounds__(kZThreads, 1) k_zfwd(const __grid_constant__ ZArgs a) {
  extern __shared__ float4 smem4[];
  constexpr int X = kZfwdX, W = kZfwdZ;
  const int* const vidx = a.vidx.ptr();
  const ZGeom& g = a.g;
  const int nx = g.nx, ny = g.ny, nz = g.nz, nzp = g.nzp, hs = g.hs, ts = g.ts, nxp = nx / 2, nzp2 = (nz + 1) / 2;
  const int vst = a.t.vst, bst = a.t.bst, R0 = g.R0, C0 = g.C0, hz = g.hz, hx = g.hx;
  const int trow = ztable_floats(g), tid = threadIdx.x, nth = blockDim.x;
  float* const tab0 = reinterpret_cast<float*>(smem4);
  float4* const geoW = reinterpret_cast<float4*>(tab0 + 2 * trow);
  int* const geoO = reinterpret_cast<int*>(geoW + (ONE ? 4 : 2) * nx);
  f2* const ZB = reinterpret_cast<f2*>(geoO + (ONE ? 4 * nx : zround(nx, 4)));
  f2* const XB = ZB + (size_t)nxp * vst;
  const int n = a.nv * ny;
  const int p0 = (int)((long long)blockIdx.x * n / gridDim.x), p1 = (int)((long long)(blockIdx.x + 1) * n / gridDim.x);
  if (p0 >= p1) return;
  const size_t Lz = (size_t)g.L * nzp;
  int slot = p0 / ny, j = p0 - slot * ny;
  int y = (int)((long long)j * a.t.ystep % ny), v = vidx[slot];
  auto table = [&](int view, int yy, int s) {  // every thread: its 16-byte pieces of the plane's table
    if (4 * tid >= trow) return;
    const float* src = a.tab + (((size_t)a.viewset[view] * ny + yy) * 2) * trow;
    for (int k = 4 * tid; k < trow; k += 4 * nth) cp16(tab0 + s * trow + k, src + k);
  };
  auto geometry = [&](int view, int yy) {
    if (tid >= nx) return;
    if constexpr (ONE) {
      const Rot1View V = a.r1[view];
      for (int x = tid; x < nx; x += nth) {
        float w[8];
        int off[4];
        one_geo(g, V, x, yy, w, off);
#pragma unroll
        for (int k = 0; k < 4; ++k) geoW[4 * x + k] = make_float4(w[2 * k], w[2 * k], w[2 * k + 1], w[2 * k + 1]);
        reinterpret_cast<int4*>(geoO)[x] = make_int4(off[0], off[1], off[2], off[3]);
      }
    } else {
      const float4 r = a.rot[view];
      for (int x = tid; x < nx; x += nth) {
        float4 w;
        int off;
        zgeo(g, r.x, r.y, r.z != 0.f, x, yy, w, off);
        geoW[2 * x] = make_float4(w.x, w.x, w.y, w.y);
        geoW[2 * x + 1] = make_float4(w.z, w.z, w.w, w.w);
        geoO[x] = off;
      }
    }
  };
  // rotated, attenuated column x at z group z4: four z as two packed pairs
  const int nz4 = (nz + 3) / 4, dq = nth / nz4, dr = nth - dq * nz4, q0 = tid / nz4, r0 = tid - q0 * nz4;
  auto sample = [&](const float* att, int d, int x, int z4, f2& lo, f2& hi) {
    if constexpr (ONE) {
      const int4 o4 = reinterpret_cast<const int4*>(geoO)[x];
      const int os[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float* p = a.img + os[k] + 4 * z4;
        const ulonglong2 t0 = ldp(p), t1 = ldp(p + d);
        const ulonglong2 w = reinterpret_cast<const ulonglong2*>(geoW)[4 * x + k];
        lo = fma2(w.y, t1.x, k ? fma2(w.x, t0.x, lo) : mul2(w.x, t0.x));
        hi = fma2(w.y, t1.y, k ? fma2(w.x, t0.y, hi) : mul2(w.x, t0.y));
      }
      const ulonglong2 at = ldp_cs(att + x * nzp + 4 * z4);
      lo = mul2(lo, at.x);
      hi = mul2(hi, at.y);
      return;
    } else {
      zsample4(a.img + geoO[x] + 4 * z4, nzp, Lz, geoW + 2 * x, att + x * nzp + 4 * z4, lo, hi);
    }
  };
  const int hi4 = (tid >> 2) & 1;
  auto gather = [&](int view, int yy) {  // unit (column pair, z group)
    const float* att = a.att + (((size_t)view * ny + yy) * nx) * nzp;
    int d = 0;
    if constexpr (ONE) d = one_delta(g, a.r1[view].mode == 0 ? 0 : a.r1[view].m);
    for (int xp = q0, z4 = r0; xp < nxp;) {
      f2 al, ah, bl, bh;
      sample(att, d, 2 * xp, z4, al, ah);
      sample(att, d, 2 * xp + 1, z4, bl, bh);
      // a lane's 32 bytes as two stores, the halves in turn by lane group of
      // four: the eight lanes of an access phase hit distinct bank groups
      float4* o = reinterpret_cast<float4*>(ZB + xp * vst + R0 + 4 * z4);
      o[hi4] = zturn(hi4 ? ah : al, hi4 ? bh : bl);
      o[hi4 ^ 1] = zturn(hi4 ? al : ah, hi4 ? bl : bh);
      xp += dq;
      z4 += dr;
      if (z4 >= nz4) {
        z4 -= nz4;
        ++xp;
      }
    }
  };
  table(v, y, 0);
  geometry(v, y);
  // the lines start zero; only their data elements are written later
  for (int k = tid; k < nxp * vst + nzp2 * bst; k += nth) ZB[k] = 0;
  cp_wait();
  __syncthreads();
  grid_wait();
  gather(v, y);
  // this thread's x tasks: rows 2 zp, 2 zp + 1, columns x0 .. x0 + X - 1
  f2 acc[NT][X];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int k = 0; k < X; ++k) acc[i][k] = 0;
  __syncthreads();
  const int nzb = (nz + W - 1) / W;
  // this thread's first z task and the step to its next; its x tasks
  const int zb0 = tid / nxp, xp0 = tid - zb0 * nxp, dzb = nth / nxp, dxz = nth - dzb * nxp;
  int xs0[NT], rowo[NT];
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    const int xb = (tid + i * nth) / nzp2;
    xs0[i] = X * xb;
    rowo[i] = (tid + i * nth - xb * nzp2) * bst;
  }
  int tb = 0;
  for (int p = p0;; ++p) {
    int slot1 = slot, y1 = y + a.t.ystep;
    if (y1 >= ny) y1 -= ny;
    if (++j == ny) {
      j = y1 = 0;
      ++slot1;
    }
    const bool more = p + 1 < p1;
    const int v1 = more && slot1 != slot ? vidx[slot1] : v;
    const float* const Wt = tab0 + tb * trow;
    const f2* const Wd = reinterpret_cast<const f2*>(Wt);
    const int4 rg = *reinterpret_cast<const int4*>(Wt + 2 * hs + ts);  // tap ranges: z pass, x pass
    if (more) {
      table(v1, y1, tb ^ 1);
      if (tid == 0)
        prefetch_l2_bulk(a.att + (((size_t)v1 * ny + y1) * nx) * nzp, (unsigned)(nx * nzp * sizeof(float)));
    }
    // phase A: z pass of p, task (column pair, W rows) -> XB
    const float* ELz = Wt + 2 * hs;
    const float* ERz = ELz + hz;
    for (int zb = zb0, xp = xp0; zb < nzb;) {
      const int z0 = W * zb;
      const f2* col = ZB + xp * vst;
      f2 o[W];
#pragma unroll
      for (int k = 0; k < W; ++k) o[k] = 0;
      zpass2<W>(Wd, rg.x, rg.y, col + z0, o);
      zclamp<W>(o, ELz, ERz, hz, z0, nz, col[R0], col[R0 + nz - 1]);
      f2* w = XB + (z0 / 2) * bst + C0 + 2 * xp;
#pragma unroll
      for (int m = 0; m < W / 2; ++m)
        if (z0 + 2 * m < nz)
          *reinterpret_cast<float4*>(w + m * bst) = zturn(o[2 * m], o[2 * m + 1]);
      xp += dxz;
      zb += dzb;
      if (xp >= nxp) {
        xp -= nxp;
        ++zb;
      }
    }
    if (more) geometry(v1, y1);
    cp_wait();
    __syncthreads();
    // phase B: x pass of p, accumulated; gather of p + 1
    const float* ELx = ERz + hz;
    const float* ERx = ELx + hx;
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const int x0 = xs0[i];
      if (x0 < nx) {
        const f2* const row = XB + rowo[i];
        // the plane's own sum first, then onto the depth sum: short chains
        f2 o[X];
#pragma unroll
        for (int k = 0; k < X; ++k) o[k] = 0;
        zpass2<X>(Wd + g.zpw, rg.z, rg.w, row + x0, o);
        zclamp<X>(o, ELx, ERx, hx, x0, nx, row[C0], row[C0 + nx - 1]);
#pragma unroll
        for (int k = 0; k < X; ++k) acc[i][k] = add2(acc[i][k], o[k]);
      }
    }
    if (more) gather(v1, y1);
    if (!more || slot1 != slot) {  // p ends the block's planes of this view: its partial view
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        const int x0 = xs0[i], zp = (tid + i * nth) % nzp2;
        if (x0 < nx) zstore_part<X>(a.part + (size_t)(blockIdx.x + slot) * nz * nx, acc[i], nx, nz, 2 * zp, x0);
#pragma unroll
        for (int k = 0; k < X; ++k) acc[i][k] = 0;
      }
    }
    if (!more) break;
    __syncthreads();
    slot = slot1;
    y = y1;
    v = v1;
    tb ^= 1;
  }
}

// ------------------------------------------------------------------------
// k_zadj<W>: adjoint convolution.  A work plane is (slot, row tile of tz rows,
// j); block b walks planes [b n / grid, (b + 1) n / grid) of the slot-major
// list of n, so blocks differ by at most one plane.  Plane j of an item is
// depth y = j ystep mod ny, ystep coprime to ny and near 0.618 ny: a short
// range of j holds narrow and wide PSF planes alike.  Per plane
//   z pass  of the view's rows (columns 2 xp, 2 xp + 1 as one pair line,
//           loaded once per item) -> XB, the plane's rows (2 zp, 2 zp + 1 as
//           one pair line, zero outside the image),
//   x pass  of XB, times the attenuation -> T.
// Each pass is the zero-padded correlation with the factor plus the folded
// padding at the two ends (z folds where the tile holds the image's first or
// last row).  Lanes of the x pass are consecutive row pairs, so the
// attenuation reads and the T stores are 256 contiguous bytes a warp (x then z
// would read and write 16 bytes at a column stride).  The plane's table
// (weights, folds, tap ranges) is copied one plane ahead and its attenuation
// prefetched into L2; an x task loads its attenuation before its FMAs, which
// hides the rest of that latency (8 outputs a task: 16 would need 32 more
// registers).  Two barriers a plane with one XB (the host then runs several
// blocks per SM, which fill each other's waits), one with two.
// Bound: FFMA2 (33.4 M warp instructions at 128x128x80, 37 taps, 15 views; the
// pipe is 43 % busy) and what the blocks wait for at their barriers.  Measured
// there: 66 us; 64x64x64, 11 taps, 64 views 38 us; 256x256x200, 65 taps, 8
// views (five row tiles, two XB) 483 us (x then z, one line a lane: 105, 92,
// 735 us).
// Shared memory (float2): [VB nxp * vst][XB nxb * (tz / 2) * bst][3 tables].
template <int W>
__global__ void __launch_bounds__(kZThreads, 1) k_zadj(const __grid_constant__ ZArgs a) {
  extern __shared__ float4 smem4[];
  const int* const vidx = a.vidx.ptr();
  const ZGeom& g = a.g;
  const int nx = g.nx, ny = g.ny, nz = g.nz, nzp = g.nzp, hs = g.hs, ts = g.ts, nxp = nx / 2;
  const int tz = a.t.tz, vst = a.t.vst, bst = a.t.bst, R0 = g.R0, C0 = g.C0, hz = g.hz, hx = g.hx;
  const int trow = ztable_floats(g), tid = threadIdx.x, nth = blockDim.x;
  f2* const VB = reinterpret_cast<f2*>(smem4);
  f2* const XB0 = VB + (size_t)nxp * vst;
  const size_t xbs = a.t.nxb > 1 ? (size_t)(tz / 2) * bst : 0;  // offset of the second row buffer
  float* const tab0 = reinterpret_cast<float*>(XB0 + (size_t)a.t.nxb * (tz / 2) * bst);
  const int ntile = a.t.ntile, n = a.nv * ntile * ny;
  const int p0 = (int)((long long)blockIdx.x * n / gridDim.x), p1 = (int)((long long)(blockIdx.x + 1) * n / gridDim.x);
  if (p0 >= p1) return;
  const int vlen = W * ((tz + W - 1) / W) + g.zpw;  // elements of a view line that the windows read
  const float rnxp = 1.0f / nxp;
  int st = p0 / ny, j = p0 - st * ny;  // (slot, tile) of the plane and its place in the item
  int y = (int)((long long)j * a.t.ystep % ny);
  int slot = st / ntile, Z0 = (st - slot * ntile) * tz, v = vidx[slot];
  auto table = [&](int view, int yy, int s) {  // every thread: its 16-byte pieces of the plane's table
    const float* src = a.tab + (((size_t)a.viewset[view] * ny + yy) * 2 + 1) * trow;
    for (int k = 4 * tid; k < trow; k += 4 * nth) cp16(tab0 + s * trow + k, src + k);
  };
  // view rows Z0 - R0 .. of the item as pair lines, zero outside the image;
  // lanes on consecutive column pairs, eight elements in flight
  auto load_view = [&]() {
    const float* V = a.views + (size_t)slot * nz * nx;
    const int tot = vlen * nxp;
    for (int k0 = tid; k0 < tot; k0 += 8 * nth) {
      float2 q[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int k = k0 + i * nth, e = zdiv(k, rnxp), xp = k - e * nxp, z = Z0 + e - R0;
        const bool in = k < tot && z >= 0 && z < nz;
        const float* s = V + (size_t)z * nx + 2 * xp;  // 4-byte aligned only: the caller's array
        q[i].x = in ? s[0] : 0.f;
        q[i].y = in ? s[1] : 0.f;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int k = k0 + i * nth, e = zdiv(k, rnxp), xp = k - e * nxp;
        if (k < tot) VB[(size_t)xp * vst + e] = pack2(q[i].x, q[i].y);
      }
    }
  };
  table(v, y, 0);
  for (int k = tid; k < a.t.nxb * (tz / 2) * bst; k += nth) XB0[k] = 0;
  grid_wait();
  load_view();
  cp_wait();
  __syncthreads();
  constexpr int X = kZadjX;  // outputs of an x task
  const int nxw = (nx + X - 1) / X;
  int tb = 0, xb2 = 0;  // table and row buffer of the plane
  for (int p = p0;;) {
    const int rows = min(tz, nz - Z0), nzp2 = (rows + 1) / 2;
    // the next plane, its table on the way
    int st1 = st, y1 = y + a.t.ystep;
    if (y1 >= ny) y1 -= ny;
    if (++j == ny) {
      j = y1 = 0;
      ++st1;
    }
    const bool more = p + 1 < p1;
    const int tb1 = tb == 2 ? 0 : tb + 1;
    const int slot1 = st1 == st ? slot : st1 / ntile;
    if (more) {  // the next plane's attenuation columns on their way into L2, too
      const int v1 = slot1 == slot ? v : vidx[slot1], Z1 = (st1 - slot1 * ntile) * tz, ln = (min(tz, nz - Z1) + 31) / 32;
      table(v1, y1, tb1);
      const float* src = a.att + (((size_t)v1 * ny + y1) * nx) * nzp + Z1;
      if (ntile == 1) {
        if (tid == 0) prefetch_l2_bulk(src, (unsigned)(nx * nzp * sizeof(float)));
      } else {
        for (int x = tid; x < nx; x += nth)
          for (int l = 0; l < ln; ++l) prefetch_l2(src + x * nzp + 32 * l);
      }
    }
    const float* const Wt = tab0 + tb * trow;
    const f2* const Wd = reinterpret_cast<const f2*>(Wt);
    const int4 rg = *reinterpret_cast<const int4*>(Wt + 2 * hs + ts);  // tap ranges: z pass, x pass
    f2* const XB = XB0 + xb2 * xbs;
    {  // z pass: task (column pair, W rows) -> XB
      const float* cLz = Wt + 2 * hs + 2 * hx;
      const float* cRz = cLz + hz;
      const int tasks = nxp * ((rows + W - 1) / W);
      for (int t = tid; t < tasks; t += nth) {
        const int zb = zdiv(t, rnxp), xp = t - zb * nxp, z0 = W * zb;
        const f2* col = VB + (size_t)xp * vst;
        f2 o[W];
#pragma unroll
        for (int k = 0; k < W; ++k) o[k] = 0;
        zpass2<W>(Wd, rg.x, rg.y, col + z0, o);
        if (Z0 + z0 == 0) o[0] = add2(o[0], zfold2(cLz, col + R0, 1, hz));
        const int kz = nz - 1 - Z0 - z0;
        if (kz >= 0 && kz < W) {
          const f2 s = zfold2(cRz, col + R0 + z0 + kz, -1, hz);
#pragma unroll
          for (int k = 0; k < W; ++k)
            if (k == kz) o[k] = add2(o[k], s);
        }
        f2* w = XB + (size_t)(z0 / 2) * bst + C0 + 2 * xp;
#pragma unroll
        for (int m = 0; m < W / 2; ++m)
          if (z0 + 2 * m < rows)
            *reinterpret_cast<float4*>(w + (size_t)m * bst) =
                zturn(o[2 * m], o[2 * m + 1]);
      }
    }
    cp_wait();
    __syncthreads();
    {  // x pass: task (row pair, X columns), times the attenuation -> T
      const float* cLx = Wt + 2 * hs;
      const float* cRx = cLx + hx;
      const float* attp = a.att + (((size_t)v * ny + y) * nx) * nzp + Z0;
      float* Tp = a.T + (((size_t)slot * ny + y) * nx) * nzp + Z0;
      const int tasks = nzp2 * nxw;
      const float rn = 1.0f / nzp2;
      for (int t = tid; t < tasks; t += nth) {
        const int xb = zdiv(t, rn), zp = t - xb * nzp2, x0 = X * xb;
        const bool whole = x0 + X <= nx;
        const int at0 = x0 * nzp + 2 * zp;
        // the attenuation first: its latency passes behind the window's FMAs
        f2 at[X];
        if (whole) {
          const float* q = attp + at0;
#pragma unroll
          for (int k = 0; k < X; ++k, q += nzp) at[k] = *reinterpret_cast<const f2*>(q);
        } else {
#pragma unroll
          for (int k = 0; k < X; ++k) at[k] = *reinterpret_cast<const f2*>(attp + at0 + min(k, nx - 1 - x0) * nzp);
        }
        const f2* row = XB + (size_t)zp * bst;
        f2 o[X];
#pragma unroll
        for (int k = 0; k < X; ++k) o[k] = 0;
        zpass2<X>(Wd + g.zpw, rg.z, rg.w, row + x0, o);
        if (x0 == 0) o[0] = add2(o[0], zfold2(cLx, row + C0, 1, hx));
        const int kx = nx - 1 - x0;
        if (kx < X) {
          const f2 s = zfold2(cRx, row + C0 + nx - 1, -1, hx);
#pragma unroll
          for (int k = 0; k < X; ++k)
            if (k == kx) o[k] = add2(o[k], s);
        }
        float* q = Tp + at0;
        if (whole) {
#pragma unroll
          for (int k = 0; k < X; ++k, q += nzp) *reinterpret_cast<f2*>(q) = mul2(at[k], o[k]);
        } else {
#pragma unroll
          for (int k = 0; k < X; ++k, q += nzp)
            if (x0 + k < nx) *reinterpret_cast<f2*>(q) = mul2(at[k], o[k]);
        }
      }
    }
    if (!more) break;
    ++p;
    y = y1;
    tb = tb1;
    if (a.t.nxb > 1) xb2 ^= 1;
    if (st1 != st) {  // the last reader of VB finished before the barrier above
      st = st1;
      slot = slot1;
      Z0 = (st - slot * ntile) * tz;
      v = vidx[slot];
      load_view();
      __syncthreads();
    } else if (a.t.nxb == 1) {
      __syncthreads();
    }
  }
}

// ------------------------------------------------------------------------
// k_zrot_adj: a block owns a tile of C = tx ty image columns over all z.  Its
// units (column, four z) are dealt to the threads of a group, kZrotU a thread,
// lanes on consecutive z of a column (16-byte loads, whole sectors); S groups
// take every S-th slot and their sums are added in group order.  The
// rotated-grid points (x, y) whose bilinear footprint contains image column
// (j1, j2) -- those with floor(s1) in {j1-1, j1} and floor(s2) in {j2-1, j2}
// -- lie within |cos| + |sin| of the inverse-rotated pixel centre, so the
// candidates are at most 3 x 3 points (four hit as a rule, three to five but
// for a few; a weight of zero is no hit).  One thread tests the nine of a
// (slot, column) pair with the forward's own position arithmetic and lists the
// hits (T column, weight) in shared memory, vb slots of the tile at a time,
// one batch ahead of the sums; lists of fewer than four end in the zero column
// zcol, so that a unit runs four unconditional loads a slot, the others under
// a branch.  A group's sum runs over its slots and hits in order.
// Bound: L1 (its tag stage is 55 % busy where an SM works: a column's 320
// bytes straddle lines) and the latency of the misses.  Measured: 128x128x80,
// 15 views 42 us; 64x64x64, 64 views 31 us; 64x64x40, 60 views 24 us;
// 256x256x200, 8 views 216 us (candidates tested in every 8-lane group: 49, 57,
// 45, 252 us).
// Epilogue (IZ layout): v = acc (+ prev); mode 1: zeros -> +Inf; mode 2:
// v = x * (v / asum); out = v (z < nz only; out may be prev or x).
template <bool ONE>
__global__ void __launch_bounds__(kZrotThreads, 2) k_zrot_adj(ZGeom g, ZRotTile r, const float* T,
                                                             int zcol, const float4* __restrict__ rot,
                                                             const Rot1View* __restrict__ r1,
                                                             const __grid_constant__ ViewList views, int nv, const float* prev,
                                                             float* out, const float* x, const float* asum,
                                                             int mode) {
  constexpr int U = kZrotU, E = kZrotList;
  const int* const vidx = views.ptr();
  extern __shared__ float4 smem4[];
  const int nth = blockDim.x, tid = threadIdx.x, nx = g.nx, ny = g.ny, n4 = g.nzp / 4, C = r.tx * r.ty;
  const float c0 = g.c0;
  // [2][nth][E]: the hits (T column, weight); the first entry's bits above the
  // column hold their count
  int2* const list = reinterpret_cast<int2*>(smem4);
  const int ntx = (nx + r.tx - 1) / r.tx;
  const int X0 = (blockIdx.x % ntx) * r.tx, Y0 = (blockIdx.x / ntx) * r.ty;
  // hits of the batch of slots from s0 on: thread q's pair is slot s0 + q / C, column q % C
  const int ps = tid / C, pc = tid - ps * C, pj1 = X0 + pc % r.tx, pj2 = Y0 + pc / r.tx;
  const float fj1 = (float)pj1, fj2 = (float)pj2, d1 = fj1 - c0, d2 = fj2 - c0;
  auto hits = [&](int s0, int buf) {
    const int s = s0 + ps;
    int2* const L0 = list + (buf * nth + tid) * E;
    int2* L = L0;
    if (ps < r.vb && s < nv && pj1 < nx && pj2 < nx) {
      if constexpr (ONE) {
        one_hits(g, r1[vidx[s]], pj1, pj2, [&](int xx, int yy, float w) {
          *L++ = make_int2((s * ny + yy) * nx + xx, __float_as_int(w));
        });
      } else {
        const float4 rt = rot[vidx[s]];
        const float cs = rt.x, sn = rt.y;
        const float xc = c0 + cs * d1 + sn * d2, yc = c0 - sn * d1 + cs * d2;
        const float rr = fabsf(cs) + fabsf(sn) + 0.01f;
        const int xlo = max(0, (int)ceilf(xc - rr)), nxc = min(nx - 1, (int)floorf(xc + rr)) - xlo;
        const int ylo = max(0, (int)ceilf(yc - rr)), nyc = min(ny - 1, (int)floorf(yc + rr)) - ylo;
        const int base = (s * ny + ylo) * nx + xlo;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const float di = __fsub_rn((float)(xlo + i), c0), ci = __fmul_rn(cs, di), si = __fmul_rn(sn, di);
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const float dj = __fsub_rn((float)(ylo + k), c0);
            const float s1 = __fadd_rn(c0, __fsub_rn(ci, __fmul_rn(sn, dj)));
            const float s2 = __fadd_rn(c0, __fadd_rn(si, __fmul_rn(cs, dj)));
            // floor(s) == j: 1 - (s - j); floor(s) == j - 1: s - (j - 1); not positive elsewhere
            const float a1 = s1 >= fj1 ? __fsub_rn(1.0f, __fsub_rn(s1, fj1)) : __fsub_rn(s1, fj1 - 1.f);
            const float a2 = s2 >= fj2 ? __fsub_rn(1.0f, __fsub_rn(s2, fj2)) : __fsub_rn(s2, fj2 - 1.f);
            if (i <= nxc && k <= nyc && fminf(a1, a2) > 0.f) {
              *L++ = make_int2(base + k * nx + i, __float_as_int(__fmul_rn(a1, a2)));
            }
          }
        }
      }
    }
    const int m = (int)(L - L0);
    for (; L < L0 + 4; ++L) *L = make_int2(zcol, 0);
    L0->x |= m << kZrotColumnBits;
  };
  // this thread's units: group, column of the tile, z group (a unit past the
  // last repeats it and is not stored)
  const int gth = nth / r.S, grp = tid / gth, gt = tid - grp * gth, units = C * n4;
  const unsigned cb = (unsigned)g.nzp * (unsigned)sizeof(float);  // bytes of a T column
  int col[U];
  const char* Tz[U];
  float4 acc[U];
#pragma unroll
  for (int i = 0; i < U; ++i) {
    const int u = min(gt + i * gth, units - 1);
    col[i] = u / n4;
    Tz[i] = reinterpret_cast<const char*>(T) + 16 * (u - col[i] * n4);
    acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  auto load = [&](int i, int c) {
    return *reinterpret_cast<const float4*>(Tz[i] + (unsigned long long)(unsigned)c * cb);
  };
  auto add = [&](float4& v, int wi, const float4& t) {
    const float w = __int_as_float(wi);
    v.x = fmaf(w, t.x, v.x);
    v.y = fmaf(w, t.y, v.y);
    v.z = fmaf(w, t.z, v.z);
    v.w = fmaf(w, t.w, v.w);
  };
  hits(0, 0);
  __syncthreads();
  grid_wait();
  for (int s0 = 0, buf = 0; s0 < nv; s0 += r.vb, buf ^= 1) {
    if (s0 + r.vb < nv) hits(s0 + r.vb, buf ^ 1);
    const int nb = min(r.vb, nv - s0);
    for (int b = grp; b < nb; b += r.S) {
      const int2* const L = list + (buf * nth + b * C) * E;
#pragma unroll
      for (int i0 = 0; i0 < U; i0 += 2) {  // two units: eight loads before the sums
        float4 t[2][4];
        int w[2][4], m[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int2* const q = L + col[i0 + i] * E;
          const int2 e0 = q[0], e1 = q[1], e2 = q[2], e3 = q[3];
          m[i] = (int)((unsigned)e0.x >> kZrotColumnBits);
          t[i][0] = load(i0 + i, e0.x & kZrotColumnMask);
          t[i][1] = load(i0 + i, e1.x);
          t[i][2] = load(i0 + i, e2.x);
          t[i][3] = load(i0 + i, e3.x);
          w[i][0] = e0.y;
          w[i][1] = e1.y;
          w[i][2] = e2.y;
          w[i][3] = e3.y;
        }
        // the slot's own sum first, then onto the view sum: short chains
        float4 v[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int h = 0; h < 4; ++h) add(v[i], w[i][h], t[i][h]);
        }
        for (int h = 4; h < max(m[0], m[1]); ++h)
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (h < m[i]) {
              const int2 e = L[col[i0 + i] * E + h];
              add(v[i], e.y, load(i0 + i, e.x));
            }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          acc[i0 + i].x += v[i].x;
          acc[i0 + i].y += v[i].y;
          acc[i0 + i].z += v[i].z;
          acc[i0 + i].w += v[i].w;
        }
      }
    }
    __syncthreads();
  }
  if (r.S > 1) {  // sums of groups 1 .. S - 1 to group 0, in order
    float4* const part = smem4;
    if (grp > 0)
#pragma unroll
      for (int i = 0; i < U; ++i) part[((grp - 1) * U + i) * gth + gt] = acc[i];
    __syncthreads();
    if (grp > 0) return;
    for (int q = 0; q < r.S - 1; ++q)
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const float4 v = part[(q * U + i) * gth + gt];
        acc[i].x += v.x;
        acc[i].y += v.y;
        acc[i].z += v.z;
        acc[i].w += v.w;
      }
  }
#pragma unroll
  for (int i = 0; i < U; ++i) {
    if (gt + i * gth >= units) continue;
    const int z = 4 * (gt + i * gth - col[i] * n4);
    const int j1 = X0 + col[i] % r.tx, j2 = Y0 + col[i] / r.tx;
    if (j1 >= nx || j2 >= nx) continue;
    const size_t o = ((size_t)(j2 + g.pad) * g.L + j1 + g.pad) * g.nzp + z;
    const float vq[4] = {acc[i].x, acc[i].y, acc[i].z, acc[i].w};
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (z + e < g.nz) {
        float v = vq[e];
        if (prev) v += prev[o + e];
        if (mode == 1 && v == 0.f) v = __int_as_float(0x7f800000);
        if (mode == 2) v = x[o + e] * (v / asum[o + e]);
        out[o + e] = v;
      }
  }
}

}  // namespace spect
