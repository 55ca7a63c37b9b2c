// zpath.cuh -- the fused SPECT projector pair on z-fastest layouts (sm_100a),
// for the common case: :two rotation, cached attenuation, separable (rank-1)
// PSF planes.
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
// k_zfwd   project! (src/project.jl:77-135): work item (slot, depth chunk);
//          per plane y the block gathers the rotated image (imrotate! :two,
//          src/rotatez.jl:331-362) column by column from IZ, multiplies the
//          attenuation plane (bulk-copied one plane ahead) and writes the
//          z-pass buffer directly; then the z pass and the x pass of the
//          replicate-boundary convolution that fft_conv! computes
//          (src/fft_convolve.jl:33-55).  The x-pass outputs stay in
//          registers across the chunk (the depth sum, src/project.jl:127-130).
//          The rotated volume never leaves the SM.
// k_zadj   backproject! (src/backproject.jl:69-124), convolution half: per
//          plane the x pass and z pass of fft_conv_adj! (src/fft_convolve.jl:
//          82-130) of the view, times the attenuation, stored as T.
// The kernels for planes too large for these kernels' shared memory are in
// zstrip.cuh (same layouts and passes, over plane tiles).
// k_zrot_adj  imrotate_adj! :two (src/rotatez.jl:390-416) and the view sum
//          (src/backproject.jl:146-153): output-stationary gather.  Groups of
//          8 lanes own one image column (x, y) over all z (8 lanes x ZPL) and
//          sum, over their views in order, the bilinear weights of the
//          rotated-grid points whose footprint covers it: the exact transpose
//          of the forward sampling, without atomics.  The EM update
//          (src/ml-os-em.jl:111-126) is its epilogue.
//
// Convolution passes.  fft_conv! equals the replicate-boundary convolution
// out[i] = sum_{m<p} w[m] in[clamp(i - h + m)] with the reversed factor w
// (the plan factors each PSF plane as a[d] b[e]).  Here the input line sits
// zero-padded in shared memory, data starting at an offset D0 = h rounded up
// to 4, and the weights are shifted right by D0 - h, so a task of W = 8 or 16
// consecutive outputs reads a window of 16-byte-aligned float4s; the clamped
// boundary is added as tail terms: the edge value times EL[i] =
// sum_{m < h - i} w[m] (i < h) or ER[n-1-i] = sum_{m > h + n-1-i} w[m]
// (i > n-1-h).  The adjoint passes are the zero-padded correlations with the
// factors themselves plus the folded padding at the two ends (cL_k, cR_k:
// sums of the factor beyond k), as the reference's padding adjoint does.
// The plan zeroes the outer taps of each factor whose summed magnitude per
// side is within 2^-27 of the factor's (below Float32 resolution; a narrow
// Gaussian plane keeps a few of its p taps) and every table, tails and folds
// included, comes from those factors; per plane and pass a range table gives
// the 8-tap blocks that hold the kept taps, and only those are run.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "bulk_copy.cuh"
#include "zpath_api.h"

#ifndef ZFWD_GU
#define ZFWD_GU 2
#endif

namespace spect {

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
// 8-byte read-only global load issued only where pred holds; (0, 0) elsewhere
// (no memory access for those lanes).  p must be 8-byte aligned.
__device__ __forceinline__ float2 ldg2_if(const float* p, bool pred) {
  unsigned a, b;
  asm("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %3, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\t"
      "@q ld.global.nc.v2.b32 {%0, %1}, [%2];\n\t}"
      : "=r"(a), "=r"(b)
      : "l"(p), "r"((int)pred));
  return make_float2(__uint_as_float(a), __uint_as_float(b));
}

// one W-output task (W = 8 or 16) over a zero-padded line, the taps
// m in [4 b4, 4 b4 + 8 nblk) in blocks of 8 (nblk <= 9): o[k] += sum_m w[m]
// line[k + m] (line and w 16-byte aligned; reads line[4 b4, 4 b4 + 8 nblk +
// W)).  Fully unrolled with a uniform early exit; the window elements are
// named by constant indices (registers, no moves): per block two new quads
// of the line and two weight quads feed 8 W FMAs.  Every output sums its
// taps in ascending m, so W does not change the result.
template <int W>
__device__ __forceinline__ void zpassw(const float* __restrict__ w, int b4, int nblk, const float* line,
                                       float (&o)[W]) {
  w += 4 * b4;
  line += 4 * b4;
  float e[W + 8 * 9];
#pragma unroll
  for (int i = 0; i < W / 4; ++i) {
    const float4 q = ld4(line + 4 * i);
    e[4 * i] = q.x;
    e[4 * i + 1] = q.y;
    e[4 * i + 2] = q.z;
    e[4 * i + 3] = q.w;
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    if (k >= nblk) break;
    const float4 q0 = ld4(line + 8 * k + W), q1 = ld4(line + 8 * k + W + 4);
    e[8 * k + W] = q0.x;
    e[8 * k + W + 1] = q0.y;
    e[8 * k + W + 2] = q0.z;
    e[8 * k + W + 3] = q0.w;
    e[8 * k + W + 4] = q1.x;
    e[8 * k + W + 5] = q1.y;
    e[8 * k + W + 6] = q1.z;
    e[8 * k + W + 7] = q1.w;
    const float4 w0 = ld4(w + 8 * k), w1 = ld4(w + 8 * k + 4);
    const float ws[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
    for (int s2 = 0; s2 < 8; ++s2)
#pragma unroll
      for (int j = 0; j < W; ++j) o[j] = fmaf(ws[s2], e[8 * k + s2 + j], o[j]);
  }
}

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
template <int W>
__device__ __forceinline__ void zpass2(const float2* __restrict__ w, int b4, int n4, const float2* line,
                                       float2 (&o)[W]) {
  const float4* w4 = reinterpret_cast<const float4*>(w + 4 * b4);
  const float4* l4 = reinterpret_cast<const float4*>(line + 4 * b4);
  float2 e[W + 4 * 18];
#pragma unroll
  for (int i = 0; i < W / 2; ++i) {
    const float4 q = l4[i];
    e[2 * i] = make_float2(q.x, q.y);
    e[2 * i + 1] = make_float2(q.z, q.w);
  }
#pragma unroll
  for (int k = 0; k < 18; ++k) {
    if (k >= n4) break;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float4 q = l4[2 * k + W / 2 + i];
      e[4 * k + W + 2 * i] = make_float2(q.x, q.y);
      e[4 * k + W + 2 * i + 1] = make_float2(q.z, q.w);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float4 q = w4[2 * k + h];
#pragma unroll
      for (int j = 0; j < W; ++j) o[j] = __ffma2_rn(make_float2(q.x, q.y), e[4 * k + 2 * h + j], o[j]);
#pragma unroll
      for (int j = 0; j < W; ++j) o[j] = __ffma2_rn(make_float2(q.z, q.w), e[4 * k + 2 * h + 1 + j], o[j]);
    }
  }
}

// sum_{k < n} c[k] v[step k] of a pair of lines: four partial sums over k mod
// 4, added as (s0 + s1) + (s2 + s3), so a round waits for one load latency
__device__ __forceinline__ float2 zfold2(const float* c, const float2* v, int step, int n) {
  float2 s[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) s[j] = make_float2(0.f, 0.f);
  int k = 0;
  for (; k + 4 <= n; k += 4)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] = __ffma2_rn(make_float2(c[k + j], c[k + j]), v[step * (k + j)], s[j]);
#pragma unroll
  for (int j = 0; j < 3; ++j)
    if (k + j < n) s[j] = __ffma2_rn(make_float2(c[k + j], c[k + j]), v[step * (k + j)], s[j]);
  return __fadd2_rn(__fadd2_rn(s[0], s[1]), __fadd2_rn(s[2], s[3]));
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
__global__ void __launch_bounds__(256) k_to_iz(ZGeom g, const float* __restrict__ img, float* __restrict__ iz) {
  __shared__ float tile[32][33];
  const int x0 = blockIdx.x * 32, y = blockIdx.y, z0 = blockIdx.z * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
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
__global__ void __launch_bounds__(256) k_from_iz(ZGeom g, const float* __restrict__ iz, float* dst,
                                                 const float* __restrict__ asum, int mode) {
  __shared__ float tile[32][33];
  const int x0 = blockIdx.x * 32, y = blockIdx.y, z0 = blockIdx.z * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
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

// k_t_to_z: adjoint planes of the split kernels ([plane][nz][nx], plane =
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

// Attenuation cache in the ATT layout: block (column x, view v), one thread
// per z (nzp threads); each walks y and scans the rotated mu-map (bilinear
// sample of the IZ-laid-out mu-map with bilinear()'s fmul/fadd order), as
// k_atten_build does.
__global__ void __launch_bounds__(256) k_zatten(ZGeom g, const float* __restrict__ muz,
                                               const float4* __restrict__ rot, float dy, float* __restrict__ att) {
  const int x = blockIdx.x, v = blockIdx.y, z = threadIdx.x;
  if (z >= g.nzp) return;
  const float4 r = rot[v];
  const bool ident = r.z != 0.f;
  const float mdy = -dy;
  float prefix = 0.f;
  const size_t Lz = (size_t)g.L * g.nzp;
  for (int y = 0; y < g.ny; ++y) {
    float4 w;
    int off;
    zgeo(g, r.x, r.y, ident, x, y, w, off);
    const float* p = muz + off + z;
    float m = __fmul_rn(w.x, p[0]);
    m = __fadd_rn(m, __fmul_rn(w.y, p[g.nzp]));
    m = __fadd_rn(m, __fmul_rn(w.z, p[Lz]));
    m = __fadd_rn(m, __fmul_rn(w.w, p[Lz + g.nzp]));
    const float e = __fadd_rn(prefix, __fmul_rn(0.5f, m));
    att[(((size_t)v * g.ny + y) * g.nx + x) * g.nzp + z] = z < g.nz ? expf(__fmul_rn(e, mdy)) : 0.f;
    prefix = __fadd_rn(prefix, m);
  }
}

// ------------------------------------------------------------------------
// k_zfwd<NT, NTH, W>: persistent forward, one block per SM, NTH threads; NT
// x-pass tasks of W outputs per thread, all of a plane's x tasks resident
// (NT * NTH >= nz * nx / W) since their outputs accumulate over the chunk.
// The block walks its planes in sequence; the attenuation plane and weights
// of the next nsf planes are bulk-copied while plane p is worked on (stage
// q % nsf holds plane q).  Two block barriers per plane: phase A runs the z
// pass of plane p (ZB -> XB) and the sample geometry of plane p + 1; phase B
// the x pass of plane p (XB -> registers) and the gather of plane p + 1
// (rotated, attenuated image -> ZB).
template <int NT, int NTH, int W>
__global__ void __launch_bounds__(NTH, 1) k_zfwd(ZArgs a) {
  constexpr int GU = ZFWD_GU;  // gather units per thread and round (4 measured ~1 % faster, with spills in some shapes)
  extern __shared__ float4 smem4[];
  const ZGeom& g = a.g;
  const int nx = g.nx, ny = g.ny, nz = g.nz, nzp = g.nzp, hs = g.hs, ts = g.ts, nsf = g.nsf;
  float* const base = reinterpret_cast<float*>(smem4);
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(base);  // nsf barriers
  const int hts = hs + ts + 4;         // weights, tails, tap ranges of one plane (4 ints)
  const int sts = nx * nzp + hts;      // stage: attenuation plane [x][nzp], then those
  float* const stage = base + 4;
  float* const Hw0 = stage + nsf * sts;           // working weights, tails, ranges: two planes
  float4* const geoW = reinterpret_cast<float4*>(Hw0 + 2 * hts);
  int* const geoO = reinterpret_cast<int*>(geoW + nx);
  float* const ZB = reinterpret_cast<float*>(geoO + zround(nx, 4));  // [x][ast], data rows R0..R0+nz-1
  float* const XB = ZB + (size_t)nx * g.ast;                          // [z][bs], data columns C0..C0+nx-1
  const int tid = threadIdx.x;
  const int nitems = a.nv * a.nchunks;
  const float rnc = 1.0f / a.nchunks;
  auto slot_of = [&](int item) { return zdiv(item, rnc); };             // item / nchunks (items < 2^20)
  auto chunk_of = [&](int item) { return item - zdiv(item, rnc) * a.nchunks; };
  const unsigned abytes = (unsigned)((size_t)nx * nzp * sizeof(float));
  auto issue = [&](int item, int y, int s) {  // one thread: attenuation plane, weights, tails of plane y
    const int sl = slot_of(item), v = a.vidx[sl], set = a.viewset[v];
    float* sA = stage + s * sts;
    float* sW = sA + nx * nzp;
    fence_proxy_async();
    mbar_expect(&bar[s], abytes + (unsigned)(hts * sizeof(float)));
    bulk_copy(&bar[s], sA, a.att + ((size_t)v * ny + y) * nx * nzp, abytes);
    bulk_copy(&bar[s], sW, a.H + ((size_t)set * ny + y) * hs, (unsigned)(hs * sizeof(float)));
    bulk_copy(&bar[s], sW + hs, a.E + ((size_t)set * ny + y) * ts, (unsigned)(ts * sizeof(float)));
    bulk_copy(&bar[s], sW + hs + ts, a.R + ((size_t)set * ny + y) * 4, 4u * sizeof(int));
  };
  auto next = [&](int& item, int& y) {
    const int yend = min(ny, chunk_of(item) * a.chunkY + a.chunkY);
    if (y + 1 < yend) {
      ++y;
    } else {
      item += gridDim.x;
      y = chunk_of(item) * a.chunkY;
    }
  };
  // the padded buffers start zero; only their data rows / columns are written later
  for (size_t k = tid; k < (size_t)nx * g.ast + (size_t)nz * g.bs; k += NTH) ZB[k] = 0.f;
  int i0 = blockIdx.x, y0 = (blockIdx.x % a.nchunks) * a.chunkY;  // plane p
  int i1 = i0, y1 = y0;
  next(i1, y1);  // p + 1
  int iq = i1, yq = y1;  // the next plane to issue
  unsigned pend = 0u;    // stages with a copy issued and not yet waited for (same in every thread)
  if (tid == 0) {
    for (int s = 0; s < nsf; ++s) mbar_init(&bar[s]);
    if (i0 < nitems) issue(i0, y0, 0);
  }
  pend = 1u;
  if (nsf > 1) {
    if (tid == 0 && iq < nitems) issue(iq, yq, 1);
    if (iq < nitems) pend |= 2u;
    next(iq, yq);
  }
  __syncthreads();
  if (!(i0 < nitems)) return;
  const int nzb = (nz + W - 1) / W, ztasks = nx * nzb, nz4 = (nz + 3) / 4, units = nx * nz4;
  const int xtasks = nz * (nx / W);
  const size_t Lz = (size_t)g.L * nzp;
  const int ast = g.ast, bs = g.bs, R0 = g.R0, C0 = g.C0, hz = g.hz, hx = g.hx;
  const int zpw = g.zpw;
  const float rnx = 1.0f / nx, rnz = 1.0f / nz, rnz4 = 1.0f / nz4;
  unsigned phases = 0u;  // parity of each barrier's next wait
  // wait for stage s; false (every thread) when a wait gave up, after the
  // copies in flight have landed
  auto staged = [&](int s) {
    const bool ok = mbar_wait(&bar[s], (phases >> s) & 1u);
    if (ok) {
      phases ^= 1u << s;
      pend &= ~(1u << s);
    }
    if (__syncthreads_or(!ok)) {
      if (tid == 0) {
        atomicExch(a.err, 1);
        for (int k = 0; k < nsf; ++k)
          if ((pend >> k) & 1u) mbar_wait(&bar[k], (phases >> k) & 1u);
      }
      return false;
    }
    return true;
  };
  // sample geometry of plane (item, y), one rotated-grid column per thread:
  // the position arithmetic of RotPos::pos with the view's (cos, sin)
  auto geometry = [&](int item, int y) {
    if (tid < nx) {
      const float4 r = a.rot[a.vidx[slot_of(item)]];
      int j1 = tid, j2 = y;
      float4 w = make_float4(1.f, 0.f, 0.f, 0.f);
      if (r.z == 0.f) {
        const float cs = r.x, sn = r.y;
        const float d1 = __fsub_rn((float)tid, g.c0), d2 = __fsub_rn((float)y, g.c0);
        const float s1 = __fadd_rn(g.c0, __fsub_rn(__fmul_rn(cs, d1), __fmul_rn(sn, d2)));
        const float s2 = __fadd_rn(g.c0, __fadd_rn(__fmul_rn(sn, d1), __fmul_rn(cs, d2)));
        const float f1 = floorf(s1), f2 = floorf(s2);
        const float t1 = __fsub_rn(s1, f1), t2 = __fsub_rn(s2, f2);
        const float u1 = __fsub_rn(1.0f, t1), u2 = __fsub_rn(1.0f, t2);
        j1 = (int)f1;
        j2 = (int)f2;
        w = make_float4(__fmul_rn(u1, u2), __fmul_rn(t1, u2), __fmul_rn(u1, t2), __fmul_rn(t1, t2));
        if (j1 < -g.pad || j1 > nx + g.pad - 2 || j2 < -g.pad || j2 > nx + g.pad - 2) {
          j1 = j2 = 0;
          w = make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
      geoW[tid] = w;
      geoO[tid] = ((j2 + g.pad) * g.L + j1 + g.pad) * nzp;
    }
  };
  // staged weights of stage s into working buffer hb; rotated, attenuated
  // plane into ZB (column x, rows R0 + z), four z at a time
  auto gather = [&](int s, int hb) {
    const float* const sA = stage + s * sts;
    const float* const sW = sA + nx * nzp;
    float* const Hw = Hw0 + hb * hts;
    for (int k = tid; k < hs + ts; k += NTH) Hw[k] = sW[k];
    if (tid < 4) reinterpret_cast<int*>(Hw + hs + ts)[tid] = reinterpret_cast<const int*>(sW + hs + ts)[tid];
    // GU units per round, all their image loads issued before any is used
    for (int u0 = tid; u0 < units; u0 += GU * NTH) {
      float4 t[GU][4];
      int xs[GU], zs[GU];
#pragma unroll
      for (int j = 0; j < GU; ++j) {
        const int u = min(u0 + j * NTH, units - 1);  // a repeated last unit stores the same values
        xs[j] = zdiv(u, rnz4);
        zs[j] = u - xs[j] * nz4;
        const float* p = a.img + geoO[xs[j]] + 4 * zs[j];
        t[j][0] = ld4(p);
        t[j][1] = ld4(p + nzp);
        t[j][2] = ld4(p + Lz);
        t[j][3] = ld4(p + Lz + nzp);
      }
#pragma unroll
      for (int j = 0; j < GU; ++j) {
        const float4 w = geoW[xs[j]];
        const float4 at = ld4(sA + xs[j] * nzp + 4 * zs[j]);
        const float4 t0 = t[j][0], t1 = t[j][1], t2 = t[j][2], t3 = t[j][3];
        float4 o;
        o.x = __fmul_rn(fmaf(w.w, t3.x, fmaf(w.z, t2.x, fmaf(w.y, t1.x, __fmul_rn(w.x, t0.x)))), at.x);
        o.y = __fmul_rn(fmaf(w.w, t3.y, fmaf(w.z, t2.y, fmaf(w.y, t1.y, __fmul_rn(w.x, t0.y)))), at.y);
        o.z = __fmul_rn(fmaf(w.w, t3.z, fmaf(w.z, t2.z, fmaf(w.y, t1.z, __fmul_rn(w.x, t0.z)))), at.z);
        o.w = __fmul_rn(fmaf(w.w, t3.w, fmaf(w.z, t2.w, fmaf(w.y, t1.w, __fmul_rn(w.x, t0.w)))), at.w);
        st4(ZB + xs[j] * ast + R0 + 4 * zs[j], o);
      }
    }
  };
  float acc[NT][W];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int k = 0; k < W; ++k) acc[i][k] = 0.f;
  // the stage that plane p's copy used is free again: the plane nsf ahead
  auto refill = [&](int s) {
    if (iq < nitems) {
      if (tid == 0) issue(iq, yq, s);
      pend |= 1u << s;
    }
    next(iq, yq);
  };
  // prologue: plane p's geometry and staged data, its gather
  geometry(i0, y0);
  if (!staged(0)) return;
  gather(0, 0);
  __syncthreads();
  refill(0);
  int hb = 0, s1 = nsf > 1 ? 1 : 0;  // working-weight buffer of plane p, stage of plane p + 1
  for (;;) {
    const bool h1 = i1 < nitems;
    const float* Hw = Hw0 + hb * hts;
    const int4 rg = *reinterpret_cast<const int4*>(Hw + hs + ts);  // tap ranges: z pass, x pass
    // phase A: z pass of p, task (x, z block) -> XB rows z, column C0 + x
    const float* ELz = Hw + hs;
    const float* ERz = ELz + hz;
    for (int t = tid; t < ztasks; t += NTH) {
      const int zb = zdiv(t, rnx), x = t - zb * nx, z0 = W * zb;
      float o[W];
#pragma unroll
      for (int k = 0; k < W; ++k) o[k] = 0.f;
      const float* col = ZB + x * ast;
      zpassw<W>(Hw, rg.x, rg.y, col + z0, o);
      if (z0 < hz) {  // clamped rows above the plane
        const float e0 = col[R0];
#pragma unroll
        for (int k = 0; k < W; ++k)
          if (z0 + k < hz) o[k] = fmaf(ELz[z0 + k], e0, o[k]);
      }
      if (z0 + W > nz - hz) {  // clamped rows below
        const float e1 = col[R0 + nz - 1];
#pragma unroll
        for (int k = 0; k < W; ++k) {
          const int kk = nz - 1 - z0 - k;
          if (kk >= 0 && kk < hz) o[k] = fmaf(ERz[kk], e1, o[k]);
        }
      }
      float* xo = XB + z0 * bs + C0 + x;
#pragma unroll
      for (int k = 0; k < W; ++k)
        if (z0 + k < nz) xo[k * bs] = o[k];
    }
    if (h1) {
      geometry(i1, y1);
      if (!staged(s1)) return;
    } else {
      __syncthreads();
    }
    // phase B: x pass of p, accumulated over the chunk; gather of p + 1
    const float* ELx = ERz + hz;
    const float* ERx = ELx + hx;
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const int t = tid + i * NTH;
      if (t < xtasks) {
        const int xb = zdiv(t, rnz), z = t - xb * nz, x0 = W * xb;
        const float* row = XB + z * bs;
        zpassw<W>(Hw + zpw, rg.z, rg.w, row + x0, acc[i]);
        if (x0 < hx) {
          const float e0 = row[C0];
#pragma unroll
          for (int k = 0; k < W; ++k)
            if (x0 + k < hx) acc[i][k] = fmaf(ELx[x0 + k], e0, acc[i][k]);
        }
        if (x0 + W > nx - hx) {
          const float e1 = row[C0 + nx - 1];
#pragma unroll
          for (int k = 0; k < W; ++k) {
            const int kk = nx - 1 - x0 - k;
            if (kk < hx) acc[i][k] = fmaf(ERx[kk], e1, acc[i][k]);
          }
        }
      }
    }
    if (h1) gather(s1, hb ^ 1);
    if (!h1 || i1 != i0) {  // p ends its item: partial view of the chunk, part[slot][ch][z][x]
      const int slot = slot_of(i0), ch = i0 - slot * a.nchunks;
      float* out = a.part + ((size_t)slot * a.nchunks + ch) * nz * nx;
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        const int t = tid + i * NTH;
        if (t < xtasks) {
          const int xb = zdiv(t, rnz), z = t - xb * nz;
          float* o = out + (size_t)z * nx + W * xb;
#pragma unroll
          for (int k = 0; k < W; k += 4) st4(o + k, make_float4(acc[i][k], acc[i][k + 1], acc[i][k + 2], acc[i][k + 3]));
        }
#pragma unroll
        for (int k = 0; k < W; ++k) acc[i][k] = 0.f;
      }
    }
    if (!h1) break;
    __syncthreads();
    refill(s1);
    i0 = i1;
    y0 = y1;
    next(i1, y1);
    hb ^= 1;
    s1 = nsf > 1 ? s1 ^ 1 : 0;
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
// attenuation reads and the T stores are 256 contiguous bytes a warp (the
// former x-then-z order read and wrote 16 bytes at a column stride, one line
// a lane: the shared-memory/L1 pipe was its bound).  The plane's table
// (weights, folds, tap ranges) is copied one plane ahead and its attenuation
// prefetched into L2; an x task loads its attenuation before its FMAs, which
// hides the rest of that latency (8 outputs a task: 16 would need 32 more
// registers).  Two barriers a plane with one XB (the host then runs several
// blocks per SM, which fill each other's waits), one with two.
// Bound: FFMA2 (13.1 M of 34.7 M warp instructions at 128x128x80, 37 taps, 15
// views; the pipe is 44 % busy) and what the blocks wait for at their
// barriers.  Measured there: 105 -> 66 us (51.9 M instructions before);
// 64x64x64, 11 taps, 64 views 92 -> 38 us; 256x256x200, 65 taps, 8 views
// (five row tiles, two XB) 735 -> 483 us.
// Shared memory (float2): [VB nxp * vst][XB nxb * (tz / 2) * bst][3 tables].
template <int W>
__global__ void __launch_bounds__(kZThreads, 1) k_zadj(ZArgs a) {
  extern __shared__ float4 smem4[];
  const ZGeom& g = a.g;
  const int nx = g.nx, ny = g.ny, nz = g.nz, nzp = g.nzp, hs = g.hs, ts = g.ts, nxp = nx / 2;
  const int tz = a.t.tz, vst = a.t.vst, bst = a.t.bst, R0 = g.R0, C0 = g.C0, hz = g.hz, hx = g.hx;
  const int trow = ztable_floats(g), tid = threadIdx.x, nth = blockDim.x;
  float2* const VB = reinterpret_cast<float2*>(smem4);
  float2* const XB0 = VB + (size_t)nxp * vst;
  const size_t xbs = a.t.nxb > 1 ? (size_t)(tz / 2) * bst : 0;  // offset of the second row buffer
  float* const tab0 = reinterpret_cast<float*>(XB0 + (size_t)a.t.nxb * (tz / 2) * bst);
  const int ntile = a.t.ntile, n = a.nv * ntile * ny;
  const int p0 = (int)((long long)blockIdx.x * n / gridDim.x), p1 = (int)((long long)(blockIdx.x + 1) * n / gridDim.x);
  if (p0 >= p1) return;
  const int vlen = W * ((tz + W - 1) / W) + g.zpw;  // elements of a view line that the windows read
  const float rnxp = 1.0f / nxp;
  int st = p0 / ny, j = p0 - st * ny;  // (slot, tile) of the plane and its place in the item
  int y = (int)((long long)j * a.t.ystep % ny);
  int slot = st / ntile, Z0 = (st - slot * ntile) * tz, v = a.vidx[slot];
  auto table = [&](int view, int yy, int s) {  // every thread: its 16-byte pieces of the plane's table
    const float* src = a.tab + ((size_t)a.viewset[view] * ny + yy) * trow;
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
        if (k < tot) VB[(size_t)xp * vst + e] = q[i];
      }
    }
  };
  table(v, y, 0);
  for (int k = tid; k < a.t.nxb * (tz / 2) * bst; k += nth) XB0[k] = make_float2(0.f, 0.f);
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
      const int v1 = slot1 == slot ? v : a.vidx[slot1], Z1 = (st1 - slot1 * ntile) * tz, ln = (min(tz, nz - Z1) + 31) / 32;
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
    const float2* const Wd = reinterpret_cast<const float2*>(Wt);
    const int4 rg = *reinterpret_cast<const int4*>(Wt + 2 * hs + ts);  // tap ranges: z pass, x pass
    float2* const XB = XB0 + xb2 * xbs;
    {  // z pass: task (column pair, W rows) -> XB
      const float* cLz = Wt + 2 * hs + 2 * hx;
      const float* cRz = cLz + hz;
      const int tasks = nxp * ((rows + W - 1) / W);
      for (int t = tid; t < tasks; t += nth) {
        const int zb = zdiv(t, rnxp), xp = t - zb * nxp, z0 = W * zb;
        const float2* col = VB + (size_t)xp * vst;
        float2 o[W];
#pragma unroll
        for (int k = 0; k < W; ++k) o[k] = make_float2(0.f, 0.f);
        zpass2<W>(Wd, rg.x, rg.y, col + z0, o);
        if (Z0 + z0 == 0) o[0] = __fadd2_rn(o[0], zfold2(cLz, col + R0, 1, hz));
        const int kz = nz - 1 - Z0 - z0;
        if (kz >= 0 && kz < W) {
          const float2 s = zfold2(cRz, col + R0 + z0 + kz, -1, hz);
#pragma unroll
          for (int k = 0; k < W; ++k)
            if (k == kz) o[k] = __fadd2_rn(o[k], s);
        }
        float2* w = XB + (size_t)(z0 / 2) * bst + C0 + 2 * xp;
#pragma unroll
        for (int m = 0; m < W / 2; ++m)
          if (z0 + 2 * m < rows)
            *reinterpret_cast<float4*>(w + (size_t)m * bst) =
                make_float4(o[2 * m].x, o[2 * m + 1].x, o[2 * m].y, o[2 * m + 1].y);
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
        float2 at[X];
        if (whole) {
          const float* q = attp + at0;
#pragma unroll
          for (int k = 0; k < X; ++k, q += nzp) at[k] = *reinterpret_cast<const float2*>(q);
        } else {
#pragma unroll
          for (int k = 0; k < X; ++k) at[k] = *reinterpret_cast<const float2*>(attp + at0 + min(k, nx - 1 - x0) * nzp);
        }
        const float2* row = XB + (size_t)zp * bst;
        float2 o[X];
#pragma unroll
        for (int k = 0; k < X; ++k) o[k] = make_float2(0.f, 0.f);
        zpass2<X>(Wd + g.zpw, rg.z, rg.w, row + x0, o);
        if (x0 == 0) o[0] = __fadd2_rn(o[0], zfold2(cLx, row + C0, 1, hx));
        const int kx = nx - 1 - x0;
        if (kx < X) {
          const float2 s = zfold2(cRx, row + C0 + nx - 1, -1, hx);
#pragma unroll
          for (int k = 0; k < X; ++k)
            if (k == kx) o[k] = __fadd2_rn(o[k], s);
        }
        float* q = Tp + at0;
        if (whole) {
#pragma unroll
          for (int k = 0; k < X; ++k, q += nzp) *reinterpret_cast<float2*>(q) = __fmul2_rn(at[k], o[k]);
        } else {
#pragma unroll
          for (int k = 0; k < X; ++k, q += nzp)
            if (x0 + k < nx) *reinterpret_cast<float2*>(q) = __fmul2_rn(at[k], o[k]);
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
      v = a.vidx[slot];
      load_view();
      __syncthreads();
    } else if (a.t.nxb == 1) {
      __syncthreads();
    }
  }
}

// ------------------------------------------------------------------------
// k_zrot_adj<ZPL, RB>: two 8-lane groups of a warp own image column p = (j1, j2)
// (grid-stride), lane l of a group the z pairs 2 l + 16 q, q < ZPL / 2 (nzp =
// 8 ZPL): 64 contiguous bytes per group and 8-byte load.  The first group
// sums the even slots, the second the odd ones; a shuffle adds the two
// partial sums (a fixed order).  Per slot, lane l of a group evaluates
// candidate l (and every lane candidate 8) and the group shares the nine by
// shuffles, summing them in the order 0..8.  For
// every slot, the rotated-grid points (x, y) whose bilinear footprint contains
// (j1, j2) -- those with floor(s1) in {j1-1, j1} and floor(s2) in {j2-1, j2}
// -- lie within |cos| + |sin| of the inverse-rotated pixel centre, so the
// candidates are at most 3 x 3 points; each is tested with the forward's own
// position arithmetic and weighted with the forward's weight product.
// RB = 0: a hit candidate's loads are issued under a branch on its offset,
// so the candidates' load latencies follow one another.  RB > 0: the
// candidates go in rounds of RB whose loads are all issued (predicated off
// for misses, which then read zero) before the round's FMAs, so up to
// RB x ZPL / 2 loads per lane are in flight; a miss adds fmaf(0, 0, acc) ==
// acc, so both forms give the same bits.
// Epilogue (IZ layout): v = acc (+ prev); mode 1: zeros -> +Inf; mode 2:
// v = x * (v / asum); out = v (z < nz only; out may be prev or x).
template <int ZPL, int RB>
__global__ void __launch_bounds__(256, (ZPL <= 14 ? 4 : 2)) k_zrot_adj(ZGeom g, const float* __restrict__ T,
                                                 const float4* __restrict__ rot, const int* __restrict__ vidx, int nv,
                                                 const float* prev, float* out, const float* x,
                                                 const float* __restrict__ asum, int mode) {
  const int lane = threadIdx.x & 7, half = (threadIdx.x >> 3) & 1;
  const int npix = (gridDim.x * blockDim.x) >> 4;
  const int nx = g.nx, ny = g.ny, nzp = g.nzp;
  const float c0 = g.c0;
  // every warp runs the same number of iterations (the shuffle needs all lanes)
  for (int p0 = (blockIdx.x * blockDim.x + (threadIdx.x & ~31)) >> 4; p0 < nx * nx; p0 += npix) {
    const int p = min(p0 + ((threadIdx.x >> 4) & 1), nx * nx - 1);
    const bool own = p0 + ((threadIdx.x >> 4) & 1) < nx * nx;
    const int j2 = p / nx, j1 = p - j2 * nx;
    const float fj1 = (float)j1, fj2 = (float)j2;
    float2 acc[ZPL / 2];
#pragma unroll
    for (int q = 0; q < ZPL / 2; ++q) acc[q] = make_float2(0.f, 0.f);
    // every lane runs the same number of rounds (the shuffles need them all)
    for (int s0 = 0; s0 < nv; s0 += 2) {
      const bool live = s0 + half < nv;
      const int s = live ? s0 + half : s0;
      const float4 r = rot[vidx[s]];
      const float cs = r.x, sn = r.y;
      const float d1 = fj1 - c0, d2 = fj2 - c0;
      const float xc = c0 + cs * d1 + sn * d2, yc = c0 - sn * d1 + cs * d2;
      const float rr = fabsf(cs) + fabsf(sn) + 0.01f;
      const int xlo = max(0, (int)ceilf(xc - rr)), xhi = min(nx - 1, (int)floorf(xc + rr));
      const int ylo = max(0, (int)ceilf(yc - rr)), yhi = min(ny - 1, (int)floorf(yc + rr));
      const float* Ts = T + (size_t)s * ny * nx * nzp + 2 * lane;
      // candidate c = 3 i + k (x offset i, y offset k): weight and column
      // offset (-1: no footprint), with the forward's own operations
      auto cand = [&](int c, float& w, int& o) {
        const int i = (c * 11) >> 5, k = c - 3 * i;  // c / 3 for c <= 8
        const int xx = min(xlo + i, nx - 1), yy = min(ylo + k, ny - 1);
        const float di = __fsub_rn((float)xx, c0), dj = __fsub_rn((float)yy, c0);
        const float s1 = __fadd_rn(c0, __fsub_rn(__fmul_rn(cs, di), __fmul_rn(sn, dj)));
        const float s2 = __fadd_rn(c0, __fadd_rn(__fmul_rn(sn, di), __fmul_rn(cs, dj)));
        const bool ok = live && xlo + i <= xhi && ylo + k <= yhi && s1 >= fj1 - 1.f && s1 < fj1 + 1.f &&
                        s2 >= fj2 - 1.f && s2 < fj2 + 1.f;
        const float f1 = floorf(s1), f2 = floorf(s2);
        const float t1 = __fsub_rn(s1, f1), t2 = __fsub_rn(s2, f2);
        const float a1 = f1 == fj1 ? __fsub_rn(1.0f, t1) : t1;
        const float a2 = f2 == fj2 ? __fsub_rn(1.0f, t2) : t2;
        w = ok ? __fmul_rn(a1, a2) : 0.f;
        o = ok ? (yy * nx + xx) * nzp : -1;
      };
      // lane l of the group evaluates candidate l, every lane candidate 8;
      // the group shares them by shuffles and sums them in the order c = 0..8
      float wl, w8;
      int ol, o8;
      cand(lane, wl, ol);
      cand(8, w8, o8);
      if constexpr (RB == 0) {
#pragma unroll
        for (int c = 0; c < 9; ++c) {
          const float w = c < 8 ? __shfl_sync(0xffffffffu, wl, c, 8) : w8;
          const int o = c < 8 ? __shfl_sync(0xffffffffu, ol, c, 8) : o8;
          if (o >= 0) {
            const float* tp = Ts + o;
#pragma unroll
            for (int q = 0; q < ZPL / 2; ++q) {
              const float2 t = *reinterpret_cast<const float2*>(tp + 16 * q);
              acc[q].x = fmaf(w, t.x, acc[q].x);
              acc[q].y = fmaf(w, t.y, acc[q].y);
            }
          }
        }
      } else {
#pragma unroll
        for (int c0 = 0; c0 < 9; c0 += RB) {
          float wk[RB];
          float2 tk[RB][ZPL / 2];
#pragma unroll
          for (int k = 0; k < RB; ++k) {
            const int c = c0 + k;
            wk[k] = 0.f;
            if (c < 9) {  // resolved at compile time
              wk[k] = c < 8 ? __shfl_sync(0xffffffffu, wl, c, 8) : w8;
              const int o = c < 8 ? __shfl_sync(0xffffffffu, ol, c, 8) : o8;
              const float* tp = Ts + max(o, 0);
#pragma unroll
              for (int q = 0; q < ZPL / 2; ++q) tk[k][q] = ldg2_if(tp + 16 * q, o >= 0);
            }
          }
#pragma unroll
          for (int k = 0; k < RB; ++k) {
            if (c0 + k < 9) {
#pragma unroll
              for (int q = 0; q < ZPL / 2; ++q) {
                acc[q].x = fmaf(wk[k], tk[k][q].x, acc[q].x);
                acc[q].y = fmaf(wk[k], tk[k][q].y, acc[q].y);
              }
            }
          }
        }
      }
    }
#pragma unroll
    for (int q = 0; q < ZPL / 2; ++q) {  // even + odd slots
      acc[q].x += __shfl_xor_sync(0xffffffffu, acc[q].x, 8);
      acc[q].y += __shfl_xor_sync(0xffffffffu, acc[q].y, 8);
    }
    if (half || !own) continue;
    const size_t o = ((size_t)(j2 + g.pad) * g.L + j1 + g.pad) * nzp + 2 * lane;
#pragma unroll
    for (int q = 0; q < ZPL / 2; ++q) {
      const float vq[2] = {acc[q].x, acc[q].y};
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const size_t oe = o + 16 * q + e;
        if (2 * lane + 16 * q + e < g.nz) {
          float v = vq[e];
          if (prev) v += prev[oe];
          if (mode == 1 && v == 0.f) v = __int_as_float(0x7f800000);
          if (mode == 2) v = x[oe] * (v / asum[oe]);
          out[oe] = v;
        }
      }
    }
  }
}

}  // namespace spect
