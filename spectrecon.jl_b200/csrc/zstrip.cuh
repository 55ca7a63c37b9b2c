// zstrip.cuh -- the forward projector for planes too large for k_zfwd's
// shared memory (e.g. 256x256x200 with a 65-tap PSF), on the same z-fastest
// layouts and with the same sampling, pair passes and plane walk as zpath.cuh,
// over plane tiles; the two passes are kernels of their own that exchange
// planes through the device buffer Q, whose rows are already the x pass's
// pair lines.
//
// forward (project!, src/project.jl:77-135):
//   k_zs_fz  item (slot, two planes y, tile of tx columns): gather the rotated,
//            attenuated columns, z pass -> Q[slot][y][row pair][x][2]
//   k_zs_fx  item (partial view of the forward walk, tile of row pairs): per
//            plane the rows of Q (copied one plane ahead), x pass accumulated
//            over the partial's planes -> part
// The adjoint is k_zadj (zpath.cuh) on row tiles.  Every output goes through
// the operations of the fused kernels in the same order (z then x), so the
// two paths agree bit for bit.
#pragma once
#include "zpath.cuh"

namespace spect {

// ------------------------------------------------------------------------
// k_zs_fz: forward gather and z pass of a tile of tx columns in two adjacent
// planes (their samples share taps: about 3.3 image columns are read for the
// eight taps of an x, where one plane reads 2.4 for four), tasks of 8 outputs
// of a column pair; the first half of the warps runs the first plane's, so a
// warp's weights stay uniform.  Two barriers an item: the z pass runs while
// the next item's taps and attenuation are prefetched into L2.  64 registers
// and tiles for 320 threads, three blocks an SM: the bound is HBM (attenuation
// and image read, Q written: 1.1 GB for 8 views of 256x256x200, 65 taps) and
// the latency of the gather's loads, not the FMAs.  Measured there: 392 us
// (16-output tasks on two blocks 411 us, one plane an item 425 us, double ZB
// with one barrier 511 us -- it takes the L1; one line a lane 394 us).
// Shared memory: [2 x 2 x (table | geoW tx x 2 float4 | geoO tx int)]
// [ZB 2 x tx / 2 * vst f2].
__global__ void __launch_bounds__(kZsThreads, 3) k_zs_fz(const __grid_constant__ ZArgs a) {
  const int* const vidx = a.vidx.ptr();
  extern __shared__ float4 smem4[];
  constexpr int W = 8;
  const ZGeom& g = a.g;
  const int nx = g.nx, ny = g.ny, nz = g.nz, nzp = g.nzp, hs = g.hs, ts = g.ts, tx = a.tx, vst = a.zvst;
  const int trow = ztable_floats(g), tid = threadIdx.x, nth = blockDim.x, R0 = g.R0, hz = g.hz;
  const int bufsz = trow + 8 * tx + zround(tx, 4), zbs = (tx / 2) * vst;
  float* const base = reinterpret_cast<float*>(smem4);
  f2* const ZB0 = reinterpret_cast<f2*>(base + 4 * bufsz);
  const int ntx = (nx + tx - 1) / tx, nyp = ny / 2, nitems = a.nv * nyp * ntx, nz4 = (nz + 3) / 4, nzb = (nz + W - 1) / W;
  const int nrp = (nz + 1) / 2;
  const size_t Lz = (size_t)g.L * nzp;
  const float rnz4 = 1.0f / nz4;
  auto place = [&](int item, int& slot, int& y, int& X0) {  // the item's slot, first plane and column
    const int xt = item % ntx, sy = item / ntx;
    slot = sy / nyp;
    y = 2 * (sy - slot * nyp);
    X0 = xt * tx;
  };
  auto prepare = [&](int item, float* buf) {  // tables and sample geometry of an item
    int slot, y, X0;
    place(item, slot, y, X0);
    const int v = vidx[slot];
    const float* src = a.tab + (((size_t)a.viewset[v] * ny + y) * 2) * trow;
    for (int k = 4 * tid; k < trow; k += 4 * nth) {
      cp16(buf + k, src + k);
      cp16(buf + bufsz + k, src + 2 * trow + k);
    }
    const float4 r = a.rot[v];
    const int cols = min(tx, nx - X0);
    for (int c = tid; c < 2 * cols; c += nth) {
      const int p = c >= cols, x = c - p * cols;
      float4* const geoW = reinterpret_cast<float4*>(buf + p * bufsz + trow);
      float4 w;
      int off;
      zgeo(g, r.x, r.y, r.z != 0.f, X0 + x, y + p, w, off);
      geoW[2 * x] = make_float4(w.x, w.x, w.y, w.y);
      geoW[2 * x + 1] = make_float4(w.z, w.z, w.w, w.w);
      reinterpret_cast<int*>(geoW + 2 * tx)[x] = off;
    }
  };
  for (int k = tid; k < 2 * zbs; k += nth) ZB0[k] = 0;  // rows outside the data stay zero
  int item = blockIdx.x, hb = 0;
  if (item < nitems) prepare(item, base);
  cp_wait();
  __syncthreads();
  grid_wait();
  const int hi4 = (tid >> 2) & 1, hth = nth / 2, pz = tid >= hth, tz = tid - pz * hth;
  for (; item < nitems; item += gridDim.x, hb ^= 1) {
    int slot, y, X0;
    place(item, slot, y, X0);
    const int txp = min(tx, nx - X0) / 2;
    const float* const buf = base + 2 * hb * bufsz;
    float* const next = base + 2 * (hb ^ 1) * bufsz;
    const bool more = item + gridDim.x < nitems;
    if (more) prepare(item + gridDim.x, next);
    for (int p = 0; p < 2; ++p) {
      const float4* const geoW = reinterpret_cast<const float4*>(buf + p * bufsz + trow);
      const int* const geoO = reinterpret_cast<const int*>(geoW + 2 * tx);
      const float* att = a.att + (((size_t)vidx[slot] * ny + y + p) * nx + X0) * nzp;
      for (int u = tid; u < txp * nz4; u += nth) {  // unit (column pair, z group)
        const int xp = zdiv(u, rnz4), z4 = u - xp * nz4;
        f2 lo[2], hi[2];
#pragma unroll
        for (int c = 0; c < 2; ++c)
          zsample4(a.img + geoO[2 * xp + c] + 4 * z4, nzp, Lz, geoW + 2 * (2 * xp + c),
                   att + (2 * xp + c) * nzp + 4 * z4, lo[c], hi[c]);
        float4* o = reinterpret_cast<float4*>(ZB0 + p * zbs + xp * vst + R0 + 4 * z4);
        o[hi4] = zturn(hi4 ? hi[0] : lo[0], hi4 ? hi[1] : lo[1]);
        o[hi4 ^ 1] = zturn(hi4 ? lo[0] : hi[0], hi4 ? lo[1] : hi[1]);
      }
    }
    cp_wait();
    __syncthreads();
    if (more) {  // the next item's taps (two runs of two columns) and attenuation on their way into L2
      int slot1, y1, X1;
      place(item + gridDim.x, slot1, y1, X1);
      const int cols = min(tx, nx - X1);
      for (int c = tid; c < 2 * cols; c += nth) {
        const int p = c >= cols, x = c - p * cols;
        const int off = reinterpret_cast<const int*>(next + p * bufsz + trow + 8 * tx)[x];
        prefetch_l2_bulk(a.img + off, 2 * nzp * (unsigned)sizeof(float));
        prefetch_l2_bulk(a.img + off + Lz, 2 * nzp * (unsigned)sizeof(float));
        if (x == 0)
          prefetch_l2_bulk(a.att + (((size_t)vidx[slot1] * ny + y1 + p) * nx + X1) * nzp,
                           cols * nzp * (unsigned)sizeof(float));
      }
    }
    // z pass: task (column pair, W rows) of plane y + pz -> Q
    const float* const Wt = buf + pz * bufsz;
    const f2* const Wd = reinterpret_cast<const f2*>(Wt);
    const int2 rg = *reinterpret_cast<const int2*>(Wt + 2 * hs + ts);
    f2* const Qp = reinterpret_cast<f2*>(a.Q) + ((size_t)slot * ny + y + pz) * nrp * nx + X0;
    const float rtxp = 1.0f / txp;
    for (int t = tz; t < txp * nzb; t += hth) {
      const int zb = zdiv(t, rtxp), xp = t - zb * txp, z0 = W * zb;
      f2 o[W];
#pragma unroll
      for (int k = 0; k < W; ++k) o[k] = 0;
      const f2* col = ZB0 + pz * zbs + xp * vst;
      zpass2<W>(Wd, rg.x, rg.y, col + z0, o);
      zclamp<W>(o, Wt + 2 * hs, Wt + 2 * hs + hz, hz, z0, nz, col[R0], col[R0 + nz - 1]);
      f2* q = Qp + (size_t)(z0 / 2) * nx + 2 * xp;
#pragma unroll
      for (int m = 0; m < W / 2; ++m)
        if (z0 + 2 * m < nz) __stcs(reinterpret_cast<float4*>(q + (size_t)m * nx), zturn(o[2 * m], o[2 * m + 1]));
    }
    __syncthreads();
  }
}

// planes [j0, j1) of partial view id (walk block + slot) of the forward walk;
// false where no block and slot of that sum meet
__device__ __forceinline__ bool zs_segment(const ZArgs& a, int id, int& slot, int& j0, int& j1) {
  const int ny = a.g.ny, n = a.nv * ny, G = a.G;
  // the walk's blocks and slots grow together: find the slot whose ids hold id
  for (slot = 0; slot < a.nv; ++slot) {
    const int b1 = zblock_of((long long)(slot + 1) * ny - 1, n, G);
    if (id <= b1 + slot) break;
  }
  if (slot == a.nv) return false;
  const int b = id - slot;
  if (b < zblock_of((long long)slot * ny, n, G)) return false;
  const int q0 = (int)((long long)b * n / G), q1 = (int)((long long)(b + 1) * n / G);
  j0 = max(q0 - slot * ny, 0);
  j1 = min(q1 - slot * ny, ny);
  return j0 < j1;
}

// ------------------------------------------------------------------------
// k_zs_fx: forward x pass and depth sum, one task of kZfwdX outputs a thread
// and plane; the rows of Q and the table of the next plane are copied
// (cp.async) while a plane is worked on, one barrier a plane, two blocks an
// SM.  Bound: FFMA2 and the shared-memory pipe; 256x256x200, 8 views 295 ->
// 255 us.  Shared memory: 2 x [XB tzp * bst f2 | table].
__global__ void __launch_bounds__(kZThreads, 1) k_zs_fx(const __grid_constant__ ZArgs a) {
  const int* const vidx = a.vidx.ptr();
  extern __shared__ float4 smem4[];
  constexpr int X = kZfwdX;
  const ZGeom& g = a.g;
  const int nx = g.nx, ny = g.ny, nz = g.nz, hs = g.hs, ts = g.ts, tzp = a.tz / 2, bst = a.xbst, C0 = g.C0, hx = g.hx;
  const int trow = ztable_floats(g), bufsz = 2 * tzp * bst + trow, tid = threadIdx.x, nth = blockDim.x;
  float* const base = reinterpret_cast<float*>(smem4);
  const int nrp = (nz + 1) / 2, ntz = (nrp + tzp - 1) / tzp, nitems = (a.G + a.nv) * ntz, n2 = nx / 2;
  for (int k = tid; k < 2 * bufsz; k += nth) base[k] = 0.f;  // columns outside the data stay zero
  __syncthreads();
  grid_wait();
  const int xb = tid / tzp, zl = tid - xb * tzp, x0 = X * xb;  // this thread's task: row pair zl, columns x0 ..
  const int dr = nth / n2, dc = nth - dr * n2, r0 = tid / n2, c0 = tid - r0 * n2;
  for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
    const int zt = item % ntz, id = item / ntz;  // partial view, planes j0 .. j1 - 1 of its slot
    int slot, j0, j1;
    if (!zs_segment(a, id, slot, j0, j1)) continue;
    const int Z0 = zt * tzp, rows = min(tzp, nrp - Z0), set = a.viewset[vidx[slot]];
    int y = (int)((long long)j0 * a.t.ystep % ny);
    const bool mine = x0 < nx && zl < rows;
    auto fetch = [&](int yy, float* buf) {  // rows (16 bytes: columns 2 c, 2 c + 1 of a row pair) and table
      const float* Qp = a.Q + (((size_t)slot * ny + yy) * nrp + Z0) * 2 * nx;
      for (int r = r0, c = c0; r < rows;) {
        cp16(buf + 2 * (r * bst + C0 + 2 * c), Qp + (size_t)r * 2 * nx + 4 * c);
        r += dr;
        c += dc;
        if (c >= n2) {
          c -= n2;
          ++r;
        }
      }
      const float* src = a.tab + (((size_t)set * ny + yy) * 2) * trow;
      for (int k = 4 * tid; k < trow; k += 4 * nth) cp16(buf + 2 * tzp * bst + k, src + k);
    };
    fetch(y, base);
    cp_wait();
    __syncthreads();
    f2 acc[X];
#pragma unroll
    for (int k = 0; k < X; ++k) acc[k] = 0;
    for (int jj = j0; jj < j1; ++jj) {
      float* const buf = base + ((jj - j0) & 1) * bufsz;
      y = y + a.t.ystep < ny ? y + a.t.ystep : y + a.t.ystep - ny;
      if (jj + 1 < j1) fetch(y, base + (((jj - j0) & 1) ^ 1) * bufsz);
      if (mine) {
        const float* Wt = buf + 2 * tzp * bst;
        const int2 rg = *reinterpret_cast<const int2*>(Wt + 2 * hs + ts + 2);
        const f2* row = reinterpret_cast<const f2*>(buf) + zl * bst;
        f2 o[X];  // the plane's own sum, then onto the depth sum, as k_zfwd
#pragma unroll
        for (int k = 0; k < X; ++k) o[k] = 0;
        zpass2<X>(reinterpret_cast<const f2*>(Wt) + g.zpw, rg.x, rg.y, row + x0, o);
        const float* EL = Wt + 2 * hs + 2 * g.hz;
        zclamp<X>(o, EL, EL + hx, hx, x0, nx, row[C0], row[C0 + nx - 1]);
#pragma unroll
        for (int k = 0; k < X; ++k) acc[k] = add2(acc[k], o[k]);
      }
      cp_wait();
      __syncthreads();
    }
    if (mine) zstore_part<X>(a.part + (size_t)id * nz * nx, acc, nx, nz, 2 * (Z0 + zl), x0);
  }
}

}  // namespace spect
