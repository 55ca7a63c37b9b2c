// zpath_api.h -- host-visible part of the fused projector pair (zpath.cuh):
// geometry of the z-fastest layouts, kernel arguments, shared-memory sizes and
// the launchers defined in zpath_inst.cu.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace spect {

// sizes shared by the zpath kernels (computed once per plan on the host)
struct ZGeom {
  int nx, ny, nz, nzp, L, pad;
  float c0;         // rotation centre (nx - 1)/2, 0-based
  int px, pz, hx, hz;
  int R0, C0;       // first data row (z pass) / column (x pass) of the padded buffers
  int zpw, xpw;     // window taps of the z and x passes (shifted, multiples of 8)
  int hs, ts;       // weight-row and tail-row lengths of one direction
};

__host__ __device__ constexpr int zround(int v, int m) { return (v + m - 1) / m * m; }
inline ZGeom zgeom_make(int nx, int ny, int nz, int px, int pz, int pad) {
  ZGeom g{};
  g.nx = nx;
  g.ny = ny;
  g.nz = nz;
  g.nzp = zround(nz, 16);
  g.pad = pad;
  g.L = nx + 2 * pad;
  g.c0 = (float)((nx - 1) * 0.5);
  g.px = px;
  g.pz = pz;
  g.hx = (px - 1) / 2;
  g.hz = (pz - 1) / 2;
  g.R0 = zround(g.hz, 4);
  g.C0 = zround(g.hx, 4);
  g.zpw = zround(g.R0 - g.hz + pz, 8);
  g.xpw = zround(g.C0 - g.hx + px, 8);
  g.hs = g.zpw + g.xpw;
  g.ts = zround(2 * g.hx + 2 * g.hz, 4) < 4 ? 4 : zround(2 * g.hx + 2 * g.hz, 4);
  return g;
}

// smallest 2 * odd >= v: pair lines (float2 elements) whose 16-byte chunk
// count is odd, so the eight lanes of a 128-bit shared access phase hit
// distinct bank groups
__host__ __device__ constexpr int zstride2(int v) {
  return ((zround(v, 2) / 2) % 2 == 1) ? zround(v, 2) : zround(v, 2) + 2;
}
// floats of one plane's table of one direction: weights of the z and x pass,
// each stored twice | tails or folds | tap ranges (first 4-tap block and
// 4-tap blocks of the z pass, then of the x pass)
__host__ __device__ inline int ztable_floats(const ZGeom& g) { return 2 * g.hs + g.ts + 4; }

// tiling of a pair-pass kernel: task width w, row tile tz (even; ntile tiles
// cover nz), strides (float2) of the z-pass and x-pass lines, row buffers,
// threads, resident blocks per SM, depth step of the plane walk, x tasks a
// thread (k_zfwd), shared memory
struct ZTile {
  int w, tz, ntile, vst, bst, nxb, nth, occ, ystep, nxt;
  size_t smem;
};
constexpr int kZfwdX = 8;       // outputs of an x-pass and of a z-pass task of k_zfwd
constexpr int kZfwdZ = 8;
constexpr int kZfwdNT = 2;      // x tasks a thread at most (their outputs stay in registers)
constexpr int kZadjX = 8;       // outputs of an x-pass task of k_zadj
constexpr int kZThreads = 640;  // threads per SM the pair-pass kernels' registers allow (96 each)

// :one rotation of a view (src/rotatez.jl:240-322): mode 0 copy (theta == 0
// mod 2pi), 1 rot_f90 only (theta close to m*pi/2), 2 rot_f90 + shears; tn =
// tan(phi/2), sn = -sin(phi), phi = theta - m*pi/2 (src/rotatez.jl:249-272)
struct Rot1View {
  double tn, sn;
  int m, mode;
};

// plan views of a call's slots: a device table, or up to kViewsInline of them
// in the kernel's own parameters (a short index list of a caller then needs no
// copy to the device, about 6 us a call and a break in the kernels' overlap)
constexpr int kViewsInline = 32;
struct ViewList {
  const int* p;
  int v[kViewsInline];
  // one pointer for either, taken once a kernel (parameter memory is
  // addressable there): a choice at every read cost k_zfwd up to 8 %
  __device__ const int* ptr() const { return p ? p : v; }
};

struct ZArgs {
  ZGeom g;
  ZTile t;
  const Rot1View* r1;   // [nview] :one rotation; null for :two
  const float* tab;     // [set][y][2][ztable_floats]: forward, adjoint tables
  const float* img;     // IZ
  const float* att;     // ATT
  const float4* rot;    // [view] (cos(2pi - theta), sin(2pi - theta), theta == 0, theta)
  ViewList vidx;        // plan view of each slot
  const int* viewset;   // [nview] PSF set of each view
  int nv;
  int G;                // blocks of the forward walk (partial views: block + slot)
  float* part;          // partial views [G + nv][nz][nx]
  const float* views;   // k_zadj input [nv][nz][nx]
  float* T;             // k_zadj output [nv][ny][nx][nzp]
  float* Q;             // plane exchange of the large-plane kernels (zstrip.cuh), [nv][ny][row pair][nx][2]
  int tx, tz;           // their column and row tile sizes
  int zvst, xbst;       // their line strides (f2)
};

// k_zfwd shared memory (zpath.cuh)
// (one: the eight taps a column of the :one rotation in place of four)
inline size_t zfwd_smem(const ZGeom& g, const ZTile& t, bool one) {
  return sizeof(float) * (2 * (size_t)ztable_floats(g) + (one ? 20 : 8) * (size_t)g.nx + (one ? 0 : zround(g.nx, 4)) +
                          2 * ((size_t)(g.nx / 2) * t.vst + (size_t)((g.nz + 1) / 2) * t.bst));
}
// k_zadj shared memory (zpath.cuh)
inline size_t zadj_smem(const ZGeom& g, const ZTile& t) {
  return sizeof(float) * (2 * ((size_t)(g.nx / 2) * t.vst + (size_t)t.nxb * (t.tz / 2) * t.bst) +
                          3 * (size_t)ztable_floats(g));
}
// depth step of a plane walk: coprime to ny, near the golden section of ny
inline int zdepth_step(int ny) {
  auto gcd = [](int a, int b) {
    while (b) {
      const int r = a % b;
      a = b;
      b = r;
    }
    return a;
  };
  int s = (int)(0.618 * ny);
  if (s < 1) s = 1;
  while (gcd(s, ny) != 1) ++s;
  return s;
}
// tiling of k_zadj: the least modelled time per view and depth.  A thread's
// task is w outputs of two lines in each pass; wider tasks read fewer shared
// bytes per FMA, row tiles cut the shared memory of a block so that several
// blocks (or a second row buffer) hide each other's barriers, and fewer than
// 16 warps per SM no longer hide the latencies.
// `want` fixes a field that is not 0, for comparisons; where nothing of that
// form fits it is left out of account.
struct ZadjForm {
  int w, ntile, nxb;
};
inline ZTile zadj_tile(const ZGeom& g, size_t optin, const ZadjForm& want = {}) {
  ZTile best{};
  double bc = 0;
  for (int w : {16, 8})
    for (int nt = 1; nt <= (g.nz + 1) / 2; ++nt) {
      if ((want.w && w != want.w) || (want.ntile && nt != want.ntile)) continue;
      ZTile t{};
      t.w = w;
      t.tz = zround((g.nz + nt - 1) / nt, nt > 1 ? 8 : 2);  // tiles of whole tasks
      t.ntile = (g.nz + t.tz - 1) / t.tz;
      if (t.ntile != nt) continue;
      t.vst = zstride2(w * ((t.tz + w - 1) / w) + g.zpw);
      t.bst = zstride2(kZadjX * ((g.nx + kZadjX - 1) / kZadjX) + g.xpw);
      const int zt = (g.nx / 2) * ((t.tz + w - 1) / w), xt = (t.tz / 2) * ((g.nx + kZadjX - 1) / kZadjX);
      const int most = w == 16 || zt > xt ? zt : xt, rounds = (most + kZThreads - 1) / kZThreads;
      t.nth = zround((most + rounds - 1) / rounds, 32);
      for (int nxb : {1, 2}) {
        if (want.nxb && nxb != want.nxb) continue;
        t.nxb = nxb;
        t.smem = zadj_smem(g, t);
        if (t.smem > optin) continue;
        const int so = (int)((optin + 1024) / (t.smem + 1024)), ro = kZThreads / t.nth;
        t.occ = so < ro ? so : ro;
        if (t.occ > 16) t.occ = 16;
        if (nxb > 1 && t.occ > 1 && !want.nxb) continue;  // several blocks overlap already
        const double warps = t.occ * t.nth / 32.0;
        const double rz = (double)((zt + t.nth - 1) / t.nth), rx = (double)((xt + t.nth - 1) / t.nth);
        double c = t.ntile * t.nth * (rz * w * (w == 8 ? 1.15 : 1.0) + rx * kZadjX * 1.15);  // thread slots x outputs
        c *= warps < 16 ? 16 / warps : 1.0;
        c *= (t.occ > 1 || nxb > 1) ? 1.0 : 1.25;
        if (!best.w || c < bc) {
          best = t;
          bc = c;
        }
      }
    }
  if (!best.w && (want.w || want.ntile || want.nxb)) return zadj_tile(g, optin);
  best.ystep = zdepth_step(g.ny);
  return best;
}

// tiling of k_zfwd (w == 0: the plane does not fit): kZfwdNT x tasks a thread
// (their outputs stay in registers over the planes); threads for them, for
// half the z tasks and for a quarter of the gather units
inline ZTile zfwd_tile(const ZGeom& g, size_t optin, bool one) {
  ZTile t{};
  const int nxw = (g.nx + kZfwdX - 1) / kZfwdX, nzb = (g.nz + kZfwdZ - 1) / kZfwdZ, xt = (g.nz + 1) / 2 * nxw;
  if (xt > kZfwdNT * kZThreads) return t;
  t.tz = zround(g.nz, 2);
  t.ntile = t.nxb = 1;
  t.vst = zstride2(kZfwdZ * nzb + g.zpw);
  t.bst = zstride2(kZfwdX * nxw + g.xpw);
  t.smem = zfwd_smem(g, t, one);
  if (t.smem > optin) return t;
  const int zh = ((g.nx / 2) * nzb + 1) / 2, gq = ((g.nx / 2) * ((g.nz + 3) / 4) + 3) / 4;
  t.nxt = xt <= kZThreads ? 1 : kZfwdNT;
  const int xh = (xt + t.nxt - 1) / t.nxt, most = xh > zh ? xh : zh;
  t.nth = zround(most > gq ? most : gq, 32);
  if (t.nth > kZThreads) t.nth = kZThreads;
  const int so = (int)((optin + 1024) / (t.smem + 1024));
  auto blocks = [&](int nth) { return so < kZThreads / nth ? so : kZThreads / nth; };
  // twice the threads where shared memory leaves the SM short of warps (one
  // slice of 128x128: 64 threads on ten blocks 49 us, 32 on fourteen 58 us)
  if (2 * t.nth <= kZThreads && 2 * blocks(2 * t.nth) > blocks(t.nth) && so * t.nth < kZThreads) t.nth *= 2;
  t.occ = blocks(t.nth);
  t.ystep = zdepth_step(g.ny);
  t.w = kZfwdX;
  return t;
}

// tiling of the large-plane kernels (zstrip.cuh): k_zs_fz on equal tiles of tx
// columns in two planes with a thread for two of its 8-output tasks, k_zs_fx on tiles of
// tz rows (about 320 tasks of kZfwdX outputs of a row pair, one a thread, so
// that two blocks share an SM); nth = 0: a tile does not fit
constexpr int kZsThreads = 320;  // k_zs_fz threads, three blocks an SM
struct ZsTiles {
  int tx, zvst, fz_nth, fz_occ, tz, xbst, fx_nth, fx_occ;
  size_t fz_smem, fx_smem;
};
inline ZsTiles zs_tiles(const ZGeom& g, size_t optin) {
  ZsTiles t{};
  auto occupancy = [&](size_t smem, int nth, int threads) {
    const int so = (int)((optin + 1024) / (smem + 1024)), ro = threads / nth;
    return so < ro ? so : ro;
  };
  const int nzb = (g.nz + 7) / 8;
  int tmax = 2 * (320 / nzb);
  if (tmax > 32) tmax = 32;
  t.tx = zround((g.nx + (g.nx + tmax - 1) / tmax - 1) / ((g.nx + tmax - 1) / tmax), 4);
  if (t.tx > g.nx) t.tx = g.nx;
  t.zvst = zstride2(8 * nzb + g.zpw);
  t.fz_smem = sizeof(float) * (4 * ((size_t)ztable_floats(g) + 8 * t.tx + zround(t.tx, 4)) + 2 * (size_t)t.tx * t.zvst);
  int nth = 2 * zround((t.tx / 2 * nzb + 1) / 2, 32);  // two tasks a thread
  if (nth > kZsThreads) nth = kZsThreads;
  const int nxw = (g.nx + kZfwdX - 1) / kZfwdX, nrp = (g.nz + 1) / 2;
  int tzp = 320 / nxw;
  if (tzp < 1) tzp = 1;
  if (tzp > nrp) tzp = nrp;
  t.tz = 2 * tzp;
  t.xbst = zstride2(kZfwdX * nxw + g.xpw);
  t.fx_smem = sizeof(float) * 2 * (2 * (size_t)tzp * t.xbst + ztable_floats(g));
  const int fxn = zround(tzp * nxw, 32);
  if (t.fz_smem > optin || t.fx_smem > optin || fxn > kZThreads) return t;
  t.fz_nth = nth;
  t.fx_nth = fxn;
  t.fz_occ = occupancy(t.fz_smem, nth, 3 * kZsThreads);
  t.fx_occ = occupancy(t.fx_smem, fxn, kZThreads);
  return t;
}

// tiling of k_zrot_adj: tiles of tx x ty image columns, S groups of threads
// over the slots, vb slots whose hits are listed at a time (one thread tests
// one column of one slot).  16 columns a tile (8 of over 160 z): the blocks
// are short enough to fill the last wave (128x128x80, 15 views: 46 us; 32
// columns 48 us, 8 columns 46 us; 256x256x200, 8 views: 226 us, 8 columns 216
// us).
constexpr int kZrotU = 2;          // units (column, four z) a thread
constexpr int kZrotList = 9;       // list entries of a pair: its candidates at most
constexpr int kZrotThreads = 512;  // nzp <= 256: 16 columns x 40 z groups / 2 = 320 threads a group at most
struct ZRotTile {
  int tx, ty, S, vb, nth, grid;
  size_t smem;
};
inline ZRotTile zrot_tile(const ZGeom& g, int nv, int sms) {
  ZRotTile r{};
  const int n4 = g.nzp / 4, C = n4 <= 40 ? 16 : 8;
  r.tx = 4;
  r.ty = C / 4;
  r.grid = ((g.nx + r.tx - 1) / r.tx) * ((g.nx + r.ty - 1) / r.ty);
  const int gth = zround((C * n4 + kZrotU - 1) / kZrotU, 32);
  // slot groups: the fewest waves of blocks times their share of the slots,
  // 15 % for each further group's lists and final sum (128x128x80, 15 views:
  // two groups 42 us, one 46 us -- its last wave is nearly empty; 64x64x64, 64
  // views: four groups 31 us)
  double best = 0;
  for (int S = 1; S <= nv && S * gth <= kZrotThreads; ++S) {
    const int slots = sms * (2 * kZrotThreads / (S * gth));
    const double cost = (double)((r.grid + slots - 1) / slots) / S * (1 + 0.15 * (S - 1));
    if (S == 1 || cost < best) {
      best = cost;
      r.S = S;
    }
  }
  r.nth = r.S * gth;
  r.vb = r.nth / C;
  r.smem = (size_t)r.nth * 2 * kZrotList * 8;
  return r;
}

// k_zrot_adj's lists keep a T column number below the count of hits in one
// word: a group's columns and the zero column behind them are numbered in
// kZrotColumnBits bits
constexpr int kZrotColumnBits = 27;
constexpr int kZrotColumnMask = (1 << kZrotColumnBits) - 1;
// views of a group whose planes hold `slot` floats a view: about 1 GiB of
// planes, and, where the gather adjoint runs, column numbers within their bits
// (single slices on the split kernels: 512 views of 512x512x1 hold 2^27
// columns in half that memory)
inline int zgroup_views(int nx, int nview, size_t slot, bool gather) {
  size_t n = ((size_t)1 << 30) / (sizeof(float) * slot);
  if (n > (size_t)nview) n = nview;
  const size_t most = (size_t)kZrotColumnMask / ((size_t)nx * nx);
  if (gather && n > most) n = most;
  return n < 1 ? 1 : (int)n;
}

// short work: nv stacks of planes of nx x nz, below about 100 us a kernel.  The
// kernels whose gathers live on L1 start early there.  Measured, two OS-EM
// iterations, none of them early and all: 8 views of 64x64x64 (2.1 M samples)
// 0.81 -> 0.69 ms; 15 and 25 views of 128x128x80 (20 M, 33 M) 2.09 -> 2.12 and
// 3.23 -> 3.32 ms; 12 views of 192x192x120 (53 M) 6.57 -> 6.88; 8 views of
// 256x256x128 (67 M) 8.13 -> 9.04; of 256x256x200 (105 M) 13.6 -> 14.4.  The line
// keeps the large losses out; the crossing itself lies below 20 M.
inline bool zearly(const ZGeom& g, int nv) { return (long long)nv * g.nx * g.ny * g.nz <= (1LL << 25); }

// launchers (zpath_inst.cu)
cudaError_t zpath_setup(int max_smem);  // shared-memory limits of the fused kernels (zrot_adj_setup's too)
cudaError_t zrot_adj_setup();
cudaError_t zfwd_launch(int grid, cudaStream_t st, const ZArgs& a);
// views (EM ratio with y, bg) of nv slots from the partial views of a walk by
// G blocks, vec (4 or 1) elements a thread
cudaError_t zreduce_launch(int grid, cudaStream_t st, const float* part, int nv, int ny, int G, int nxz, int vec,
                           float* out, const float* y, const float* bg, const ViewList& vidx);
cudaError_t zadj_launch(int grid, cudaStream_t st, const ZArgs& a);
cudaError_t zrot_adj_launch(const ZGeom& g, int sms, cudaStream_t st, const float* T, size_t zero, const float4* rot,
                            const Rot1View* r1, const ViewList& vidx, int nv, const float* prev, float* out, const float* x,
                            const float* asum, int mode);  // T[zero ..]: a column of zeros; r1: null for :two
cudaError_t zto_iz_launch(const ZGeom& g, cudaStream_t st, const float* img, float* iz);
cudaError_t zrot_fwd_launch(const ZGeom& g, int planes, cudaStream_t st, const float* iz, const float4* rot,
                            const int* vidx, float* P);
cudaError_t zt_to_z_launch(const ZGeom& g, int planes, cudaStream_t st, const float* src, float* dst,
                            const float* att, const int* vidx);
cudaError_t zfrom_iz_launch(const ZGeom& g, cudaStream_t st, const float* iz, float* dst, const float* asum, int mode);
// large-plane kernels
cudaError_t zs_fz_launch(const ZsTiles& t, int grid, cudaStream_t st, const ZArgs& a);
cudaError_t zs_fx_launch(const ZsTiles& t, int grid, cudaStream_t st, const ZArgs& a);
cudaError_t zatten_launch(const ZGeom& g, int nview, cudaStream_t st, const float* muz, const float4* rot,
                          const Rot1View* r1, float dy, float* att);

}  // namespace spect
