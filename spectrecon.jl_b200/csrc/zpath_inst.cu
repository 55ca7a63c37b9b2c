// zpath_inst.cu -- instantiations and launchers of the fused projector pair
// (zpath.cuh) and of the large-plane kernels (zstrip.cuh), compiled as a unit
// of its own.
#include "zpath.cuh"
#include "zstrip.cuh"

namespace spect {

namespace {
constexpr int kGridY = 65535;  // blocks of a grid's second dimension at most
// [x tasks a thread - 1][rotation :two, :one]
void (*const kZfwd[2][2])(const ZArgs) = {{k_zfwd<1, false>, k_zfwd<1, true>}, {k_zfwd<2, false>, k_zfwd<2, true>}};
// launch with programmatic stream serialisation (grid_wait, zpath.cuh) where
// `early`: the blocks of a kernel start as the one before it in the stream
// runs out, which hides its launch latency and its prologue; a kernel after
// another library's or a copy starts when that has ended, as ever.  An SM that
// never idles keeps its split of L1 and shared memory, so the kernels whose
// gathers live on L1 start early only where they are short (zearly).
// Measured, all against none: projection of 8 views of 64x64x64 26.6 -> 20.4
// us, OS-EM on 90x90x53 1295 -> 1104 us; OS-EM on 256x256x200 33.3 -> 35.0 ms
// (and 33.3 with the rule).
template <class... P, class... A>
cudaError_t launch_next(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}
void (*const kZadj[2])(const ZArgs) = {k_zadj<8>, k_zadj<16>};

}  // namespace

cudaError_t zrot_adj_setup() {
  cudaError_t e = cudaSuccess;
  for (const void* k : {(const void*)k_zrot_adj<false>, (const void*)k_zrot_adj<true>})
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kZrotThreads * 2 * kZrotList * 8);
  return e;
}

cudaError_t zpath_setup(int max_smem) {
  cudaError_t e = zrot_adj_setup();
  for (const auto k : {kZfwd[0][0], kZfwd[0][1], kZfwd[1][0], kZfwd[1][1], kZadj[0], kZadj[1], k_zs_fz, k_zs_fx})
    if (e == cudaSuccess) e = cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
  return e;
}

cudaError_t zfwd_launch(int grid, cudaStream_t st, const ZArgs& a) {
  return launch_next(zearly(a.g, a.nv), kZfwd[a.t.nxt - 1][a.r1 ? 1 : 0], grid, a.t.nth, a.t.smem, st, a);
}

cudaError_t zreduce_launch(int grid, cudaStream_t st, const float* part, int nv, int ny, int G, int nxz, int vec,
                           float* out, const float* y, const float* bg, const ViewList& vidx) {
  return launch_next(true, vec == 4 ? k_reduce_parts<4> : k_reduce_parts<1>, grid, 256, 0, st, part, nv, ny, G, nxz, out, y,
                     bg, vidx);
}

cudaError_t zadj_launch(int grid, cudaStream_t st, const ZArgs& a) {
  return launch_next(true, kZadj[a.t.w == 16 ? 1 : 0], grid, a.t.nth, a.t.smem, st, a);
}

cudaError_t zrot_adj_launch(const ZGeom& g, int sms, cudaStream_t st, const float* T, size_t zero, const float4* rot,
                            const Rot1View* r1, const ViewList& vidx, int nv, const float* prev, float* out, const float* x,
                            const float* asum, int mode) {
  if (zero / g.nzp > (size_t)kZrotColumnMask) return cudaErrorInvalidValue;  // zgroup_views rules it out
  const ZRotTile r = zrot_tile(g, nv, sms);
  const auto kernel = r1 ? k_zrot_adj<true> : k_zrot_adj<false>;
  return launch_next(zearly(g, nv), kernel, r.grid, r.nth, r.smem, st, g, r, T, (int)(zero / g.nzp), rot, r1, vidx, nv, prev, out, x,
                     asum, mode);
}

cudaError_t zs_fz_launch(const ZsTiles& t, int grid, cudaStream_t st, const ZArgs& a) {
  return launch_next(zearly(a.g, a.nv), k_zs_fz, grid, t.fz_nth, t.fz_smem, st, a);
}
cudaError_t zs_fx_launch(const ZsTiles& t, int grid, cudaStream_t st, const ZArgs& a) {
  return launch_next(true, k_zs_fx, grid, t.fx_nth, t.fx_smem, st, a);
}

cudaError_t zto_iz_launch(const ZGeom& g, cudaStream_t st, const float* img, float* iz) {
  return launch_next(true, k_to_iz, dim3((g.nx + 31) / 32, g.ny, (g.nzp + 31) / 32), dim3(32, 8), 0, st, g, img, iz);
}

cudaError_t zrot_fwd_launch(const ZGeom& g, int planes, cudaStream_t st, const float* iz, const float4* rot,
                            const int* vidx, float* P) {
  return launch_next(zearly(g, planes / g.ny), k_zrot_fwd, dim3(planes, (g.nx + 31) / 32), 256,
                     sizeof(float) * 33 * zround(g.nz, 4), st, g, iz, rot, vidx, P);
}

cudaError_t zt_to_z_launch(const ZGeom& g, int planes, cudaStream_t st, const float* src, float* dst,
                            const float* att, const int* vidx) {
  const int step = kGridY / g.ny * g.ny;  // whole slots a launch
  for (int p0 = 0; p0 < planes; p0 += step) {
    const int n = planes - p0 < step ? planes - p0 : step;
    k_t_to_z<<<dim3((g.nx + 31) / 32, n, (g.nzp + 31) / 32), dim3(32, 8), 0, st>>>(
        g, src + (size_t)p0 * g.nz * g.nx, dst + (size_t)p0 * g.nx * g.nzp, att, vidx + p0 / g.ny);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t zfrom_iz_launch(const ZGeom& g, cudaStream_t st, const float* iz, float* dst, const float* asum, int mode) {
  return launch_next(true, k_from_iz, dim3((g.nx + 31) / 32, g.ny, (g.nz + 31) / 32), dim3(32, 8), 0, st, g, iz, dst, asum,
                     mode);
}

cudaError_t zatten_launch(const ZGeom& g, int nview, cudaStream_t st, const float* muz, const float4* rot,
                          const Rot1View* r1, float dy, float* att) {
  const size_t stack = (size_t)g.ny * g.nx * g.nzp;  // floats of a view
  for (int v0 = 0; v0 < nview; v0 += kGridY) {
    const dim3 grid(g.nx, nview - v0 < kGridY ? nview - v0 : kGridY);
    if (r1) k_zatten<true><<<grid, g.nzp, 0, st>>>(g, muz, rot + v0, r1 + v0, dy, att + v0 * stack);
    else k_zatten<false><<<grid, g.nzp, 0, st>>>(g, muz, rot + v0, r1, dy, att + v0 * stack);
  }
  return cudaGetLastError();
}

}  // namespace spect
