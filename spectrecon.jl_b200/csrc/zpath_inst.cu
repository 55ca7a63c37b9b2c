// zpath_inst.cu -- instantiations and launchers of the fused projector pair
// (zpath.cuh) and of the large-plane kernels (zstrip.cuh), compiled as a unit
// of its own.
#include "zpath.cuh"
#include "zstrip.cuh"

namespace spect {

namespace {
// [x tasks a thread - 1][rotation :two, :one]
const void* const kZfwd[2][2] = {{(const void*)k_zfwd<1, false>, (const void*)k_zfwd<1, true>},
                                 {(const void*)k_zfwd<2, false>, (const void*)k_zfwd<2, true>}};
const void* const kZadj[2] = {(const void*)k_zadj<8>, (const void*)k_zadj<16>};

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
  for (const void* k : {kZfwd[0][0], kZfwd[0][1], kZfwd[1][0], kZfwd[1][1]})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
  for (const void* k : {(const void*)k_zs_fz, (const void*)k_zs_fx})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
  for (const void* k : kZadj)
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
  return e;
}

cudaError_t zfwd_launch(int grid, cudaStream_t st, const ZArgs& a) {
  ZArgs c = a;
  void* args[] = {&c};
  return cudaLaunchKernel(kZfwd[a.t.nxt - 1][a.r1 ? 1 : 0], dim3(grid), dim3(a.t.nth), args, a.t.smem, st);
}

cudaError_t zreduce_launch(int grid, cudaStream_t st, const float* part, int nv, int ny, int G, int nxz, float* out,
                           const float* y, const float* bg, const int* vidx) {
  if (nxz % 4 == 0) k_reduce_parts<4><<<grid, 256, 0, st>>>(part, nv, ny, G, nxz, out, y, bg, vidx);
  else k_reduce_parts<1><<<grid, 256, 0, st>>>(part, nv, ny, G, nxz, out, y, bg, vidx);
  return cudaGetLastError();
}

cudaError_t zadj_launch(int grid, cudaStream_t st, const ZArgs& a) {
  ZArgs c = a;
  void* args[] = {&c};
  return cudaLaunchKernel(kZadj[a.t.w == 16 ? 1 : 0], dim3(grid), dim3(a.t.nth), args, a.t.smem, st);
}

cudaError_t zrot_adj_launch(const ZGeom& g, int sms, cudaStream_t st, const float* T, size_t zero, const float4* rot,
                            const Rot1View* r1, const int* vidx, int nv, const float* prev, float* out, const float* x,
                            const float* asum, int mode) {
  const ZRotTile r = zrot_tile(g, nv, sms);
  const auto kernel = r1 ? k_zrot_adj<true> : k_zrot_adj<false>;
  kernel<<<r.grid, r.nth, r.smem, st>>>(g, r, T, (int)(zero / g.nzp), rot, r1, vidx, nv, prev, out, x, asum, mode);
  return cudaGetLastError();
}

cudaError_t zs_fz_launch(const ZsTiles& t, int grid, cudaStream_t st, const ZArgs& a) {
  k_zs_fz<<<grid, t.fz_nth, t.fz_smem, st>>>(a);
  return cudaGetLastError();
}
cudaError_t zs_fx_launch(const ZsTiles& t, int grid, cudaStream_t st, const ZArgs& a) {
  k_zs_fx<<<grid, t.fx_nth, t.fx_smem, st>>>(a);
  return cudaGetLastError();
}

cudaError_t zto_iz_launch(const ZGeom& g, cudaStream_t st, const float* img, float* iz) {
  k_to_iz<<<dim3((g.nx + 31) / 32, g.ny, (g.nzp + 31) / 32), dim3(32, 8), 0, st>>>(g, img, iz);
  return cudaGetLastError();
}

cudaError_t zt_to_z_launch(const ZGeom& g, int planes, cudaStream_t st, const float* src, float* dst,
                            const float* att, const int* vidx) {
  k_t_to_z<<<dim3((g.nx + 31) / 32, planes, (g.nzp + 31) / 32), dim3(32, 8), 0, st>>>(g, src, dst, att, vidx);
  return cudaGetLastError();
}

cudaError_t zfrom_iz_launch(const ZGeom& g, cudaStream_t st, const float* iz, float* dst, const float* asum, int mode) {
  k_from_iz<<<dim3((g.nx + 31) / 32, g.ny, (g.nz + 31) / 32), dim3(32, 8), 0, st>>>(g, iz, dst, asum, mode);
  return cudaGetLastError();
}

cudaError_t zatten_launch(const ZGeom& g, int nview, cudaStream_t st, const float* muz, const float4* rot,
                          const Rot1View* r1, float dy, float* att) {
  if (r1) k_zatten<true><<<dim3(g.nx, nview), g.nzp, 0, st>>>(g, muz, rot, r1, dy, att);
  else k_zatten<false><<<dim3(g.nx, nview), g.nzp, 0, st>>>(g, muz, rot, r1, dy, att);
  return cudaGetLastError();
}

}  // namespace spect
