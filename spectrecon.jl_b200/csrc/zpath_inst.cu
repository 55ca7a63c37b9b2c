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

namespace {
// k_zs_fz: 512 threads (index 0, 1) or 256 (index 2, 3: two blocks per SM at these registers)
const void* const kZsFz[4] = {(const void*)k_zs_fz<kZsNth, 8>, (const void*)k_zs_fz<kZsNth, 16>,
                              (const void*)k_zs_fz<kZsNth / 2, 8>, (const void*)k_zs_fz<kZsNth / 2, 16>};
const void* const kZsFx[2] = {(const void*)k_zs_fx<kZsNthX, 8>, (const void*)k_zs_fx<kZsNthX, 16>};
cudaError_t zs_launch(const void* k, int nth, int grid, size_t smem, cudaStream_t st, const ZArgs& a) {
  ZArgs c = a;
  void* args[] = {&c};
  return cudaLaunchKernel(k, dim3(grid), dim3(nth), args, smem, st);
}
}  // namespace

cudaError_t zstrip_setup(int max_smem) {
  for (int i = 0; i < 2; ++i)
    for (const void* k : {kZsFz[i], kZsFz[i + 2], kZsFx[i]}) {
      const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
      if (e != cudaSuccess) return e;
    }
  return cudaSuccess;
}

cudaError_t zstrip_occupancy(int w, int fz_nth, const size_t smem[2], int occ[2]) {
  const int i = w == 16 ? 1 : 0, f = fz_nth == kZsNth ? i : i + 2;
  const void* ks[2] = {kZsFz[f], kZsFx[i]};
  const int nth[2] = {fz_nth, kZsNthX};
  for (int j = 0; j < 2; ++j) {
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ[j], ks[j], nth[j], smem[j]);
    if (e != cudaSuccess) return e;
    if (occ[j] < 1) occ[j] = 1;
  }
  return cudaSuccess;
}

cudaError_t zs_fz_launch(int w, int nth, int grid, size_t smem, cudaStream_t st, const ZArgs& a) {
  return zs_launch(kZsFz[(w == 16 ? 1 : 0) + (nth == kZsNth ? 0 : 2)], nth, grid, smem, st, a);
}
cudaError_t zs_fx_launch(int w, int grid, size_t smem, cudaStream_t st, const ZArgs& a) {
  return zs_launch(kZsFx[w == 16 ? 1 : 0], kZsNthX, grid, smem, st, a);
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
