// Per-kernel fluxes from one process on two devices, with a stand-in for the CUDA runtime (this
// program's own functions take its place): memory is the host's, a launch is only looked at.  A kernel
// that asks for more than 48 KB of shared memory must have been allowed it on the device it runs on.
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <utility>
#include <vector>

#include "aph_hydro.h"

static int g_device = 0, g_large = 0, g_refused = 0;
static std::map<std::pair<int, const void *>, size_t> g_allowed;  // (device, kernel) -> bytes
static dim3 g_grid, g_block;
static size_t g_smem;
static cudaStream_t g_stream;

extern "C" {
cudaError_t cudaGetDevice(int *d) { return *d = g_device, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { return *p = std::calloc(1, n), cudaSuccess; }
cudaError_t cudaFree(void *p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { return std::memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemset(void *d, int v, size_t n) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) g_allowed[{g_device, f}] = (size_t)v;
  return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st *stream) {
  return g_grid = grid, g_block = block, g_smem = smem, g_stream = stream, 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
  *grid = g_grid, *block = g_block, *smem = g_smem, *(cudaStream_t *)stream = g_stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) { return *k = (cudaKernel_t)f, cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void **, size_t smem, cudaStream_t) {
  if (smem <= 48 * 1024) return cudaSuccess;
  ++g_large;
  auto it = g_allowed.find({g_device, (const void *)k});
  if (it == g_allowed.end() || it->second < smem) ++g_refused;
  return cudaSuccess;
}
}

int main() {
  // 64 blocks of 32^2 cells: seven lines to a segment of PPM, some 54 KB
  const int n = 32, ng = 3, ni = n + 2 * ng, nblocks = 64;
  std::vector<double> field(8 * ni * ni, 1.0);
  aph_hydro_params p{};
  p.ndim = 2;
  p.nghost = ng;
  p.nvar = 5;
  p.recon = APH_RECON_PPM;
  p.rsolver = APH_RSOLVER_HLLC;
  p.gm1 = 1.4 - 1.0;
  p.dfloor = p.pfloor = 1e-15;
  p.cfl = 0.4;
  p.exact = 1;
  aph_block b{};
  b.cons = b.prim = b.gamma = b.flux[0] = b.flux[1] = field.data();
  b.nx[0] = b.nx[1] = n;
  b.nx[2] = 1;
  b.dx[0] = b.dx[1] = 1.0 / n;
  b.dx[2] = 1.0;
  const std::vector<aph_block> blocks(nblocks, b);
  for (g_device = 0; g_device < 2; ++g_device) {
    aph_pack pack = nullptr;
    if (aph_pack_create(&p, blocks.data(), nblocks, &pack) != APH_OK ||
        aph_hydro_calculate_fluxes(pack, p.recon, p.rsolver, nullptr) != APH_OK) {
      std::fprintf(stderr, "%s\n", aph_last_error());
      return 2;
    }
    std::printf("device %d: %d launches above 48 KB, %d not allowed there\n", g_device, g_large, g_refused);
    aph_pack_destroy(pack);
  }
  std::fflush(stdout);
  std::_Exit(g_large == 4 && g_refused == 0 ? 0 : 1);
}
