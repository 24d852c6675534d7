// bfvm_layout.cu -- conversion between the reference field layout and the
// device layout.
//
// Reference: one flat array, index ((i*ny + j)*nz + k)*S + d, z fastest with
// substrates interleaved (Cartesian_Mesh::voxel_index,
// BioFVM/BioFVM_mesh.cpp:1149-1158; Microenvironment::density_vector,
// BioFVM/BioFVM_microenvironment.cpp:1123-1130).
// Device:    f[d][k][j][i] with rows padded to nxp, x fastest.
// For each y-plane j the conversion is one transpose of the plane's rows x by
// the columns c = k*S + d, contiguous in the reference layout: column c is row
// (d, k, j) of the device field.  A block stages 64 x by 64 columns; both its
// loads and its stores are whole 256-byte rows, 16 loads in flight per thread.
// Bound by HBM: 512 MB each way at 200^3 x 4, pack and unpack together 211 us
// (4.9 TB/s).  (One transpose per substrate had read or written every 32-byte
// sector of the reference layout S times, 8 bytes of it each: 305 us, pack 104
// and unpack 206.)
#include "bfvm_internal.h"

namespace bfvm {

namespace {

constexpr int kLX = 64;  // x per block
constexpr int kLC = 64;  // columns (k*S + d) per block

// FP32 fields hold rho - off[s] (off null for FP64, where values are exact).
template <typename T>
__global__ void __launch_bounds__(256) pack_kernel(const double* __restrict__ aos, T* __restrict__ f, int nx, int ny,
                                                   int nz, int S, int nxp, const double* __restrict__ off) {
  __shared__ double tile[kLX][kLC + 1];
  const int c0 = blockIdx.x * kLC, i0 = blockIdx.y * kLX, j = blockIdx.z;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int nc = nz * S;
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const int r = ty + 8 * (m / 2), c = tx + 32 * (m % 2);
    if (i0 + r < nx && c0 + c < nc) tile[r][c] = aos[(static_cast<size_t>(i0 + r) * ny + j) * nc + c0 + c];
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    const int c = ty + 8 * m, col = c0 + c;
    if (col < nc) {
      const int k = col / S, s = col - k * S;
      const double o = off ? off[s] : 0.0;
      T* row = f + ((static_cast<size_t>(s) * nz + k) * ny + j) * nxp + i0;
#pragma unroll
      for (int i = tx; i < kLX; i += 32)
        if (i0 + i < nx) row[i] = static_cast<T>(off ? tile[i][c] - o : tile[i][c]);
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) unpack_kernel(const T* __restrict__ f, double* __restrict__ aos, int nx, int ny,
                                                     int nz, int S, int nxp, const double* __restrict__ off) {
  __shared__ double tile[kLX][kLC + 1];
  const int c0 = blockIdx.x * kLC, i0 = blockIdx.y * kLX, j = blockIdx.z;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int nc = nz * S;
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    const int c = ty + 8 * m, col = c0 + c;
    if (col < nc) {
      const int k = col / S, s = col - k * S;
      const double o = off ? off[s] : 0.0;
      const T* row = f + ((static_cast<size_t>(s) * nz + k) * ny + j) * nxp + i0;
#pragma unroll
      for (int i = tx; i < kLX; i += 32)
        if (i0 + i < nx) tile[i][c] = off ? static_cast<double>(row[i]) + o : static_cast<double>(row[i]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const int r = ty + 8 * (m / 2), c = tx + 32 * (m % 2);
    if (i0 + r < nx && c0 + c < nc) aos[(static_cast<size_t>(i0 + r) * ny + j) * nc + c0 + c] = tile[r][c];
  }
}

}  // namespace

template <typename T>
cudaError_t launch_pack(const double* aos, T* f, int nx, int ny, int nz, int S, int nxp, const double* off,
                        cudaStream_t st) {
  const dim3 grid((nz * S + kLC - 1) / kLC, (nx + kLX - 1) / kLX, ny), block(32, 8);
  pack_kernel<T><<<grid, block, 0, st>>>(aos, f, nx, ny, nz, S, nxp, off);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_unpack(const T* f, double* aos, int nx, int ny, int nz, int S, int nxp, const double* off,
                          cudaStream_t st) {
  const dim3 grid((nz * S + kLC - 1) / kLC, (nx + kLX - 1) / kLX, ny), block(32, 8);
  unpack_kernel<T><<<grid, block, 0, st>>>(f, aos, nx, ny, nz, S, nxp, off);
  return cudaGetLastError();
}

template cudaError_t launch_pack<double>(const double*, double*, int, int, int, int, int, const double*,
                                         cudaStream_t);
template cudaError_t launch_pack<float>(const double*, float*, int, int, int, int, int, const double*, cudaStream_t);
template cudaError_t launch_unpack<double>(const double*, double*, int, int, int, int, int, const double*,
                                           cudaStream_t);
template cudaError_t launch_unpack<float>(const float*, double*, int, int, int, int, int, const double*,
                                          cudaStream_t);

}  // namespace bfvm
