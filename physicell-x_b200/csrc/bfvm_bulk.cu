// bfvm_bulk.cu -- bulk (per-voxel) sources and sinks.
//
// Reference: Microenvironment::simulate_bulk_sources_and_sinks
// (BioFVM/BioFVM_microenvironment.cpp:1327-1368).  The reference asks three
// host callbacks for every voxel's supply rate S, target density T and
// uptake rate U; here they are device arrays in the field's device layout,
// uploaded once (bfvm_set_bulk_rates), and one elementwise pass applies
//     temp2 = T * S;  rho = fma(dt, temp2, rho);     (the reference's g++
//     temp3 = ((U + S) * dt) + 1;  rho /= temp3;      build contracts the
//                                                     first update, not temp3)
// so FP64 results equal the reference's bit for bit.  The pass reads the
// field, the three rate arrays and writes the field: 40 bytes per
// voxel-substrate in FP64 (36 in FP32).
#include <type_traits>

#include "bfvm_internal.h"

namespace bfvm {

namespace {

// A warp per row at a time, two neighbouring voxels per lane (rows are whole
// 128-byte lines, so the 16-byte loads are aligned; a row's last pair may end
// in its padding, which is read and not written).  Bound by HBM; with one
// voxel per thread of a flat index, a 64-bit division each, the pass took
// 83 us at 160 x 200 x 120 x 3, now 69.
template <typename T>
__global__ void __launch_bounds__(256) bulk_kernel(T* __restrict__ f, const double* __restrict__ rates, size_t plane,
                                                   int nx, int nxp, long long rows, int rows_per_s, double dt,
                                                   const double* __restrict__ off) {
  using Pair = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
  const int lane = threadIdx.x & 31;
  const long long nw = static_cast<long long>(gridDim.x) * (blockDim.x / 32);
  for (long long r = static_cast<long long>(blockIdx.x) * (blockDim.x / 32) + threadIdx.x / 32; r < rows; r += nw) {
    const double o = off ? off[r / rows_per_s] : 0.0;
    const size_t q0 = static_cast<size_t>(r) * nxp;
#pragma unroll 2
    for (int i = 2 * lane; i < nx; i += 64) {
      const size_t q = q0 + i;
      const double2 s_rate = __ldg(reinterpret_cast<const double2*>(rates + q));
      const double2 target = __ldg(reinterpret_cast<const double2*>(rates + plane + q));
      const double2 u_rate = __ldg(reinterpret_cast<const double2*>(rates + 2 * plane + q));
      const Pair in = *reinterpret_cast<const Pair*>(f + q);
      auto one = [&](double rho, double sr, double tg, double ur) {
        double t2 = tg;
        t2 *= sr;
        rho = __fma_rn(dt, t2, rho);
        double t3 = ur;
        t3 += sr;
        t3 *= dt;
        t3 += 1.0;
        rho /= t3;
        return rho;
      };
      Pair res;
      res.x = static_cast<T>(one(static_cast<double>(in.x) + o, s_rate.x, target.x, u_rate.x) - o);
      if (i + 1 < nx) {
        res.y = static_cast<T>(one(static_cast<double>(in.y) + o, s_rate.y, target.y, u_rate.y) - o);
        *reinterpret_cast<Pair*>(f + q) = res;
      } else {
        f[q] = res.x;
      }
    }
  }
}

}  // namespace

template <typename T>
cudaError_t launch_bulk(T* f, const double* rates, int nx, int ny, int nz, int S, int nxp, double dt,
                        const double* off, int sm_count, cudaStream_t st) {
  const long long rows = static_cast<long long>(S) * nz * ny;
  const size_t plane = static_cast<size_t>(rows) * nxp;
  long long blocks = (rows + 7) / 8;
  const long long cap = static_cast<long long>(sm_count) * 8;
  if (blocks > cap) blocks = cap;
  bulk_kernel<T><<<static_cast<unsigned>(blocks), 256, 0, st>>>(f, rates, plane, nx, nxp, rows, nz * ny, dt, off);
  return cudaGetLastError();
}

template cudaError_t launch_bulk<double>(double*, const double*, int, int, int, int, int, double, const double*, int,
                                         cudaStream_t);
template cudaError_t launch_bulk<float>(float*, const double*, int, int, int, int, int, double, const double*, int,
                                        cudaStream_t);

}  // namespace bfvm
