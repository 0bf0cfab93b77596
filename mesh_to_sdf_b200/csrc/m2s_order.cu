// Distance-ordered cell list: the voxel viewer's index buffer
// (mesh_to_sdf_client/src/sdf.rs:63-71) computed on the device.
//
// The client sorts 0..n by `data[i].total_cmp(&data[j])` with rayon's stable
// `par_sort_by`, then takes `minmax` of the data as its iso limits.  Here each
// distance becomes a 32-bit key that orders like total_cmp (negative floats:
// all bits flipped; others: sign bit set) as the library's stable LSD radix
// sort (m2s_sort.cu) first reads it, its index being its value — equal
// distances keep index order, as in the stable sort — and the same read that
// counts the digits finds the extremes (16.7M cells 1.08 -> 0.57 ms).
#include <cuda_runtime.h>

#include "m2s_internal.cuh"

using namespace m2s;

extern "C" {

int m2s_sort_cells_by_distance_device(const float* d_sdf, uint64_t n, uint32_t* d_order, float* d_minmax,
                                      void* stream) {
  if (n && (!d_sdf || !d_order)) return M2S_ERR_INVALID_ARGUMENT;
  int st;
  if ((st = require_device())) return st;
  return sort_floats(d_sdf, n, d_order, d_minmax, (cudaStream_t)stream);
}

int m2s_sort_cells_by_distance(const float* sdf, uint64_t n, uint32_t* order, float minmax[2], void* stream) {
  if (n && (!sdf || !order)) return M2S_ERR_INVALID_ARGUMENT;
  if (n > 0xFFFFFFFFull) return M2S_ERR_INVALID_ARGUMENT;
  int st;
  if ((st = require_device())) return st;
  if (n == 0) return M2S_OK;
  cudaStream_t s = (cudaStream_t)stream;
  DevBuf<float> d, mm;
  DevBuf<uint32_t> o;
  if ((st = d.alloc(n, s)) || (st = o.alloc(n, s)) || (st = mm.alloc(2, s))) return st;
  M2S_CUDA(cudaMemcpyAsync(d.p, sdf, 4 * n, cudaMemcpyHostToDevice, s));
  if ((st = sort_floats(d.p, n, o.p, minmax ? mm.p : nullptr, s))) return st;
  M2S_CUDA(cudaMemcpyAsync(order, o.p, 4 * n, cudaMemcpyDeviceToHost, s));
  if (minmax) M2S_CUDA(cudaMemcpyAsync(minmax, mm.p, 8, cudaMemcpyDeviceToHost, s));
  M2S_CUDA(cudaStreamSynchronize(s));
  return M2S_OK;
}

}  // extern "C"
