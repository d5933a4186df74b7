// patch.cuh -- device pieces of the kernels over cell patches (PatchPlan).
#pragma once

#include "launch.cuh"

namespace db2 {
namespace dev {

// A patch's plan arrays and staging sizes.
struct PatchView {
  const PatchHdr* hdr;
  const uint16_t* conn;
  const uint32_t* nodes;
  const uint4* chunks;
  double* partial;
  int64_t npartial;
  int stride;           // staged cells of a local node
  int nx, nv;           // room for the patch's nodes (even) and vertices
  uint32_t ahead;       // patches in flight on the device
};

__device__ __forceinline__ PatchHdr patch_header(const PatchHdr* hdr, uint32_t i) {
  const uint4* s = reinterpret_cast<const uint4*>(hdr + i);
  const uint4 a = __ldg(s), b = __ldg(s + 1);
  PatchHdr h;
  h.cell0 = a.x;
  h.node0 = a.y;
  h.chunk0 = a.z;
  h.chunks = a.w;
  h.ncells = uint16_t(b.x & 0xffffu);
  h.nnodes = uint16_t(b.x >> 16);
  h.nverts = uint16_t(b.y & 0xffffu);
  h.ngroups = uint16_t(b.y >> 16);
  return h;
}

// Copies the patch's jobs to shared memory (16-byte cp.async; complete after
// patch_jobs_wait and a barrier).
__device__ __forceinline__ void patch_jobs_copy(const PatchView& q, const PatchHdr& h, unsigned char* jobs) {
  const uint4* src = q.chunks + h.chunk0;
  const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(jobs));
  for (uint32_t i = threadIdx.x; i < h.chunks; i += blockDim.x)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 16u * i), "l"(src + i) : "memory");
}
__device__ __forceinline__ void patch_jobs_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Sends the plan data of a patch that starts later to L2.
template <int K>
__device__ __forceinline__ void patch_prefetch(const PatchView& q, const PatchHdr& h) {
  auto prefetch = [](const void* p, uint32_t bytes) {
    const char* b = static_cast<const char*>(p);
    for (uint32_t i = 128u * threadIdx.x; i < bytes; i += 128u * blockDim.x)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(b + i));
  };
  constexpr uint32_t KC = patch_conn(K) / 4;
  prefetch(q.nodes + h.node0, h.nnodes * 4u);
  prefetch(reinterpret_cast<const uint2*>(q.conn) + size_t(h.cell0) * KC, h.ncells * KC * 8u);
  prefetch(q.chunks + h.chunk0, h.chunks * 16u);
}

// A cell's local nodes (8 x each).
template <int K>
struct PatchCell {
  static constexpr int KC = patch_conn(K) / 4;
  uint2 w[KC];
  __device__ __forceinline__ void load(const PatchView& q, const PatchHdr& h, int c) {
    const uint2* conn = reinterpret_cast<const uint2*>(q.conn) + (size_t(h.cell0) + c) * KC;
#pragma unroll
    for (int i = 0; i < KC; ++i) w[i] = __ldg(conn + i);
  }
  __device__ __forceinline__ uint32_t off(int j) const {
    const uint32_t v = (j & 2) ? w[j >> 2].y : w[j >> 2].x;
    return (j & 1) ? v >> 16 : v & 0xffffu;
  }
};

struct PatchJobs {
  const uint32_t* dest;
  const PatchGroup* groups;
  const uint16_t* codes;
};
__device__ __forceinline__ PatchJobs patch_jobs(const PatchHdr& h, const unsigned char* jobs) {
  PatchJobs J;
  J.dest = reinterpret_cast<const uint32_t*>(jobs);
  J.groups = reinterpret_cast<const PatchGroup*>(jobs + 128u * h.ngroups);
  J.codes = reinterpret_cast<const uint16_t*>(jobs + 128u * h.ngroups +
                                              PatchPlan::pad16(h.ngroups * uint32_t(sizeof(PatchGroup))));
  return J;
}

// Nodes shared between patches: their partial sums in patch order.
template <int BS>
__global__ void __launch_bounds__(256) k_patch_sum(const uint32_t* __restrict__ shared,
                                                   const uint32_t* __restrict__ ptr, int64_t n,
                                                   const double* __restrict__ partial, int64_t npartial,
                                                   double* __restrict__ y, int64_t nnodes) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t node = __ldg(shared + i), s0 = __ldg(ptr + i), s1 = __ldg(ptr + i + 1);
  double acc[BS];
#pragma unroll
  for (int e = 0; e < BS; ++e) acc[e] = 0.0;
  for (uint32_t s = s0; s < s1; ++s)
#pragma unroll
    for (int e = 0; e < BS; ++e) acc[e] += __ldg(partial + int64_t(e) * npartial + s);
#pragma unroll
  for (int e = 0; e < BS; ++e) y[int64_t(e) * nnodes + node] = acc[e];
}

}  // namespace dev

// The view of a pattern's patches, for a kernel with `ctas` blocks an SM.
dev::PatchView patch_view(const PatchPlan& B, int ctas);

}  // namespace db2
