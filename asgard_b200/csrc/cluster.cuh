// Thread-block clusters: barrier, rank, and stores to the shared memory of
// every CTA of a cluster.
#pragma once

namespace asgk
{
// every thread of every CTA of the cluster; orders shared-memory accesses
// before it (remote ones too) before those after it
__device__ __forceinline__ void cluster_sync()
{
  __syncwarp(); // the barrier's aligned form is taken by whole warps
  asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
               "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ int cluster_rank()
{
  int r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// *p = v in the shared memory of all CS CTAs of the cluster
template<int CS, typename T>
__device__ __forceinline__ void put_all(T *p, T v)
{
  static_assert(sizeof(T) == 4 || sizeof(T) == 8, "float or double");
  unsigned const a = static_cast<unsigned>(__cvta_generic_to_shared(p));
#pragma unroll
  for (int r = 0; r < CS; r++)
  {
    unsigned ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(r));
    if constexpr (sizeof(T) == 8)
      asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(ra), "d"(v) : "memory");
    else
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(ra), "f"(v) : "memory");
  }
}
} // namespace asgk
