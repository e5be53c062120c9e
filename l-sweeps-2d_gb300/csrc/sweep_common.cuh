// Shared by the sweep-front kernels: PTX helpers (clusters, mbarriers with
// bounded waits, bulk copies, remote stores) and the right-hand sides of a slot.
#pragma once
#include "common.cuh"
#include "internal.h"

#include <cuda_bf16.h>

namespace lsw {

constexpr unsigned kSuspendNs = 1000000;          // try_wait sleeps up to 1 ms (woken by the phase)

__device__ __forceinline__ unsigned saddr(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned mapa(unsigned a, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_init(uint64_t* b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(b)) : "memory");
}
// arrive on the barrier at the same offset in CTA `rank` of the cluster (release, cluster scope)
__device__ __forceinline__ void mbar_arrive_remote(uint64_t* b, unsigned rank) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(mapa(saddr(b), rank))
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* b, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(saddr(b)), "r"(parity), "r"(kSuspendNs)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* b, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(saddr(b)), "r"(parity), "r"(kSuspendNs)
      : "memory");
  return ok != 0;
}
// Bounded wait (see the file comment): gives up after `limit` clock cycles,
// or at once when the CTA's abort flag is up (abort_flag == nullptr: a wait
// that only the limit ends, for the drain before leaving).
template <bool CLUSTER>
__device__ __forceinline__ bool mbar_wait(uint64_t* b, unsigned parity, int* err, volatile int* abort_flag,
                                          long long limit) {
  auto tw = [&]() { return CLUSTER ? mbar_try_wait_cluster(b, parity) : mbar_try_wait(b, parity); };
  if (tw()) return true;
  const long long t0 = clock64();
  while (true) {
    if (abort_flag && *abort_flag) return false;
    if (tw()) return true;
    if (clock64() - t0 > limit) {
      if (abort_flag) *abort_flag = 1;
      atomicOr(err, 2);
      return false;
    }
  }
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   saddr(dst)),
               "l"(src), "r"(bytes), "r"(saddr(bar))
               : "memory");
}
__device__ __forceinline__ void named_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
// store into CTA `rank`'s shared memory; the bytes complete the transaction
// count of that CTA's mbarrier at the same offset as `bar`
__device__ __forceinline__ void st_async(float2* p, unsigned rank, float2 v, uint64_t* bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(
                   mapa(saddr(p), rank)),
               "f"(v.x), "f"(v.y), "r"(mapa(saddr(bar), rank))
               : "memory");
}
__device__ __forceinline__ void st_async2(float2* p, unsigned rank, float2 v0, float2 v1, uint64_t* bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                   mapa(saddr(p), rank)),
               "f"(v0.x), "f"(v0.y), "f"(v1.x), "f"(v1.y), "r"(mapa(saddr(bar), rank))
               : "memory");
}
__device__ __forceinline__ void st_async(double2* p, unsigned rank, double2 v, uint64_t* bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(
                   mapa(saddr(p), rank)),
               "d"(v.x), "d"(v.y), "r"(mapa(saddr(bar), rank))
               : "memory");
}
__device__ __forceinline__ void red_add(float2* p, float2 v) {
  atomicAdd(&p->x, v.x);
  atomicAdd(&p->y, v.y);
}
__device__ __forceinline__ void red_add(double2* p, double2 v) {
  atomicAdd(&p->x, v.x);
  atomicAdd(&p->y, v.y);
}

// D += A B, m16n8k16, bf16 operands, FP32 accumulation
__device__ __forceinline__ void mma_bf16(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3,
                                         unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
               "{%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ bool is_line(int gnode, int m, int N) {
  // interface lines k_b(J), k_b(J)+1 for J = 0..N-2 (the trace1/traceN rows
  // zeroed by getSeparatedRHS)
  if (gnode < m || gnode > (m + 1) * (N - 1)) return false;
  const int r = gnode % (m + 1);
  return r == m || r == 0;
}

struct SlotCoef {
  double2 c_oi_x, c_io_x, c_oi_y, c_io_y;
};

template <typename T>
__device__ __forceinline__ cx_t<T> rhs_elem(const FrontArgs& a, const DevCell& cl, const DevSlot& s,
                                            const SlotCoef& cf, const cx_t<T>* tr, int k, int j) {
  using C = cx_t<T>;
  C z = czero<C>();
  switch (s.kind) {
    case SK_CELLVEC: {
      const double2 v = a.x_in[(long long)s.rhs * a.x_stride + (long long)k * cl.ny + j];
      return to_c(v, z);
    }
    case SK_DIR_X: {
      if (k == s.xo) return cmul(to_c(cf.c_oi_x, z), tr[s.in_lr1 + j]);
      if (k == s.xi) return cneg(cmul(to_c(cf.c_io_x, z), tr[s.in_lr0 + j]));
      return z;
    }
    case SK_DIR_Y: {
      if (j == s.yo) return cmul(to_c(cf.c_oi_y, z), tr[s.in_ud1 + k]);
      if (j == s.yi) return cneg(cmul(to_c(cf.c_io_y, z), tr[s.in_ud0 + k]));
      return z;
    }
    case SK_CORNER: {
      // L-shaped sources: trace0 set L0 = {(xo, y): y inside yo} u {(x, yo): x inside xo},
      // trace1 set L1 likewise on (xi, yi) (computeLTraceIndexSets, 1119-1277);
      // rhs[L0] = A01 v1, rhs[L1] = -A10 v0 with the trace values of extractLTraces
      // (UD0 > LR0 > UD1 > LR1 where lines cross).
      const bool yin_o = (j - s.yo) * s.dy > 0;
      const bool yin_i = (j - s.yi) * s.dy > 0;
      if (k == s.xo) {
        if (!yin_o) return z;
        const C v = (j == s.yi) ? tr[s.in_ud1 + s.xi] : tr[s.in_lr1 + j];
        return cmul(to_c(cf.c_oi_x, z), v);
      }
      const bool xin_i = (k - s.xi) * s.dx > 0;
      if (k == s.xi) {
        if (j == s.yo) return cmul(to_c(cf.c_oi_y, z), tr[s.in_ud1 + k]);
        if (j == s.yi) {
          C r = cneg(cmul(to_c(cf.c_io_x, z), tr[s.in_lr0 + j]));
          cfms(r, to_c(cf.c_io_y, z), tr[s.in_ud0 + k]);
          return r;
        }
        if (yin_i) return cneg(cmul(to_c(cf.c_io_x, z), tr[s.in_lr0 + j]));
        return z;
      }
      if (xin_i) {
        if (j == s.yo) return cmul(to_c(cf.c_oi_y, z), tr[s.in_ud1 + k]);
        if (j == s.yi) return cneg(cmul(to_c(cf.c_io_y, z), tr[s.in_ud0 + k]));
      }
      return z;
    }
    default:
      return z;
  }
}

}  // namespace lsw
