// What an issuing warp of the dK/dV kernel has to see before it issues the products of query half h of item n.
//
// Two warps issue: `scores` S^T = K Q^T and dV += P^T dO, the other one dP^T = V dO^T and dK += dS^T Q. Per half they
// issue their second product of item n (dV or dK) and then their first product of item n + 1 over the columns it has read.
// Every operand and what says that it is there:
//
//   product        operand          covered by
//   S^T(n + 1)     K                kv_full, in front of the loop
//                  Q(n + 1)         WAIT_NEXT (q_full) at half 0
//                  S^T columns      WAIT_IN: P^T(n) of the half is in them, and dV(n) of the half is issued before, by this warp
//   dV(n)          P^T(n)           WAIT_IN (p_ready of the half)
//                  dO(n)            WAIT_TILE (do_full) at half 0. p_ready does not cover it: a compute warp arrives there
//                                   before it waits for dP^T(n), the only other product that reads dO(n)
//   dP^T(n + 1)    V                kv_full, in front of the loop
//                  dO(n + 1)        WAIT_NEXT (do_full) at half 0
//                  dP^T columns     WAIT_IN: dS^T(n) of the half is in them, and dK(n) of the half is issued before
//   dK(n)          dS^T(n)          WAIT_IN (ds_ready of the half)
//                  Q(n)             WAIT_IN too: dS^T(n) was computed from S^T(n), whose MMA had waited for q_full
//
// Plain C++ for the host as well, where a model of the kernel's roles runs on it.
#pragma once

#if defined(__CUDACC__)
#define ZX_DW_FN __host__ __device__ __forceinline__
#else
#define ZX_DW_FN inline
#endif

namespace zx {

enum DkdvWait : unsigned {
  WAIT_IN = 1,     // p_ready (scores) or ds_ready of half h, item n
  WAIT_NEXT = 2,   // q_full (scores) or do_full of item n + 1: operand of the next item's first product
  WAIT_TILE = 4,   // do_full of item n: operand of dV
};

ZX_DW_FN constexpr unsigned dkdv_waits(bool scores, int h, bool has_next) {
  return WAIT_IN | (h == 0 && has_next ? WAIT_NEXT : 0u) | (h == 0 && scores ? WAIT_TILE : 0u);
}

}  // namespace zx
