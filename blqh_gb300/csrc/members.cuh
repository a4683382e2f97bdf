// Orbit-member table shared by the spinful and the monolayer row generators:
// every member of every representative's translation orbit -> (representative
// index << 5) | translations that lead to it, in open addressing with linear
// probing over at least twice as many slots as members. One lookup replaces the
// reference's loop over the right-hand translations with a search for each.
#pragma once

#include "blqh_internal.h"

constexpr uint64_t MEMBER_EMPTY = ~0ULL;

struct MemberTable {
  const uint64_t* key;  // MEMBER_EMPTY: free
  const uint32_t* val;
  uint64_t mask;        // slots - 1
};

// 64-bit mixing (the finalizer of MurmurHash3) for the slots.
__device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x ^= x >> 33;
  x *= 0xff51afd7ed558ccdULL;
  x ^= x >> 33;
  x *= 0xc4ceb9fe1a85ec53ULL;
  x ^= x >> 33;
  return x;
}

__device__ __forceinline__ bool member_find(const MemberTable& T, uint64_t m, uint32_t* out) {
  uint64_t h = mix64(m) & T.mask;
  for (uint64_t probe = 0; probe <= T.mask; probe++) {
    const uint64_t k = __ldg(T.key + h);
    if (k == m) {
      *out = __ldg(T.val + h);
      return true;
    }
    if (k == MEMBER_EMPTY) return false;
    h = (h + 1) & T.mask;
  }
  return false;
}

// Every member rot(id_i, k), k in [0, period_i) (k = 0 only without translation
// symmetry), keyed to (i << 5) | k.
template <class ROT>
__global__ void k_member_insert(ROT rot, const uint64_t* __restrict__ id, const uint8_t* __restrict__ period,
                                int64_t dim, int orbits, uint64_t* __restrict__ key, uint32_t* __restrict__ val,
                                uint64_t mask, int* err) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += (int64_t)gridDim.x * blockDim.x) {
    const int P = orbits ? period[i] : 1;
    for (int k = 0; k < P; k++) {
      const uint64_t m = k == 0 ? id[i] : rot(id[i], k);
      uint64_t h = mix64(m) & mask;
      bool done = false;
      for (uint64_t probe = 0; probe <= mask; probe++) {
        const unsigned long long prev = atomicCAS(reinterpret_cast<unsigned long long*>(key + h),
                                                  (unsigned long long)MEMBER_EMPTY, (unsigned long long)m);
        if (prev == MEMBER_EMPTY || prev == m) {
          val[h] = (uint32_t)(i << 5) | (uint32_t)k;
          done = true;
          break;
        }
        h = (h + 1) & mask;
      }
      if (!done) atomicExch(err, 1);
    }
  }
}

// The table of a basis (at most `per_orbit` members per representative), in buffers owned by `G`.
template <class ROT>
MemberTable build_members(blqh_ctx* ctx, DevBufs& G, const blqh_basis* B, ROT rot, int orbits, int per_orbit,
                          int* derr) {
  const int64_t members = B->dim * (orbits ? per_orbit : 1);
  uint64_t slots = 1024;
  while (slots < (uint64_t)(2 * members)) slots <<= 1;
  uint64_t* key = G.add(static_cast<uint64_t*>(dev_alloc(ctx, slots * (sizeof(uint64_t) + sizeof(uint32_t)))));
  uint32_t* val = reinterpret_cast<uint32_t*>(key + slots);
  BLQH_TRY_CUDA(ctx, cudaMemsetAsync(key, 0xFF, slots * 8, ctx->stream));
  TimerScope tb(ctx, TM_BUILD);
  k_member_insert<<<grid_for(ctx, B->dim, 256), 256, 0, ctx->stream>>>(rot, B->d_id, B->d_period, B->dim, orbits, key,
                                                                       val, slots - 1, derr);
  BLQH_TRY_CUDA(ctx, cudaGetLastError());
  count_launch(ctx, TM_BUILD, 1);
  return {key, val, slots - 1};
}
