/* blqh_gpu_debug.h — inspection entry points of libblqh_gpu.so.
 *
 * They expose internals that the tests check. Not part of the reference's
 * interface. blqh_debug_sector_index needs no device.
 */
#ifndef BLQH_GPU_DEBUG_H
#define BLQH_GPU_DEBUG_H

#include "blqh_gpu.h"

#ifdef __cplusplus
extern "C" {
#endif

/* Dense index of each state among those the reference's depth-first
 * enumeration inserts into basis_set (BLQH_without_spin/basis.cpp:199-259),
 * i.e. its insertion order; -1 for states outside the sector. nvalid_out
 * (optional) receives the number of such states. */
int blqh_debug_sector_index(const blqh_sector* s, int64_t n, const uint64_t* states, int64_t* index_out,
                            int64_t* nvalid_out);

/* Layout the mixed-precision SpMV reads for this matrix: 1 when the
 * blocked copy (row blocks x column tiles, x staged in shared memory) has been
 * built with (2-byte column, FP32 value) entries, 2 when it has been built in
 * dictionary form (4-byte entries: column | index into a shared-memory value
 * table; real matrices with few distinct values), 0 when the row-wise CSR
 * kernels are used; -1 for a null matrix. */
int blqh_debug_spmv_layout(const blqh_csr* M);

/* The product of the Lanczos recurrence: x receives the vector after the last
 * step (the start vector before the first one) and y = H x, computed as the
 * next step would, from the split input that the last step left. Host arrays
 * of dim doubles, 2 dim when complex. */
int blqh_debug_lanczos_product(blqh_lanczos* L, double* x, double* y);

/* The Gram-Schmidt dots of complex sectors: h[k] = sum_i conj(V_k[i]) w[i] for
 * nk vectors of n doubles (n even, host arrays). form: 0 = FP64, in the order
 * of the plain pass; 1, 2 = fixed-point planes in tiles of 1024 and of 256
 * doubles; 3 = fixed-point planes of the batched instances. */
int blqh_debug_dots(blqh_ctx* ctx, int64_t n, int nk, const double* V, const double* w, int form, double* h);

/* The Gram-Schmidt correction of the batched complex instances, w -= sum_k h_k V_k,
 * in the form that the coefficients' size selects there (host arrays as above). */
int blqh_debug_batch_update(blqh_ctx* ctx, int64_t n, int nk, const double* V, double* w, const double* h);

/* The n-th device allocation that the library makes for this context from now
 * on fails with BLQH_ERR_NOMEM, once (n = 0: none). Returns what was left of
 * the previous request: 0 when it has been met (or none was made). */
int blqh_debug_fail_alloc(blqh_ctx* ctx, int n);

/* Device memory that this context takes to be free when it decides on storage
 * that a call can do without (-1: what the device says). */
int blqh_debug_free_bytes(blqh_ctx* ctx, int64_t bytes);

#ifdef __cplusplus
}
#endif
#endif
