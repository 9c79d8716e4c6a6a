/*
 * rbrp_gb300_testing.h - diagnostic entry points of the GB300 RBRP library.
 *
 * Not part of the reference's interface (no counterpart in gpu/rbrp.hpp or
 * gpu/rid.hpp): they let tests and benchmarks select between the kernel
 * variants that compute the same quantity, so each can be checked against
 * the other and against the CPU oracle, and shorten the limit of the bounded
 * device-side waits so that the timeout path can be tested.
 */
#ifndef RBRP_GB300_TESTING_H
#define RBRP_GB300_TESTING_H

#include "rbrp_gb300.h"

#ifdef __cplusplus
extern "C" {
#endif

/* Projection and update kernels: 0 = tensor cores (default), 1 = CUDA cores.  FP32
 * residual form: tcgen05 / TMEM / TMA 3xTF32 or FFMA, both to ~1e-8 relative.
 * FP64 form: BF16 slices (b > 8) or the fixed-point copy (b <= 8), or the FP64 pipe. */
rbrp_status rbrp_set_variant(rbrp_handle h, int variant);

/* T = R11^{-1} R12: 0 = exact BF16 slice products on the tensor cores, or the FP64 pipe
 * for small ranks (default; FP64-accurate), 1 = FP64 pipe throughout. */
rbrp_status rbrp_set_tsolve_fp64(rbrp_handle h, int on);

/* Limit, in SM clock cycles, of the bounded device-side waits of kernels launched
 * through this handle: the grid barrier of the LU pivots (rbrp_lupp_pivots_f64)
 * and the mbarrier waits of the tcgen05 kernels (projection, update, the slice
 * products of the FP64 form and of the T solve, the adjoint's and the sketch's
 * GEMMs).  0 restores the default
 * (~2 s).  A limit of a few cycles makes a wait run out: the kernel then exits
 * cleanly and the call returns RBRP_ERR_DEVICE_TIMEOUT, which is how the tests
 * exercise that path without faulting or hanging a GPU.  The waits that let an
 * aborting kernel's own copies and MMAs finish keep the default limit. */
rbrp_status rbrp_set_wait_budget(rbrp_handle h, long long cycles);

/* Device memory, in bytes, that the handle's allocations find free from now on (0: what
 * there is): an allocation of more fails as it would on a full device, without filling one.
 * Memory that the handle already holds and could release counts against it. */
rbrp_status rbrp_set_memory_limit(rbrp_handle h, size_t bytes);

/* Device memory, in bytes, that the handle holds for the slices or the fixed-point copy of the
 * last FP64 matrix: scratch that any of its allocations that finds no room gives back. */
rbrp_status rbrp_scratch_bytes(rbrp_handle h, size_t* bytes);

/* The arithmetic of the last successful single-matrix run, as a sum of RBRP_FORM_*: results are
 * reproducible bit for bit within one form.  Which of them a run takes follows from its
 * parameters and sizes and, for the first three, from whether their scratch fits into half of
 * the free device memory. */
enum {
  RBRP_FORM_SLICES = 1,        /* FP64 projection as BF16 slices on the tensor cores */
  RBRP_FORM_SLICED_CGS = 2,    /* with room for the basis: Gram-Schmidt products too, where large */
  RBRP_FORM_FIXED_POINT = 4,   /* FP64 projection of b <= 8 from a fixed-point copy of A */
  RBRP_FORM_FIXED_ORDER = 8,   /* FP64: every sum in one order whatever the launch */
  RBRP_FORM_T_FP64 = 16        /* T by substitution on the FP64 pipe */
};
rbrp_status rbrp_last_form(rbrp_handle h, int* form);

#ifdef __cplusplus
}
#endif
#endif /* RBRP_GB300_TESTING_H */
