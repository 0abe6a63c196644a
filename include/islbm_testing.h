/* islbm_testing.h - hooks for testing the step kernels: their failure path and their choice.
 *
 * No reference counterpart. The tiled step kernel waits for its shared-memory copies with
 * bounded waits (about a second); when one runs out, the kernel records the fault in the
 * solve's controller, stops starting copies, waits (bounded again) for those in flight and
 * completes, so the device context stays usable; islbm_sync then returns ISLBM_ERR_CUDA.
 * This hook makes such a wait run out without faulting anything: the copies of one plane are
 * simply never started.
 */
#ifndef ISLBM_TESTING_H
#define ISLBM_TESTING_H

#include "islbm.h"

#ifdef __cplusplus
extern "C" {
#endif

/* From the next islbm_step on, the tiled kernel skips the copies of wall-normal plane `plane`
 * (0 <= plane < NZ); -1 turns the drill off. The solve's state is undefined afterwards. */
ISLBM_API int islbm_fault_drill(islbm_handle *h, int plane);

/* The kernel that steps this solve. */
enum { ISLBM_STEP_GATHER = 0, ISLBM_STEP_CHUNK = 1, ISLBM_STEP_TILED = 2, ISLBM_STEP_PAIRED = 3, ISLBM_STEP_ROLES = 4 };
ISLBM_API int islbm_step_kernel(const islbm_handle *h, int *kernel);

/* From the next islbm_step on, a solve that steps with the role-specialised kernel steps with the
 * paired one, whose results are the same bits (runs that compare the two). */
ISLBM_API int islbm_use_paired(islbm_handle *h);

#ifdef __cplusplus
}
#endif
#endif
