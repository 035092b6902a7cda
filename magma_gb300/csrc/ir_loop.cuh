// ir_loop.cuh -- the host loop of the refinement drivers (ir.cu).  No CUDA in it, so
// that its control flow is tested on the CPU with a device of the test's own.
#pragma once

namespace mlu {

// The refinement iterations: correct(it) tests convergence and corrects, resid(it)
// forms the residual that correct(it) tests.  `look` (null: all itermax iterations run)
// lets the host see how many matrices are still being refined: look->post(it) asks for
// the number after resid(it), look->wait(&left) waits for the answer; both return
// nonzero on failure, which ends the loop with that value.  *done: the iterations
// enqueued, so the last residual is resid(*done).
//
// An iteration without work is two launches of about 2.3 us, and thirty of them were
// most of a call on a small batch (SPD refinement of 256 matrices of order 256: 1196 us,
// 876 when the loop ends).  Waiting with nothing enqueued idles the device for about
// 15 us, so the next iteration is enqueued before the host waits, and it asks after 2,
// 4, 8, 16, ... iterations only: a batch with a matrix that never converges pays for few
// questions (n = 33, one matrix of 16 not converging: 990 us without any, 1230 with a
// wait after every second iteration).
template <typename Look, typename C, typename R>
int ir_iterate(int itermax, Look *look, C correct, R resid, int *done)
{
    int asked = -3, it = 0;                    // (nothing asked yet)
    for (; it < itermax; it++) {
        if (it == asked + 2) {
            int left = 1;
            const int rc = look->wait(&left);
            if (rc != 0) return rc;
            if (left == 0) break;                // correct(asked + 1) has marked them
        }
        correct(it);
        resid(it + 1);
        if (look != nullptr && it > 0 && ((it + 1) & it) == 0 && it + 2 < itermax) {
            const int rc = look->post(it + 1);
            if (rc != 0) return rc;
            asked = it;
        }
    }
    *done = it;
    return 0;
}

}  // namespace mlu
