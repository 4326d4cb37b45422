/*
 * step_loop.cuh -- the order of a launch that takes many steps: what each
 * block of the grid does between the grid barriers, and the barrier's wait.
 * Templates on the block, so that the many-step kernel (mh2d_staged.cuh) and a
 * test that runs blocks as host threads share the order.
 */
#ifndef HYDRO_GPU_STEP_LOOP_CUH
#define HYDRO_GPU_STEP_LOOP_CUH

#ifdef __CUDACC__
#define LOOP_FN __host__ __device__ __forceinline__
#else
#define LOOP_FN inline
#endif

namespace hydro {

/* Count in on a counter that only grows and wait until it has reached
 * `target`; false when `polls` looks were not enough. */
#ifdef __CUDACC__
#pragma nv_exec_check_disable
#endif
template <class C>
LOOP_FN bool arrive_and_wait(C &c, unsigned target, int polls)
{
    if (c.arrive() + 1u == target) return true;
    while (c.count() - target > 0x7fffffffu)
        if (--polls <= 0) return false;
    return true;
}

/*
 * Up to `most` steps of one block.  begin: whether the step has a dt; faces and
 * barrier: false when a wait gave up; failed: whether the step has failed (and
 * what there is to do then); advance: the clock and the next dt, false after
 * the last step.
 *
 * Faces record errors; read_error looks at the error word between the barrier
 * behind the faces and the barrier behind the update.  Every error of the step
 * is in by then and no block can have reached the next step's faces, so all
 * blocks see the same word and leave together.  (Read behind the update's
 * barrier, it can be the error of the next step, which a faster block has
 * already begun.)
 *
 * Functions and not a class, because a class's members stay in registers for
 * the whole launch: 64^2 20.4 us a step, 256^2 50.1; as here 20.3 and 49.7.
 */
#ifdef __CUDACC__
#pragma nv_exec_check_disable
#endif
template <class Begin, class Faces, class Barrier, class ReadError, class Update, class Failed, class Advance>
LOOP_FN void step_loop(int most, Begin begin, Faces faces, Barrier barrier, ReadError read_error, Update update, Failed failed,
                       Advance advance)
{
    for (int it = 0; it < most; it++) {
        if (!begin() || !faces() || !barrier()) return;
        read_error();
        update();
        if (!barrier() || failed() || !advance()) return;
    }
}

}  // namespace hydro

#endif
