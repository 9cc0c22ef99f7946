// The order of launches of a run of steps, apart from what is launched.
#pragma once

namespace lbgb {

// nsteps steps by launches of next(left) steps each: launch(n, done) advances n
// steps after `done`, 0 on success.  *done: the steps launched.
template <class Next, class Launch>
int run_steps(int nsteps, Next next, Launch launch, int *done) {
    *done = 0;
    while (*done < nsteps) {
        const int n = next(nsteps - *done), rc = launch(n, *done);
        if (rc) return rc;
        *done += n;
    }
    return 0;
}

// And moves a device counter by the steps launched, bump(steps), also where a
// launch in the middle fails: their random numbers are not drawn again.
template <class Next, class Launch, class Bump>
int run_counted_steps(int nsteps, Next next, Launch launch, Bump bump) {
    int done = 0;
    const int rc = run_steps(nsteps, next, launch, &done), rb = done > 0 ? bump(done) : 0;
    return rc ? rc : rb;
}

}  // namespace lbgb
