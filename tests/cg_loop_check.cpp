// The host loop of the conjugate gradients (cg_loop.h) with fakes in the place of the
// runtime: a refused launch, a failed wait and a state that never reports the end.
#include <cstdio>
#include <initializer_list>

#include "../openpixi_gb300/csrc/cg_loop.h"

using namespace opx;

struct Fake {
    long refuse_at = -1, fail_at = -1, done_at = -1, queued = 0, looked = 0;
    bool run(long batches) {
        return cg_batches(
            batches,
            [&](long k) {
                queued++;
                return k != refuse_at;
            },
            [&](long k) {
                looked++;
                return k == fail_at ? CG_FAILED : (k == done_at ? CG_DONE : CG_GOES_ON);
            });
    }
};

static int bad = 0;
static void need(bool ok, const char *what) {
    if (!ok) { bad++; std::printf("wrong: %s\n", what); }
}

int main() {
    Fake a;
    a.done_at = 4;
    need(a.run(100) && a.queued == 6 && a.looked == 5, "ends one batch behind the one that is done");
    for (long at : {0L, 1L, 7L}) {
        Fake b;
        b.refuse_at = at;
        need(!b.run(100) && b.queued == at + 1 && b.looked == (at > 0 ? at - 1 : 0), "a refused launch ends the loop");
        Fake c;
        c.fail_at = at;
        need(!c.run(100) && c.looked == at + 1, "a failed wait ends the loop");
    }
    for (long n : {1L, 2L, 625L}) {
        Fake d;
        need(d.run(n) && d.queued == n && d.looked == n, "a state that never reports the end");
        Fake e;
        e.done_at = n - 1;
        need(e.run(n) && e.queued == n && e.looked == n, "done with the last batch");
    }
    std::printf(bad ? "%d wrong\n" : "ok\n", bad);
    return bad != 0;
}
