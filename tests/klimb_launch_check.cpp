// CPU check of the K-limb passes' launches (csrc/klimb_plan.hpp) for every form
// that a residue takes between stages (K limbs, W words) and every log_n up to 24:
// the elements, threads and shared memory that the launch takes from the plan are
// within what the kernel is built for, the blocks cover the transform, and the
// swapping pass's pair of tiles exists.  Built and run by tests/test_klimb_launch.py;
// prints "ok" and exits 0 on success.
#include <cstdio>
#include <initializer_list>

#include "klimb_plan.hpp"

namespace {

int fails = 0;
void expect(bool c, const char* what, unsigned K, unsigned W, unsigned lg) {
    if (!c && fails++ < 20) std::printf("FAIL K=%u W=%u log_n=%u: %s\n", K, W, lg, what);
}

}  // namespace

int main() {
    struct Form {
        unsigned K, W;
    };
    for (Form f : {Form{2, 2}, Form{3, 3}, Form{3, 2}, Form{11, 11}, Form{11, 8}}) {
        for (unsigned lg = 1; lg <= 24; lg++) {
            const nttb::KlimbPlan P = nttb::klimb_plan(f.K, lg);
            const unsigned long n = 1ul << lg;
            auto block = [&](unsigned long elements) {
                expect(elements >= 2 && elements / 2 <= nttb::klimb_max_threads(f.K), "threads", f.K, f.W, lg);
                expect(nttb::klimb_smem_bytes(f.K, f.W, elements) <= nttb::kKlimbSmemMax, "shared memory", f.K, f.W, lg);
            };
            if (P.single_tile) {
                block(n);
                continue;
            }
            for (unsigned i = 0; i < P.n_passes; i++) {
                const nttb::KlimbPass& q = P.pass[i];
                const unsigned long elements = nttb::klimb_pass_elements(q, i == 0);
                block(elements);
                // the roots of a tile, (2^r - 1) 2^logC, are gathered two per thread
                expect(((1ul << q.r) - 1) << q.logC <= elements, "roots", f.K, f.W, lg);
                if (i == 0) {
                    expect(q.s0 == 0 && 2 * q.r <= lg, "the swapping pass's bits", f.K, f.W, lg);
                    expect(elements == 2ul << (2 * q.r), "a pair of tiles", f.K, f.W, lg);
                } else {
                    expect(n % elements == 0, "whole blocks", f.K, f.W, lg);
                }
            }
        }
    }
    if (fails) {
        std::printf("%d failures\n", fails);
        return 1;
    }
    std::printf("ok\n");
    return 0;
}
