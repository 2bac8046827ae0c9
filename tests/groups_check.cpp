// CPU check of csrc/fk_groups.h: over unit lengths, chunk sizes and group bounds, the
// MMA issuer's walk (chunks of each group) takes every stage once and in order, no
// chunk leaves its group or crosses a bound, and the epilogue's chunk count is the
// issuer's.
#include <cstdio>

#include "fk_groups.h"

int main() {
    for (int nst = 1; nst <= 40; ++nst)
        for (int grp = 1; grp <= 2; ++grp)
            for (int ch = 1; ch <= 4; ++ch)
                for (int bound = 0; bound <= 9; ++bound) {
                    int next = 0;
                    for (int sg0 = 0; sg0 < nst;) {
                        const int sg1 = fk::group_end(sg0, nst, grp * ch, bound);
                        int chunks = 0;
                        for (int st0 = sg0; st0 < sg1; st0 += ch, ++chunks) {
                            const int st1 = fk::chunk_end(st0, ch, sg1);
                            for (int st = st0; st < st1; ++st) {
                                if (st != next++ || st >= sg1 || (bound && st / bound != sg0 / bound)) {
                                    std::printf("FAIL nst %d grp %d ch %d bound %d stage %d\n", nst, grp, ch, bound, st);
                                    return 1;
                                }
                            }
                        }
                        if (sg1 <= sg0 || chunks > grp || chunks != fk::group_chunks(sg0, sg1, ch)) {
                            std::printf("FAIL nst %d grp %d ch %d bound %d group %d\n", nst, grp, ch, bound, sg0);
                            return 1;
                        }
                        sg0 = sg1;
                    }
                    if (next != nst) {
                        std::printf("FAIL nst %d grp %d ch %d bound %d: %d stages\n", nst, grp, ch, bound, next);
                        return 1;
                    }
                }
    std::printf("ok\n");
    return 0;
}
