// Checks bsg::pass_cfg (csrc/bsg_internal.h) on the CPU: compiled and run by
// tests/test_launch_order.py.  Returns the number of shapes and pass counts
// whose first pass would be launched programmatically, or whose later passes
// are not what the shape says.
#include <cstdio>

#include "bsg_internal.h"

int main() {
    int bad = 0;
    for (int lp = 0; lp <= 8; ++lp)
        for (int pdl = 0; pdl <= 1; ++pdl)
            for (int runs : {1, 2, 3, 100}) {
                const bsg::MapCfg cfg{1, 256, 0, lp, pdl};
                for (int j = 0; j < runs; ++j) {
                    const bsg::MapCfg c = bsg::pass_cfg(cfg, j, runs);
                    if (c.pdl != (j == 0 ? 0 : pdl)) {
                        std::printf("load path %d, pdl %d: pass %d of %d has pdl %d\n", lp, pdl, j, runs, c.pdl);
                        ++bad;
                    }
                }
            }
    return bad ? 1 : 0;
}
