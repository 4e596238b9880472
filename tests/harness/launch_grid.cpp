// Test harness (CPU): the blocks of a pass's kernels (launch_grid.h) stay within the launch shape's
// cap of resident warps per SM, for every kernel, and cover the work where there is no cap.
#include <cstdio>
#include "../../graphaligner_gb300/csrc/launch_grid.h"

int main()
{
    const uint64_t sms = 152;
    for (uint32_t wpb = 1; wpb <= 4; wpb++)
        for (uint32_t cap : { 0u, 1u, 2u, 5u, 1000u, 0xffffffffu })
            for (uint64_t fillWarps : { (uint64_t)1, (uint64_t)wpb })
                for (uint64_t mediumFit : { (uint64_t)0, (uint64_t)5 })
                    for (uint64_t pending : { (uint64_t)1, (uint64_t)7, (uint64_t)609, (uint64_t)100000 })
                    {
                        const ga_launch_shape sh { wpb, cap, 0, 64 };
                        const uint64_t fillFit = 20 / fillWarps, traceFit = 16 / wpb, resumeCap = std::min<uint64_t>(pending, 8192);
                        const gadev::LaunchGrid g = gadev::launch_grid(sh, sms, fillFit, fillWarps, mediumFit, traceFit, pending, resumeCap);
                        const uint64_t most = cap ? sms * wpb * cap : ~0ULL;      // warps
                        bool ok = g.fill * fillWarps <= most && g.medium <= most && g.trace * wpb <= most;
                        ok = ok && g.fill >= 1 && g.trace >= 1 && (g.medium >= 1) == (mediumFit > 0);
                        ok = ok && g.fill <= sms * fillFit && g.medium <= sms * mediumFit && g.trace <= sms * traceFit && g.medium <= resumeCap;
                        if (!cap)
                        {
                            ok = ok && (g.fill == sms * fillFit || g.fill * fillWarps >= pending) && (g.trace == sms * traceFit || g.trace * wpb >= pending);
                            ok = ok && (g.medium == sms * mediumFit || g.medium == resumeCap);
                        }
                        if (!ok)
                        {
                            printf("FAIL warps %u cap %u fill warps %llu pending %llu: %llu %llu %llu\n", wpb, cap, (unsigned long long)fillWarps,
                                (unsigned long long)pending, (unsigned long long)g.fill, (unsigned long long)g.medium, (unsigned long long)g.trace);
                            return 1;
                        }
                    }
    printf("ok\n");
    return 0;
}
