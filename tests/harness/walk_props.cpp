// Checks the traceback's step bits (diagonal_rows, up_run) against the scores of columns made
// by myers_step: every cell below row 0 and right of column 0 of random node-slices.
#include <cstdio>
#include <cstdlib>
#include <random>
#include "../../graphaligner_gb300/csrc/wordslice.cuh"
using namespace gadev;

int main()
{
    std::mt19937_64 rng(12345);
    for (int round = 0; round < 3000; round++)
    {
        const int columns = 2 + (int)(rng() % 63);
        u64 eqs[4] = {0, 0, 0, 0};
        for (int r = 0; r < 64; r++) eqs[rng() % 4] |= 1ULL << r;
        WS ws = round % 3 == 0 ? ws_source((i32)(rng() % 1000)) : ws_make(0, 0, 0);
        if (round % 3)
        {
            const u64 a = rng(), b = rng();
            ws.VP = a & (round % 3 == 1 ? b : kAllOnes);
            ws.VN = ~a & rng();
            ws.end = (i32)(rng() % 1000);
        }
        const bool forced = round % 5 == 0;
        if (forced) { ws.VP &= ~1ULL; ws.VN |= 1; }
        WS prev = ws;
        for (int c = 1; c < columns; c++)
        {
            const u64 eq = eqs[rng() % 4] & (forced ? ~1ULL : kAllOnes);
            const u32 h = forced ? 1 : (u32)(rng() % 3);
            u64 Ph, Mh, Xh;
            WS nw = myers_step(eq, prev, h == 1, h == 2, Ph, Mh, Xh);
            const u64 diagonal = diagonal_rows(eq, Xh, prev.VN);
            if (forced && ((nw.VP & 1) || !(nw.VN & 1))) { printf("forced first row: column %d\n", c); return 1; }
            for (int r = 1; r < 64; r++)
            {
                const i32 here = ws_value(nw, r), corner = ws_value(prev, r - 1);
                const bool match = (eq >> r) & 1;
                const bool want = corner == here - (match ? 0 : 1);
                if (want != (bool)((diagonal >> r) & 1)) { printf("diagonal: column %d row %d\n", c, r); return 1; }
                if (ws_value(nw, r - 1) != here - 1 && !want && ws_value(prev, r) != here - 1) { printf("no step: column %d row %d\n", c, r); return 1; }
                u32 run = 0;
                int at = r;
                while (at > 0 && ws_value(nw, at - 1) == ws_value(nw, at) - 1) { at--; run++; }
                const u32 got = (nw.VP >> r) & 1 ? up_run(nw.VP, (u32)r) : 0;
                if (run != got) { printf("run up: column %d row %d: %u, not %u\n", c, r, got, run); return 1; }
            }
            prev = nw;
        }
    }
    printf("ok\n");
    return 0;
}
