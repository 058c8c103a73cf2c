// Host entry points over polysplat_gb300/csrc/tile_test.h, built by
// tests/test_tile_candidates.py.
#include "../polysplat_gb300/csrc/tile_test.h"

using namespace gsr;

// For n Gaussians (centre 2, conic 3, power): tiles of [x0, x1) x [y0, y1) that
// pass the test (hits), those of them outside the row candidates (lost), and
// the candidates, with the kind of band.
extern "C" void tile_candidates(int n, const float* ctr, const float* con, const float* power, int bx, int by, int x0,
                                int x1, int y0, int y1, int* kind, long long* hits, long long* lost, long long* cand)
{
    for (int i = 0; i < n; i++) {
        const float2 c = {ctr[2 * i], ctr[2 * i + 1]};
        const float3 q = {con[3 * i], con[3 * i + 1], con[3 * i + 2]};
        const Band b = make_band(q, power[i], c, x0, x1, bx);
        kind[i] = b.kind;
        hits[i] = lost[i] = cand[i] = 0;
        for (int y = y0; y < y1; y++) {
            int lo = x0, hi = x1 - 1;
            if (b.kind != kBandFull && !band_columns(b, y, by, bx, x0, x1, lo, hi)) lo = 1, hi = 0;
            cand[i] += hi >= lo ? hi - lo + 1 : 0;
            for (int x = x0; x < x1; x++)
                if (tile_hit(x, y, bx, by, c, q, power[i])) {
                    hits[i]++;
                    if (x < lo || x > hi) lost[i]++;
                }
        }
    }
}
