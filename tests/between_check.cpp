// mcg_between_nodes against the interpolation's own arithmetic (built and run
// by tests/test_between_nodes.py with -ffp-contract=off): where it says so, the
// voxel of a vertex is one of the nodes of its edge (the same one along the
// other two axes) or the one before them, and the first sample of its normal
// one of the nodes; and that this does not hold for cells and sides that it
// leaves out.  Prints what was outside.
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include "unpack.h"

static uint64_t state = 88172645463325252ull;
static uint64_t next_random() {
    state ^= state << 13;
    state ^= state >> 7;
    state ^= state << 17;
    return state;
}

// float -> int as the GPU converts: NaN to 0, otherwise to the nearest int
static int whole(float f) {
    if (f != f) return 0;
    if (f >= 2147483648.0f) return INT32_MAX;
    if (f <= -2147483648.0f) return INT32_MIN;
    return (int)f;
}

// vertices on edges along one axis of a volume of `side` voxels; how many lie elsewhere
static long outside(float cell, int side, int n) {
    long bad = 0;
    for (int k = 0; k < n; ++k) {
        const uint64_t r = next_random();
        int lo = (int)(r % (uint64_t)(side - 1));
        if (k % 4 == 0) lo = side - 2 - (int)(r % 64 % (uint64_t)(side - 1));
        if (k % 64 == 1) lo = 0;
        const bool down = (r >> 40) & 1;
        // distances of 16 bits on either side of zero
        const float f0 = mcg_unpack_tsdf(-1 - (int)((r >> 8) % (k % 3 ? 32768 : 3)));
        const float f1 = mcg_unpack_tsdf((int)((r >> 24) % (k % 5 ? 32768 : 3)));
        const float g0 = down ? f1 : f0, g1 = down ? f0 : f1;
        const float t = (0.0f - g0) / (g1 - g0 + 1e-15f);
        const int a = down ? lo + 1 : lo, b = down ? lo : lo + 1;
        const float p0 = ((float)a + 0.5f) * cell, p1 = ((float)b + 0.5f) * cell;
        const float d = p1 - p0, s = t * d, p = p0 + s, q = p / cell;
        const int vox = whole(floorf(q - 0.5f)), first = whole(q);
        const bool along = vox >= lo - 1 && vox <= lo + 1 && first >= lo && first <= lo + 1;
        // along another axis both nodes have the lower one's coordinate
        const float c = down ? p1 : p0, e = t * (c - c), o = c + e, u = o / cell;
        const int vox2 = whole(floorf(u - 0.5f)), first2 = whole(u);
        if (!along || vox2 < lo - 1 || vox2 > lo || first2 != lo) ++bad;
    }
    return bad;
}

int main() {
    long bad = 0, used = 0;
    const int sides[] = {2, 3, 34, 129, 513, 1025, 65537, 1 << 20, (1 << 21) - 1, 1 << 21};
    for (int i = 0; i < 400; ++i)
        for (const int side : sides) {
            float cell = ldexpf(1.0f + (float)(next_random() & 0x7fffff) / 8388608.0f, (int)(next_random() % 166) - 83);
            if (i == 0) cell = 1.0000001e-25f;
            if (i == 1) cell = 0.9999999e25f;
            if (i == 2) cell = ldexpf(1.0f + 8388607.0f / 8388608.0f, -7);
            if (!mcg_between_nodes(cell, side)) continue;
            ++used;
            bad += outside(cell, side, 4000);
        }
    printf("%ld cells and sides, %ld outside\n", used, bad);
    bool ok = bad == 0 && used > 3000;
    // left out, and why
    const float inf = INFINITY;
    const struct {
        float cell;
        int side;
    } rest[] = {{inf, 50}, {1e36f, 512}, {1.7e37f, 40}, {1.5e-45f, 70}, {0.0037f, 6000000}};
    for (const auto &r : rest) {
        const long n = outside(r.cell, r.side, 100000);
        printf("cell %g, side %d: %ld of 100000 outside\n", r.cell, r.side, n);
        ok = ok && n > 0 && !mcg_between_nodes(r.cell, r.side);
    }
    ok = ok && !mcg_between_nodes(NAN, 50);
    // the tile's test, also where i - org does not fit an int
    ok = ok && mcg_in_tile(32, 32, 36) && mcg_in_tile(67, 32, 36) && !mcg_in_tile(68, 32, 36) && !mcg_in_tile(31, 32, 36) &&
         !mcg_in_tile(INT32_MAX, 0, 36) && !mcg_in_tile(INT32_MIN, 0, 36) && !mcg_in_tile(INT32_MIN, 8, 36) &&
         !mcg_in_tile(-1, 0, 36) && !mcg_in_tile(0, 40, 36);
    return ok ? 0 : 1;
}
