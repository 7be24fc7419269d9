// Integer rules that the march's kernels share with the host, checked without
// a GPU: prints one "ok <name>" line per rule (tests/test_cpu_device_rules.py).
#include <stdio.h>
#include "radchan.h"
#include "rc_device.cuh"

using namespace rc;

static int fail(const char *what, long long at) {
    printf("bad %s at %lld\n", what, at);
    return 1;
}

// A cell's coordinate never reads as a wall, for any number of table rows;
// those below the codes are stored as they are, the others are reported.
static int coords() {
    for (int w = 0; w < 6; ++w)
        for (int t = 0; t <= 6; ++t) {
            const int code = halo_code(t, w);
            if (code < kSpecular || code > 0xffff) return fail("halo code", code);
            if (t != 1 && t != 3 && (code < kBlack || code - kBlack != w)) return fail("wall of a code", code);
        }
    if (kPeriodic >= kBlack || kSpecular >= kBlack || 255 * 256 >= kSpecular) return fail("order of the codes", 0);
    for (int q = 0; q <= 1000 * 256; ++q) {
        bool cut_c, cut_w;
        const int c = cell_coord(q, false, cut_c), wv = cell_coord(q, true, cut_w);
        if (c >= kSpecular) return fail("cell reads as a wall", q);
        if (cut_c ? q < kSpecular : c != q) return fail("cell coordinate", q);
        if (cut_w ? q <= 0xffff : wv != q) return fail("wall coordinate", q);
    }
    printf("ok coords\n");
    return 0;
}

// The cell of an emitted bundle, for every edge that params_validate accepts.
static int packing() {
    const int some[] = {0, 1, 2, 255, 256, 32766, 32767, 32768, 32769, 65534, 65535};
    for (int j = 0; j <= 65535; ++j)
        for (int i : some) {
            const unsigned a = pack_ij(i, j), b = pack_ij(j, i);
            if (unpack_i(a) != i || unpack_j(a) != j || unpack_i(b) != j || unpack_j(b) != i) return fail("packing", j);
        }
    printf("ok packing\n");
    return 0;
}

// Offsets of cells in a pyramid of almost 2^32 entries, halo included.
static int offsets() {
    const int dims[][3] = {{1289, 1289, 1289}, {65535, 16380, 2}, {2, 30000, 35000}, {1, 1, 65535}, {1023, 1023, 1023}};
    for (auto &n : dims) {
        const int im = n[0], jm = n[1], km = n[2];
        const int is[] = {0, 1, im, im + 1}, js[] = {0, 1, jm, jm + 1}, ks[] = {0, 1, km, km + 1};
        for (int i : is)
            for (int j : js)
                for (int k : ks) {
                    const long long want = i + (im + 2LL) * (j + (jm + 2LL) * k);
                    if (want > 0xffffffffLL) return fail("the grid itself", want);
                    if ((long long)cell_index(i, j, k, im, jm) != want) return fail("offset", want);
                }
    }
    printf("ok offsets\n");
    return 0;
}

int main() {
    int bad = 0;
    bad |= offsets();
    bad |= coords();
    bad |= packing();
    return bad;
}
