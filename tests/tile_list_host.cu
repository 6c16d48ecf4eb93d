// Host checks of the pair kernel's tile list on its own rules (mfree_kernels.cuh);
// prints "ok", or what failed.  Needs no GPU.
#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>

#include "mfree_kernels.cuh"

using namespace mfree;

// the tiles of one bundle, cut as the kernel cuts them: in runs, where empty
// levels are skipped, and a tile is as deep as the rule allows
static long long cut(const Params &P, const std::vector<int> &level) {
    const int nz = P.gnz;
    std::vector<int> below(nz + 1, 0);
    for (int z = 0; z < nz; z++) below[z + 1] = below[z] + level[z];
    auto upto = [&](int z) { return below[z < 0 ? 0 : z > nz ? nz : z]; };
    long long tiles = 0;
    for (int z0 = 0; z0 < nz;) {
        if (level[z0] == 0) {
            z0++;
            continue;
        }
        int d = 1;
        const int z_end = std::min((z0 / TILE_RUN + 1) * TILE_RUN, nz);
        while (!tile_too_deep(P, z0, z_end, d + 1, upto(z0 + d + 1) - upto(z0), upto(z0 + d + 3) - upto(z0 - 2))) d++;
        tiles++;
        z0 += d;
    }
    return tiles;
}

// max_tiles against the tiles of bundles of lo to hi particles a level
static int check_bound() {
    std::mt19937 rng(1);
    const int ranges[][2] = {{0, 1}, {0, 4}, {20, 40}, {60, 110}, {69, 75}, {90, 105}, {100, 500}};
    for (auto &r : ranges)
        for (int nz : {1, 2, 9, 33, 100, 257})
            for (int tile_z : {1, 5, TILE_Z_MAX})
                for (int cap : {32, 120, 205, 240}) {
                    Params P{};
                    P.gnx = 3 * TX - 1, P.gny = 2 * TY, P.gnz = nz;
                    P.tile_z = tile_z, P.tile_cap = cap;
                    long long tiles = 0, n = 0;
                    for (int b = 0; b < num_bundles(P); b++) {
                        std::vector<int> level(nz);
                        for (int &l : level) n += l = std::uniform_int_distribution<int>(r[0], r[1])(rng);
                        tiles += cut(P, level);
                    }
                    P.n_init = int(n);
                    if (tiles > max_tiles(P)) {
                        printf("%lld tiles, bound %lld: levels of %d to %d, nz %d, tile_z %d, tile_cap %d\n", tiles,
                               max_tiles(P), r[0], r[1], nz, tile_z, cap);
                        return 1;
                    }
                }
    return 0;
}

// bundle_below with cell starts whose sum over a bundle's columns passes 2^31
static int check_count() {
    Params P{};
    P.gnx = 2 * TX + 1, P.gny = TY + 2, P.gnz = 40;
    std::vector<int> first(size_t(P.gnx) * P.gny * P.gnz + 1);
    for (long long start : {0ll, 134217700ll, 2147000000ll}) {  // cell 0 begins there; 3 particles a cell
        for (size_t c = 0; c < first.size(); c++) first[c] = int(start + 3 * (long long)c);
        for (int b = 0; b < num_bundles(P); b++) {
            const TileGeo G = tile_geo(P, b * P.gnz, 1);
            const int cx = P.gnx - G.X0 < TX ? P.gnx - G.X0 : TX, cy = P.gny - G.Y0 < TY ? P.gny - G.Y0 : TY;
            for (int z0 = 0; z0 <= P.gnz; z0 += 5)
                for (int z = z0; z <= P.gnz; z++) {
                    const int n = int(bundle_below(P.gnx, P.gny, P.gnz, first.data(), G, z) - bundle_below(P.gnx, P.gny, P.gnz, first.data(), G, z0));
                    if (n != 3 * cx * cy * (z - z0)) {
                        printf("bundle %d, levels %d to %d from %lld: %d\n", b, z0, z, start, n);
                        return 1;
                    }
                }
        }
    }
    return 0;
}

int main() {
    if (check_bound() || check_count()) return 1;
    printf("ok\n");
    return 0;
}
