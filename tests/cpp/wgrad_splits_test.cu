// The weight gradient's work split (wgrad_config): every unit in exactly one split and no split without
// units, over the network's layers at many sizes and batches and over random shapes.
#include "isti_unet_conv.cuh"

#include <cstdio>
#include <random>

static bool check(int taps, int n, int h, int w, int cin, int cout)
{
    isti_unet::WgradConfig c;
    if (!isti_unet::wgrad_config(taps, n, h, w, cin, cout, c))
        return printf("%d taps, %d x %d x %d, %d -> %d: refused\n", taps, n, h, w, cin, cout), false;
    const bool ok = c.splits >= 1 && c.units_per_split >= 1 && (long long)(c.splits - 1) * c.units_per_split < c.n_units &&
                    (long long)c.splits * c.units_per_split >= c.n_units && c.splits * c.grid_y * c.grid_z <= 152;
    if (!ok)
        printf("%d taps, %d x %d x %d, %d -> %d: %d units in %d splits of %d\n", taps, n, h, w, cin, cout, c.n_units, c.splits, c.units_per_split);
    return ok;
}

int main()
{
    // taps, cin, cout and the level (image halved that often) of the network's layers
    const int layers[][4] = {{9, 16, 32, 0}, {9, 32, 64, 1}, {9, 64, 96, 2}, {9, 96, 128, 3}, {1, 128, 96, 3},
                             {9, 96, 96, 2}, {1, 96, 64, 2}, {9, 64, 64, 1}, {1, 64, 32, 1}, {9, 32, 32, 0}};
    long bad = 0;
    for (int n = 1; n <= 9; n++)
        for (int h = 8; h <= 560; h += 24)
            for (int w = 16; w <= 560; w += 8)
                for (const int(&l)[4] : layers)
                    bad += !check(l[0], n, h >> l[3], w >> l[3], l[1], l[2]);
    std::mt19937 rng(7);
    for (int i = 0; i < 200000; i++)
        bad += !check(rng() % 2 ? 9 : 1, 1 + rng() % 8, 1 + rng() % 600, 1 + rng() % 600, 16 * (1 + rng() % 16), 16 * (1 + rng() % 8));
    if (bad)
        return printf("%ld shapes\n", bad), 1;
    printf("ok\n");
}
