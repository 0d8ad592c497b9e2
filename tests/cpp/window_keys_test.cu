// The windows' key selection as minima (window_keys) against the reference's scan (src/renderer.cu:148-175)
// on host: random tiles with ties, +-0, +-inf, NaN, empty and border keys, both centre offsets.
#include "isti_kernels.cuh"

#include <cstdio>
#include <cstring>
#include <random>

template <int SW>
long check(std::mt19937_64 &rng, long tiles)
{
    using T = isti::Tile<SW>;
    unsigned long long tile[T::ELEMS];
    const uint32_t special[] = {0u, 0x80000000u, 0x7f800000u, 0xff800000u, 0x7fc00000u, 0xffc00000u, 0xfefefefeu, 1u, 0x7f7fffffu, 0xbf000000u};
    long bad = 0;
    for (long i = 0; i < tiles; i++)
    {
        const unsigned mix = (unsigned)(rng() % 5); // how often special, how many ties
        for (unsigned long long &k : tile)
        {
            uint32_t hi = 0x3f000000u + (uint32_t)(rng() % (mix == 0 ? 3 : 4000));
            if (mix && rng() % (mix == 4 ? 2 : 12) == 0)
                hi = special[rng() % (sizeof special / sizeof special[0])];
            k = (unsigned long long)hi << 32 | (uint32_t)rng();
        }
        const int col = SW + (int)(rng() % (T::W - 2 * SW));
        for (int below = 0; below < 2; below++)
        {
            const bool wanted[isti::ROWS] = {true, true};
            isti::KeyWords got[isti::ROWS];
            isti::window_keys<SW>(tile, col, below, wanted, got);
            for (int r = 0; r < isti::ROWS; r++)
            {
                const unsigned long long want = isti::window_key_in_order<SW>(tile, SW + (r == 0 ? 0 : below), col);
                bad += ((unsigned long long)got[r].hi << 32 | got[r].lo) != want;
            }
        }
    }
    return bad;
}

int main()
{
    std::mt19937_64 rng(11);
    const long n = 200000, bad = check<1>(rng, n) + check<3>(rng, n);
    if (bad)
    {
        std::printf("%ld windows differ\n", bad);
        return 1;
    }
    std::printf("ok %ld windows\n", 8 * n);
    return 0;
}
