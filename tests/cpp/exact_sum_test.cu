// ExactSum (csrc/isti_device.cuh) on the host: the correctly rounded sum, so never further from the exact one
// (128-bit integers) than a running double sum, for values as SSIM and FLIP have them and for small ones.
#include "isti_device.cuh"

#include <cmath>
#include <cstdio>
#include <random>

int main()
{
    std::mt19937_64 rng(3);
    std::uniform_real_distribution<float> unit(0.5f, 1.0f);
    long further = 0;
    for (int i = 0; i < 400000; i++)
    {
        isti::ExactSum s;
        double d = 0.0;
        __int128 exact = 0; // units of 2^-64
        const int n = 1 + rng() % 32, spread = rng() % 40;
        for (int k = 0; k < n; k++)
        {
            float v = std::ldexp(unit(rng), -(int)(rng() % (spread + 1)));
            if (i % 4 != 0 && rng() % 2)
                v = -v;
            if (rng() % 20 == 0)
                v = i % 16 == 1 ? 0x1.fffffep1f : (float)(int)(rng() % 3) - 1.0f;
            s.add(v);
            d += v;
            exact += (__int128)std::ldexp((double)v, 64);
        }
        auto error = [&](double x) {
            const __int128 e = (__int128)std::ldexp(x, 64) - exact;
            return e < 0 ? -e : e;
        };
        further += error(s.value()) > error(d);
    }
    if (further)
        return printf("%ld sums further off than double\n", further), 1;
    printf("ok\n");
}
