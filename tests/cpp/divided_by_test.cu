// divided_by (csrc/isti_device.cuh) against the host's division, for every significand.
#include "isti_device.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>

template <int D>
static bool check()
{
    for (uint32_t m = 1u << 23; m < 1u << 24; m++)
        for (int e = -30; e <= -10; e += 20)
            for (int s = -1; s <= 1; s += 2)
            {
                const float x = s * std::ldexp((float)m, e);
                volatile float d = (float)D, want = x / d;
                const float got = isti::divided_by<D>(x), w = want;
                if (memcmp(&got, &w, 4) != 0)
                    return printf("%a / %d: %a, not %a\n", x, D, got, w), false;
            }
    return true;
}

int main()
{
    if (!check<116>() || !check<200>() || !check<255>() || !check<500>())
        return 1;
    printf("ok\n");
}
