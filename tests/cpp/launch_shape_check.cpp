// Prints "grid threads chunk" of the transport's launch shape for the arguments
// photons SMs resident-CTAs ctas_per_sm threads warp_chunk, one line per six.
#include <cstdio>
#include <cstdlib>

#include "../../crysplight_b200/csrc/cl_launch.h"

int main(int argc, char** argv)
{
    for (int i = 1; i + 5 < argc; i += 6) {
        cl::LaunchSetting set;
        set.ctas_per_sm = atoi(argv[i + 3]);
        set.threads = atoi(argv[i + 4]);
        set.warp_chunk = atoi(argv[i + 5]);
        const cl::LaunchShape s = cl::launch_shape(atoll(argv[i]), atoi(argv[i + 1]), atoi(argv[i + 2]), set);
        printf("%lld %d %d\n", (long long)s.grid, s.threads, (int)s.warp_chunk);
    }
    return 0;
}
