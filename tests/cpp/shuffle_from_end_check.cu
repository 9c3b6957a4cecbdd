// Which windows are unpacked from their end: prints 1 or 0 per window size in MB (of 1e6 bytes, all
// ranks of a device together) on standard input, for an L2 of 126 MiB.  Host code only.
#include "shuffle.cu"

#include <cstdio>

using namespace dcb;

int main()
{
    double mb;
    while (std::scanf("%lf", &mb) == 1)
        std::printf("%d\n", shf_from_the_end(mb * 1e6, 126.0 * 1048576.0) ? 1 : 0);
    return 0;
}
