// Jobs of a re-distribution that are larger than 31-bit indices reach: prints, per job on
// standard input (run, then four extents), how many pieces it is dealt out in, the cells of
// the largest, whether the pieces cover it, and the cells per unit of work.  Host code only.
#include "shuffle.cu"

#include <cstdio>

using namespace dcb;

int main()
{
    long long v[5];
    while (std::scanf("%lld %lld %lld %lld %lld", v, v + 1, v + 2, v + 3, v + 4) == 5)
    {
        ShfJob j;
        std::memset(&j, 0, sizeof(j));
        j.len = v[0], j.rows = 1;
        long long a = v[0] + 2, b = v[0]; // a halo on one side: runs do not merge
        for (int k = 0; k < 4; ++k)
        {
            j.ext[k] = v[k + 1];
            j.a_stride[k] = a, j.b_stride[k] = b;
            j.rows *= v[k + 1];
            a *= v[k + 1], b *= v[k + 1];
        }
        const long long total = j.rows * j.len;
        std::vector<ShfJob> jobs;
        long long units = 0, cells = 0, most = 0, next = 0;
        bool in_order = true;
        add_jobs(j, &jobs, &units);
        for (const ShfJob& q : jobs)
        {
            const long long n = q.rows * q.len;
            cells += n;
            most = n > most ? n : most;
            in_order = in_order && q.b_off == next; // the dense side: one piece behind the other
            next += n;
        }
        std::printf("%zu %lld %d %lld\n", jobs.size(), most, cells == total && in_order ? 1 : 0, total / units);
    }
    return 0;
}
