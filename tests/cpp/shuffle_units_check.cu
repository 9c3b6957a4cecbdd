// How full a re-distribution's units are: prints, per way of access and run length on standard input,
// the accesses of a job of many such runs in percent of those that its units have room for.  Host code
// only.
#include "shuffle.cu"

#include <cstdio>

using namespace dcb;

int main()
{
    long long len;
    while (std::scanf("%lld", &len) == 1)
        for (int way : {SHF_CELL, SHF_VEC, SHF_PIECE})
        {
            ShfJob j;
            std::memset(&j, 0, sizeof(j));
            j.len = len, j.rows = 1;
            for (int k = 0; k < 4; ++k)
                j.ext[k] = k == 0 ? 100000 : 1;
            j.a_stride[0] = j.b_stride[0] = len + (len % 4 == 0 ? 4 : 1);
            finish_job(&j);
            if (shf_way(j.vec, j.len, way == SHF_VEC) != way && way != SHF_CELL)
                continue;
            const double chunk = SHF_THREADS * (way == SHF_PIECE ? shf_unroll<SHF_PIECE> : shf_unroll<SHF_VEC>);
            std::printf("%lld %d %d\n", len, way, (int) (100.0 * (double) j.rows * (double) j.per_run[way] / ((double) j.units[way] * chunk)));
        }
    return 0;
}
