// Pieces of four of a run that is not aligned: prints how many (run length, start) pairs have every
// cell in one piece, none outside the run, and enough pieces counted.  Host code only.
#include "shuffle.cu"

#include <cstdio>

using namespace dcb;

int main()
{
    int good = 0, pairs = 0;
    for (long long len = SHF_PIECE_MIN; len < 4200; len += len < 80 ? 1 : 37)
        for (int head = 0; head < 4; ++head, ++pairs)
        {
            ShfJob j;
            std::memset(&j, 0, sizeof(j));
            j.len = len, j.rows = 1;
            for (int k = 0; k < 4; ++k)
                j.ext[k] = 1;
            finish_job(&j);
            std::vector<int> seen((size_t) len, 0);
            bool ok = true;
            for (long long q = 0; q < j.per_run[SHF_PIECE]; ++q)
            {
                const ShfRange r = shf_range(head, q, len);
                ok = ok && (head + r.e) % 4 == 0;
                for (int i = r.lo; i < r.hi; ++i)
                    if (r.e + i < 0 || r.e + i >= len || seen[(size_t) (r.e + i)]++)
                        ok = false;
            }
            for (int n : seen)
                ok = ok && n == 1;
            good += ok;
        }
    std::printf("%d %d\n", good, pairs);
    return 0;
}
