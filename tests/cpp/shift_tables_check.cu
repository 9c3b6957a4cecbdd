// Layouts of the shift kernel whose issuers' tables have to fit fewer bytes.  Per geometry and limit
// on standard input,
//   n c k d h w f stride limit   (d = 0: 2-D; padding (f - 1) / 2, dense tensors, fp32)
// prints per pass: laid out, bytes of the tables, streamed, rows of a column, longest chain, cost.
// Host code only; links against the library.
#define main planner_main
#include "conv_planner_check.cu"
#undef main

int main()
{
    int v[9];
    while (std::scanf("%d %d %d %d %d %d %d %d %d", v, v + 1, v + 2, v + 3, v + 4, v + 5, v + 6, v + 7, v + 8) == 9)
    {
        const ConvGeom g = geom(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]);
        for (int tr = 0; tr < 2; ++tr)
        {
            ShTables t;
            const bool ok = ShBuilder(g, tr == 1, DCB_MATH_FP32, 148, v[8]).build(&t);
            if (ok)
                std::printf("1 %zu %d %d %d %.0f\n", t.issue.size(), t.g.stream, t.g.th, t.chain, t.cost);
            else
                std::printf("0 0 0 0 0 0\n");
        }
    }
    return 0;
}
