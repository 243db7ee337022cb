// nudged() on the host: every cell of a surface against the rule in 64 bits, and the cells that a
// surface without a maximum hands in (INT_MAX over the surface's width): the corner lies inside the
// window whatever the geometry.
#include <climits>
#include <cstdio>

#include "kernels.cuh"

using namespace ampcor_b200;

int main()
{
    int bad = 0;
    for (int R : {1, 16, 64})
        for (int M : {0, 1, 2, 8, 31})
            for (int m = 0; m <= M; ++m) {
                const int W = R + 2 * M, C = W - R + 1, E = R + 2 * m;
                auto check = [&](int u, int v) {
                    auto corner = [&](long long x) {
                        long long c = x - m;
                        if (c < 0) c = 0;
                        if (c + E > W) c = W - E;
                        return c;
                    };
                    const CoarseOut o = nudged(u, v, R, W, m);
                    if (o.u != u || o.v != v || o.top != corner(u) || o.left != corner(v)) {
                        if (bad++ < 5) printf("R %d M %d m %d cell %d %d: %d %d\n", R, M, m, u, v, o.top, o.left);
                    }
                };
                for (int u = -1; u < C; ++u)
                    for (int v = -1; v < C; ++v) check(u, v);
                check(INT_MAX / C, INT_MAX % C);
                check(INT_MAX, INT_MAX);
            }
    printf("%d wrong\n", bad);
    return bad != 0;
}
