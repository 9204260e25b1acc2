// Test harness: the shares of lpm-cpp_b200/csrc/shares.cuh on the host.  For every number of slices up to
// argv[1] and a cluster of at most argv[2] CTAs, prints one line: slices, CTAs, then the CTAs + 1 bounds.
#include <cstdio>
#include <cstdlib>

#include "shares.cuh"

int main(int argc, char **argv)
{
    if (argc != 3)
        return 2;
    for (int n = 1; n <= std::atoi(argv[1]); ++n)
    {
        const int nc = lpm::share_ctas(n, std::atoi(argv[2]));
        std::printf("%d %d %d", n, nc, lpm::share_most(n, nc));
        for (int k = 0; k <= nc; ++k)
            std::printf(" %d", lpm::share_begin(n, nc, k));
        std::printf("\n");
    }
    return 0;
}
