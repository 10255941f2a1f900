// The fixed-point circle of csrc/qsg_host.h against put_twiddle of every entry:
// the words have to be the same.  Prints one JSON line: n -> differing entries.
#include <cstdio>

#include "../../qusim_gb300/csrc/qsg_host.h"

int main()
{
    using namespace qsg_host;
    std::printf("{");
    const char *sep = "";
    for (long n : {8L, 16L, 24L, 4096L, 6000L, 131072L}) {
        const CircleLD ld(n);
        const CircleFixed fx(n);
        long diff = 0;
        for (long m = 0; m < 2 * n; ++m) {  // (the grid's products run beyond one turn)
            long double re, im;
            ld.at(m, &re, &im);
            int32_t want[4], got[4];
            put_twiddle(3, reinterpret_cast<unsigned char *>(want), re, im);
            fx.at(m, got);
            diff += std::memcmp(want, got, 16) != 0;
        }
        std::printf("%s\"%ld\": %ld", sep, n, diff);
        sep = ", ";
    }
    std::printf("}\n");
    return 0;
}
