// Prints the seed of every pair of orders a >= b >= 0 below 512 (pfsoftlib_b200/csrc/dd.cuh), as the high and low part
// of a double-double in hexadecimal.
#include <cstdio>

#include "dd.cuh"

int main()
{
    for (int a = 0; a < 512; ++a)
        for (int b = 0; b <= a; ++b) {
            const pfsoft_dev::dd s = pfsoft_dev::delta_seed(a, b);
            std::printf("%a %a\n", s.h, s.l);
        }
    return 0;
}
