// fftb_line_inst.cu -- explicit instantiations of the line kernel.
//
// Compiled several times with -DFFTB_REAL=float|double and -DFFTB_PART=k (k in [0,
// FFTB_LINE_NPARTS)) so the instantiation work spreads over parallel compiler processes; each
// object exports one table of kernels.
#include "fftb_line.cuh"

#ifndef FFTB_REAL
#define FFTB_REAL float
#endif
#ifndef FFTB_PART
#define FFTB_PART 0
#endif
#ifndef FFTB_LINE_NPARTS
#define FFTB_LINE_NPARTS 1
#endif

#define FFTB_CAT2(a, b) a##b
#define FFTB_CAT(a, b) FFTB_CAT2(a, b)
#define FFTB_CAT4(a, b, c, d) FFTB_CAT(FFTB_CAT(a, b), FFTB_CAT(c, d))

namespace {
// The complex line lengths with a kernel (R2C / C2R of even n run n/2, everything else n): every
// product of 2, 3, 5 and 7 up to 4096, and 11 and 13 times a power of two up to 832.
constexpr bool has_line(int n)
{
    int m = n;
    for (int p : {2, 3, 5, 7})
        while (m % p == 0) m /= p;
    if (m == 1) return true;
    return (m == 11 || m == 13) && (n / m & (n / m - 1)) == 0 && n <= 832;
}
constexpr int count_lines()
{
    int c = 0;
    for (int n = 1; n <= 4096; ++n) c += has_line(n);
    return c;
}
constexpr int kCount = count_lines();
struct Lengths {
    int n[kCount];
};
constexpr Lengths make_lengths()
{
    Lengths l{};
    int c = 0;
    for (int n = 1; n <= 4096; ++n)
        if (has_line(n)) l.n[c++] = n;
    return l;
}
constexpr Lengths kLengths = make_lengths();

template <int I> void fill_table(fftb::LineKernelInfo *out, int cap, int &n)
{
    if constexpr (I < kCount) {
        if (n + 1 < cap) {
            out[n] = fftb::line_kernel_info<FFTB_REAL, kLengths.n[I], true>();
            out[n + 1] = fftb::line_kernel_info<FFTB_REAL, kLengths.n[I], false>();
        }
        n += 2;
        fill_table<I + FFTB_LINE_NPARTS>(out, cap, n);
    }
}
} // namespace

extern "C" int FFTB_CAT4(fftb_line_table_, FFTB_REAL, _part, FFTB_PART)(fftb::LineKernelInfo *out, int cap)
{
    int n = 0;
    fill_table<FFTB_PART>(out, cap, n);
    return n;
}
