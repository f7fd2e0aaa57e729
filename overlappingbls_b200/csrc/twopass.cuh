// twopass.cuh -- line transforms with one shared-memory exchange.
//
// A line of length N = R0*R1 is transformed in two passes: R1 butterflies of radix R0,
// one exchange through shared memory with the twiddles w_N^(r j), R0 butterflies of radix
// R1.  The spectrum is left in registers with butterfly j holding the bins j + r*R0, so a
// spectral operation and the first pass of the transform back need no exchange; the
// 3/2-rule partner of length 3N/2 keeps R0 and takes the radix 3*R1/2, whose zero third
// never reaches an instruction (DftPad, DftUnpad).  Forward, operation and backward are
// four butterfly passes and two exchanges, against four exchanges of the three-radix plans
// of fft2.cuh.
//
// What bounds the line kernels is the shared-memory/L1 data pipe, which the three-radix
// kernels kept 68-76% busy at 50% instruction issue and 21-34% of HBM (512x512x64, FP32);
// an exchange costs a store and a load of every element there.
//
// The lines of a CTA share its threads: in every pass the (butterfly, line) pairs are dealt
// to consecutive threads, so a pass with fewer butterflies than threads leaves whole warps
// idle, not lanes.  Exchange rows are padded to an odd pitch: consecutive butterflies then
// store to different banks (an even pitch would put them on the same half of the banks).
#pragma once
#include "fft2.cuh"

namespace obl {

// N = R0*R1, R1 even (the 3/2 rule's split), R0 a multiple of 4.  The splits keep the two
// radices within a factor of two, so that no pass leaves most threads without a butterfly:
// 320 as 20*16 took 43 us for the ddy of 102 levels, as 32*10 66 us, and 384 as 24*16 44 us,
// as 32*12 62 us.
template <int N> struct TwoPass;
template <> struct TwoPass<32> { static constexpr int R0 = 8, R1 = 4; };
template <> struct TwoPass<48> { static constexpr int R0 = 8, R1 = 6; };
template <> struct TwoPass<64> { static constexpr int R0 = 8, R1 = 8; };
template <> struct TwoPass<80> { static constexpr int R0 = 8, R1 = 10; };
template <> struct TwoPass<96> { static constexpr int R0 = 8, R1 = 12; };
template <> struct TwoPass<128> { static constexpr int R0 = 16, R1 = 8; };
template <> struct TwoPass<160> { static constexpr int R0 = 16, R1 = 10; };
template <> struct TwoPass<192> { static constexpr int R0 = 16, R1 = 12; };
template <> struct TwoPass<240> { static constexpr int R0 = 20, R1 = 12; };
template <> struct TwoPass<256> { static constexpr int R0 = 16, R1 = 16; };
template <> struct TwoPass<320> { static constexpr int R0 = 20, R1 = 16; };
template <> struct TwoPass<384> { static constexpr int R0 = 24, R1 = 16; };
template <> struct TwoPass<512> { static constexpr int R0 = 32, R1 = 16; };
template <> struct TwoPass<640> { static constexpr int R0 = 32, R1 = 20; };

constexpr int tp_pitch(int r) { return r | 1; }

// ----------------------------------------------------------------------------- codelets
template <bool FWD> struct Dft<20, FWD> : DftComp<4, 5, FWD> {};
template <bool FWD> struct Dft<24, FWD> : DftComp<3, 8, FWD> {};
template <bool FWD> struct Dft<32, FWD> : DftComp<4, 8, FWD> {};

// Backward DFT of length 3R/2 of R bins: bins 0..R/2-1 and R/2..R-1 of v are the first and
// the last third's, the middle third is zero.  As A = R/2 radix-3 butterflies over
// {l, l + A, l + 2A} with a zero middle input, then three A-point ones:
//   emit(q + 3p, X) for q = 0..2, p = 0..A-1.
template <int R> struct DftPad {
    static constexpr int A = R / 2, R2 = 3 * A;
    template <typename C, class F> __device__ __forceinline__ static void run(const C *v, F &&emit)
    {
        using T = decltype(v[0].x);
        const T h = (T)0.5, s3 = (T)ct::cos2pi(1, 12);   // sin(2 pi/3) = cos(2 pi/12)
        For<0, 3>::run([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            C t[A];
            For<0, A>::run([&](auto lc) {
                constexpr int l = decltype(lc)::value;
                const C a = v[l], b = v[l + A];
                C x;
                if constexpr (q == 0) {
                    x = cadd(a, b);
                } else {
                    // a + b*exp(+-2 pi i 2q/3): b*(-1/2 -+ i s3)
                    const C m = mul_mi<false>(cscale(b, s3));
                    x.x = a.x - h * b.x;
                    x.y = a.y - h * b.y;
                    x = q == 1 ? csub(x, m) : cadd(x, m);
                }
                t[l] = twc<R2, l * q, false>(x);
            });
            Dft<A, false>::run(t);
            For<0, A>::run([&](auto pc) { constexpr int p = decltype(pc)::value; emit(std::integral_constant<int, q + 3 * p>{}, t[p]); });
        });
    }
};

// Forward DFT of length 3R/2 of x, of which only bins 0..A-1 and 2A..3A-1 (A = R/2) are
// kept, in v[0..R-1]: three A-point DFTs over x[l + 3m], then radix-3 ones with two outputs.
template <int R> struct DftUnpad {
    static constexpr int A = R / 2, R2 = 3 * A;
    template <typename C> __device__ __forceinline__ static void run(const C *x, C *v)
    {
        using T = decltype(x[0].x);
        const T h = (T)0.5, s3 = (T)ct::cos2pi(1, 12);
        C y[R2];
        For<0, 3>::run([&](auto lc) {
            constexpr int l = decltype(lc)::value;
            C t[A];
            For<0, A>::run([&](auto mc) { constexpr int m = decltype(mc)::value; t[m] = x[l + 3 * m]; });
            Dft<A, true>::run(t);
            For<0, A>::run([&](auto qc) {
                constexpr int q = decltype(qc)::value;
                y[l * A + q] = twc<R2, l * q, true>(t[q]);
            });
        });
        For<0, A>::run([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            const C a = y[q], b = y[A + q], c = y[2 * A + q];
            const C s = cadd(b, c), d = cscale(csub(b, c), s3);
            v[q] = cadd(a, s);                               // bin q
            // bin q + 2A: a + b w^2 + c w^4, w = exp(-2 pi i/3): a - s/2 + i s3 (b - c)
            C t;
            t.x = a.x - h * s.x;
            t.y = a.y - h * s.y;
            v[A + q] = cadd(t, mul_mi<false>(d));
        });
    }
};

} // namespace obl
