// lines.cuh -- batched 1D spectral line operations along x (rows) and y (columns).
//
// These kernels are the building blocks of every hot-path routine:
//   rows    (x direction, contiguous):  ddx, x-pad, x-unpad, x r2c, x c2r
//   columns (y direction, strided):     ddy, y-pad, y-unpad, y c2c forward/backward
// Real lines are transformed two at a time as one complex line (z = a + i b): every
// spectral operation used here is a real-to-real linear map acting on Z[k] and Z[N-k]
// symmetrically (i*k multipliers with signed k, truncation / zero extension), so
// Re(IFFT(op(FFT(z)))) = op(a) and Im(...) = op(b), exactly what the reference's
// per-line r2c -> op -> c2r computes (004_derivatives.f90:33-39,
// 108_01_padd.f90:102-127,163-190).
//
// Rows and columns are loaded from global memory straight into registers in the layout of
// the first FFT pass and exchanged through shared memory; a column CTA's WB adjacent lines
// make its accesses row segments (the on-GPU replacement of the reference's mpi_alltoall
// pencil transposes, 203_fftn_mpi.f90:71-371).
//
// Accuracy: before a real line is transformed, its first value is subtracted (exact
// by Sterbenz's lemma for fields with a large mean such as theta ~ 300 K) and the
// scale is applied after the subtraction; derivatives ignore the constant, padding
// adds it back.  FP32 FFT errors then scale with the fluctuations, not with the mean.
#pragma once
#include <cuda.h>   // CUtensorMap and its enums (the encoder is reached through the runtime)
#include <cstdint>
#include <vector>

#include "async.cuh"
#include "twopass.cuh"

namespace obl {

// (OP_FILT: forward and backward on complex columns, the Nyquist bin dropped between)
enum LineOp : int { OP_DERIV = 0, OP_PAD = 1, OP_UNPAD = 2, OP_FWD = 3, OP_INV = 4, OP_FILT = 5 };
// twiddle tables of a length: the three-radix plans of fft2.cuh, and (+ ROLE_TP) the
// two-pass ones of twopass.cuh
enum PlanRole : int { ROLE_FWD = 0, ROLE_BWD = 1, ROLE_PADFWD = 2, ROLE_PADBWD = 3, ROLE_TP = 4 };

template <typename T> struct RowArgs {
    const void *src;          // real rows (DERIV/PAD/UNPAD/FWD) or complex rows (INV)
    void *dst;                // real rows (DERIV/PAD/UNPAD/INV) or complex rows (FWD)
    long long src_stride;     // elements (of the row's type) between consecutive rows
    long long dst_stride;
    long long npairs;         // number of row pairs (rows 2p, 2p+1)
    T scale;                  // multiplies the input at load
    const double *ktab;       // DERIV: k[0..N/2] (the Nyquist entry is 0)
    const C2<T> *twF, *twB;   // plan twiddle tables of the forward / backward transforms
    T pad_scale;              // INV with pad_mode: dst pad columns *= pad_scale
    int pad_mode;
};

template <typename T> struct ColArgs {
    const void *src;
    void *dst;
    long long src_row, dst_row;      // elements between rows
    long long src_plane, dst_plane;  // elements between planes
    int ncols;                       // real columns (real ops) / complex columns
    int nlev;
    T scale;                         // multiplies the input at load
    const double *ktab;              // DERIV: k[0..N/2]
    const C2<T> *twF, *twB;
    int pad_copy;                    // UNPAD: also write columns 0,1 into ncols, ncols+1
    int zero_nyq;                    // FWD: zero the Nyquist row (203_fftn_mpi.f90:33)
    int tma;                         // FP32 y-pad: input tile by tensor-map copies (k_tp_cols_tma)
    int pf_ahead;                    // those also ask L2 for the tile of plane z + pf_ahead (0 = none)
    int *wait_err;                   // set to 1 when such a copy's bounded wait gave up
};

// ----------------------------------------------------------------------------- configuration
template <int N, int OP> struct LineCfg;
template <int N> struct LineCfg<N, OP_DERIV> {
    static constexpr int NI = N, NO = N;
    using PF = FwdPlan<N>;
    using PB = BwdPlan<N>;
};
template <int N> struct LineCfg<N, OP_PAD> {
    static constexpr int NI = N, NO = 3 * N / 2;
    using PF = FwdPlan<N>;
    using PB = PadBwdPlan<N>;
};
template <int N> struct LineCfg<N, OP_FWD> : LineCfg<N, OP_DERIV> {};
template <int N> struct LineCfg<N, OP_INV> : LineCfg<N, OP_DERIV> {};

template <int N, int OP> struct LineDerived {
    using Cfg = LineCfg<N, OP>;
    static constexpr int NI = Cfg::NI, NO = Cfg::NO;
    using PF = typename Cfg::PF;
    using PB = typename Cfg::PB;
    static constexpr int llf = LL_<NI, PF>::v, llb = LL_<NO, PB>::v;
    static constexpr int LL = llf < llb ? llf : llb;
    static constexpr int LPW = 32 / LL;
    static constexpr int rf = Regs<NI, LL, PF>::v, rb = Regs<NO, LL, PB>::v;
    static constexpr int VR = rf > rb ? rf : rb;
    static constexpr int NM = NI > NO ? NI : NO;
    static constexpr int TF = tw_size<NI, PF>(), TB = tw_size<NO, PB>();
    static constexpr int RFL = PlanInfo<PF>::last, RB0 = PlanInfo<PB>::first;
    static constexpr int RF0 = PlanInfo<PF>::first, RBL = PlanInfo<PB>::last;
};

// ----------------------------------------------------------------------------- register ops
// v in D(R) of length N: v *= i*k_signed (ktab[N/2] = 0 drops the Nyquist mode)
template <typename T, int N, int R, int LL>
__device__ __forceinline__ void reg_deriv(C2<T> *v, const double *ktab, int t)
{
    using G = Geo<N, R, LL>;
#pragma unroll
    for (int b = 0; b < G::PER; ++b) {
        const int j = t + LL * b;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int k = j + r * G::NB;
            const int kc = (G::FULL || j < G::NB) ? k : 0;
            const T kk = (kc <= N / 2) ? (T)ktab[kc] : -(T)ktab[N - kc];
            const C2<T> z = v[b * R + r];
            v[b * R + r] = mk<T>(-kk * z.y, kk * z.x);
        }
    }
}

// D(R) of length N  ->  D(3R/2) of length 3N/2, zero-extended, Nyquist bin dropped
template <typename T, int N, int R, int LL>
__device__ __forceinline__ void reg_pad(const C2<T> *v, C2<T> *w, int t)
{
    using G = Geo<N, R, LL>;
    constexpr int R2 = 3 * R / 2, H = R / 2;
#pragma unroll
    for (int b = 0; b < G::PER; ++b) {
        const int j = t + LL * b;
#pragma unroll
        for (int r2 = 0; r2 < R2; ++r2) {
            C2<T> x = mk<T>(0, 0);
            if (r2 < H) x = v[b * R + r2];
            else if (r2 >= R) x = v[b * R + (r2 - H)];
            if (r2 == R && j == 0) x = mk<T>(0, 0);   // source bin N/2 (Nyquist)
            w[b * R2 + r2] = x;
        }
    }
}

// ----------------------------------------------------------------------------- column kernel
template <typename T, bool REAL, int LPW> struct ColTile {
    static constexpr int LINES = 8 * LPW;                  // lines per CTA (8 warps)
    static constexpr int W = REAL ? 2 * LINES : LINES;     // tile columns (elements)
    static constexpr int S = W + 1;                        // odd row stride
};

// The whole CTA processes column tile tx of plane z: coalesced tile load, one line per
// LL lanes through forward -> op -> backward in registers (the tile column is the
// exchange scratch), coalesced store.  Contains __syncthreads(): call uniformly.
template <typename T, int N, int OP, bool REAL>
__device__ __forceinline__ void col_unit(const ColArgs<T> &a, int z, int tx, const C2<T> *twF,
                                         const C2<T> *twB,
                                         typename std::conditional<REAL, T, C2<T>>::type *tile)
{
    using C = C2<T>;
    using E = typename std::conditional<REAL, T, C>::type;
    using D = LineDerived<N, OP>;
    constexpr int NI = D::NI, NO = D::NO, LL = D::LL, LPW = D::LPW, VR = D::VR;
    using TT = ColTile<T, REAL, LPW>;
    constexpr int W = TT::W, S = TT::S;

    const int c0 = tx * W;
    const int nc = min(W, a.ncols - c0);
    const E *src = reinterpret_cast<const E *>(a.src) + (long long)z * a.src_plane + c0;
    E *dst = reinterpret_cast<E *>(a.dst) + (long long)z * a.dst_plane + c0;

    // Tile load: 256 threads, UNR independent L2-only loads (ld.global.cg) in flight per
    // thread before the shared-memory stores, so the loop is not latency-serialised.
    // L2-only loads are also what the cluster-fused kernels need for data other CTAs wrote.
    {
        constexpr int TOT = NI * W, PERT = (TOT + 255) / 256, UNR = PERT < 8 ? PERT : 8;
#pragma unroll 1
        for (int b0 = 0; b0 < PERT; b0 += UNR) {
            E buf[UNR];
#pragma unroll
            for (int u = 0; u < UNR; ++u) {
                const int idx = threadIdx.x + 256 * (b0 + u);
                const int r = idx / W, c = idx - r * W;
                E v;
                if constexpr (REAL) v = (T)0;
                else v = mk<T>(0, 0);
                if (idx < TOT && c < nc) v = __ldcg(src + (long long)r * a.src_row + c);
                buf[u] = v;
            }
#pragma unroll
            for (int u = 0; u < UNR; ++u) {
                const int idx = threadIdx.x + 256 * (b0 + u);
                const int r = idx / W, c = idx - r * W;
                if (idx < TOT) tile[sidx(r) * S + c] = buf[u];
            }
        }
    }
    __syncthreads();

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane / LL, t = lane % LL;
    const int l = warp * LPW + g;
    const int c = REAL ? 2 * l : l;
    const bool act = c < nc;
    const int cc = act ? c : 0;
    C v[VR];
    T cr = 0, ci = 0;

    static_assert(OP == OP_DERIV || OP == OP_PAD || OP == OP_FWD, "the passes of the cluster-fused kernel");
    auto body = [&](auto &acc) {
        {
            using G = Geo<NI, D::RF0, LL>;
            if constexpr (REAL) {
                const C c0v = acc.ld(0);
                cr = c0v.x;
                ci = c0v.y;
            }
#pragma unroll
            for (int b = 0; b < G::PER; ++b) {
                const int j = t + LL * b;
#pragma unroll
                for (int r = 0; r < D::RF0; ++r) {
                    C x = mk<T>(0, 0);
                    if (G::FULL || j < G::NB) {
                        x = acc.ld(j + r * G::NB);
                        x.x = (x.x - cr) * a.scale;
                        x.y = (x.y - ci) * a.scale;
                    }
                    v[b * D::RF0 + r] = x;
                }
            }
            __syncwarp();
            fft_regs<NI, typename D::PF, LL, true>(v, acc, twF, t);
        }
        if constexpr (OP == OP_FWD) {
            using G = Geo<NI, D::RFL, LL>;
#pragma unroll
            for (int b = 0; b < G::PER; ++b) {
                const int j = t + LL * b;
                if (G::FULL || j < G::NB)
#pragma unroll
                    for (int r = 0; r < D::RFL; ++r) {
                        const int i = j + r * G::NB;
                        C x = v[b * D::RFL + r];
                        if (a.zero_nyq && i == NI / 2) x = mk<T>(0, 0);
                        acc.st(i, x);
                    }
            }
        } else {
            C w[VR];
            C *vb = v;
            if constexpr (OP == OP_DERIV) reg_deriv<T, N, D::RFL, LL>(v, a.ktab, t);
            if constexpr (OP == OP_PAD) { reg_pad<T, N, D::RFL, LL>(v, w, t); vb = w; }
            fft_regs<NO, typename D::PB, LL, false>(vb, acc, twB, t);
            using G = Geo<NO, D::RBL, LL>;
            const T ar = OP == OP_PAD ? cr : (T)0;
            const T ai = OP == OP_PAD ? ci : (T)0;
#pragma unroll
            for (int b = 0; b < G::PER; ++b) {
                const int j = t + LL * b;
                if (G::FULL || j < G::NB)
#pragma unroll
                    for (int r = 0; r < D::RBL; ++r) {
                        C x = vb[b * D::RBL + r];
                        x.x += ar;
                        x.y += ai;
                        acc.st(j + r * G::NB, x);
                    }
            }
        }
    };
    if constexpr (REAL) {
        TilePair<T> acc{tile, S, cc, act};
        body(acc);
    } else {
        TileCol<C> acc{tile, S, cc, act};
        body(acc);
    }
    __syncthreads();

    for (int idx = threadIdx.x; idx < NO * W; idx += blockDim.x) {
        const int r = idx / W, cx = idx - r * W;
        if (cx < nc) dst[(long long)r * a.dst_row + cx] = tile[sidx(r) * S + cx];
    }
    __syncthreads();   // the tile may be reused by the caller's next unit
}

#ifndef OBL_COL_PF
#define OBL_COL_PF 2   // y-pad column kernel: L2 prefetch distance in quarters of a residency window (0 = off)
#endif
// ----------------------------------------------------------------------------- two-pass columns
// Geometry of a line operation: RI, RO the second radices of its input and output
// transforms, PI and PO the pitches of their exchanges, ROWS the exchange rows of one line
// (a forward-only transform takes radix R1 first and exchanges R0 rows of pitch PO).
template <int N, int OP> struct TpLine {
    static constexpr int R0 = TwoPass<N>::R0, R1 = TwoPass<N>::R1;
    static constexpr int RI = OP == OP_UNPAD ? 3 * R1 / 2 : R1, RO = OP == OP_PAD ? 3 * R1 / 2 : R1;
    static constexpr int NI = R0 * RI, NO = R0 * RO;
    static constexpr int PI = tp_pitch(R0), PO = tp_pitch(RO);
    static constexpr int rows_in = OP == OP_INV || OP == OP_FWD ? 0 : RI * PI, rows_out = R0 * PO;
    static constexpr int ROWS = rows_in > rows_out ? rows_in : rows_out;
};

// v (bins j + r*R0 of a line of N) *= i*k_signed (ktab[N/2] = 0 drops the Nyquist mode)
template <typename T, int N, int R0, int R1>
__device__ __forceinline__ void tp_deriv(C2<T> (&v)[R1], const double *ktab, int j)
{
#pragma unroll
    for (int r = 0; r < R1; ++r) {
        const int k = j + r * R0;
        const T kk = k <= N / 2 ? (T)ktab[k] : -(T)ktab[N - k];
        v[r] = mk<T>(-kk * v[r].y, kk * v[r].x);
    }
}

// One CTA unit: the WB adjacent complex lines (WB real column pairs, or WB complex columns)
// bx*WB.. of plane z, NT threads.  Thread t serves line t % WB in every pass, so the WB
// lanes of a butterfly read and store WB adjacent pairs; the exchange is line-minor
// (element row e of line l at buf[e*WB + l]).
// SMEM_IN: the unit's input is already in buf, row i of line l at buf[i*WB + l].
template <typename T, int N, int OP, bool REAL, int NT, int WB, bool SMEM_IN = false>
__device__ __forceinline__ void tp_cols_unit(const ColArgs<T> &a, int bx, int z, C2<T> *buf)
{
    using C = C2<T>;
    using E = typename std::conditional<REAL, T, C>::type;
    using D = TpLine<N, OP>;
    constexpr int R0 = D::R0, RI = D::RI, RO = D::RO;
    constexpr int I1 = RI * WB, I2 = R0 * WB, I3 = RO * WB;       // butterflies of the three mappings
    constexpr int PER1 = (I1 + NT - 1) / NT, PER2 = I2 / NT;
    static_assert(NT % WB == 0 && I2 % NT == 0, "whole butterflies per thread in the middle passes");
    static_assert(!SMEM_IN || PER1 == 1, "an input tile is read before its exchange overwrites it");
    const int tid = threadIdx.x, line = tid % WB;
    const int gl = bx * WB + line;                         // global line index
    const int nlines = REAL ? a.ncols / 2 : a.ncols;
    const bool act = gl < nlines;
    const int glc = act ? gl : 0;
    const E *srcz = reinterpret_cast<const E *>(a.src) + (long long)z * a.src_plane;
    E *dstz = reinterpret_cast<E *>(a.dst) + (long long)z * a.dst_plane;
    // the checked build tests each element's level, column and plane offset against the
    // extents the arguments give (nlev planes of src_plane / dst_plane, rows of src_row / dst_row)
    auto col_ok = [&](int i, int col, int row, long long plane, int site) {
        const int ce = REAL ? 2 * col + 1 : col;
        return ck_in(z, a.nlev, site) && ck_in(ce, row, site) && ck_in((long long)i * row + ce, plane, site);
    };
    auto gld = [&](int i) -> C {
        if constexpr (SMEM_IN) return buf[i * WB + line];
        else {
            if (OBL_CHECK && !col_ok(i, glc, a.src_row, a.src_plane, CK_COL_LOAD)) return mk<T>(0, 0);
            if constexpr (REAL) return __ldcg(reinterpret_cast<const C *>(srcz + (long long)i * a.src_row + 2 * glc));
            else return __ldcg(srcz + (long long)i * a.src_row + glc);
        }
    };
    auto gst = [&](int i, C v) {
        if (OBL_CHECK && !col_ok(i, gl, a.dst_row, a.dst_plane, CK_COL_STORE)) return;
        if constexpr (REAL) *reinterpret_cast<C *>(dstz + (long long)i * a.dst_row + 2 * gl) = v;
        else dstz[(long long)i * a.dst_row + gl] = v;
    };
    if constexpr (OP == OP_FWD) {
        // forward only: radix R1 first, so that every thread loads; twB's table is w_N^(r k),
        // k < R1
        constexpr int PF = tp_pitch(D::R1);
#pragma unroll
        for (int b = 0; b < PER2; ++b) {
            const int j = (tid + b * NT) / WB;
            C x[D::R1];
#pragma unroll
            for (int r = 0; r < D::R1; ++r) x[r] = act ? gld(j + r * R0) : mk<T>(0, 0);
#pragma unroll
            for (int r = 0; r < D::R1; ++r) x[r] = cscale(x[r], a.scale);
            Dft<D::R1, true>::run(x);
#pragma unroll
            for (int r = 0; r < D::R1; ++r) buf[(j * PF + r) * WB + line] = x[r];
        }
        __syncthreads();
#pragma unroll 1
        for (int f = tid; f < D::R1 * WB; f += NT) {
            const int j = f / WB;
            C x[R0];
#pragma unroll
            for (int r = 0; r < R0; ++r) x[r] = buf[(r * PF + j) * WB + line];
#pragma unroll
            for (int r = 1; r < R0; ++r) x[r] = cmul(x[r], __ldg(a.twB + r * D::R1 + j));
            Dft<R0, true>::run(x);
            if (act) {
#pragma unroll
                for (int r = 0; r < R0; ++r)
                    gst(j + r * D::R1, r == R0 / 2 && a.zero_nyq && j == 0 ? mk<T>(0, 0) : x[r]);   // bin N/2
            }
        }
        return;
    }
    C cref = mk<T>(0, 0);
    C v[PER2][D::R1];

    if constexpr (OP != OP_INV) {
        if constexpr (REAL) cref = gld(0);
#pragma unroll
        for (int b = 0; b < PER1; ++b) {
            const int f = tid + b * NT, j = f / WB;
            const bool on = I1 % NT == 0 || f < I1;
            C x[R0];
            if (on) {
#pragma unroll
                for (int r = 0; r < R0; ++r) x[r] = act ? gld(j + r * RI) : mk<T>(0, 0);
                // (a loop of its own: arithmetic inside the conditional load kept the loads
                // from being issued together; ddy of 512 lines 0.669 -> 0.566 ms per step)
#pragma unroll
                for (int r = 0; r < R0; ++r) x[r] = cscale(csub(x[r], cref), a.scale);
            }
            if constexpr (SMEM_IN) __syncthreads();   // the tile is read before the exchange overwrites it
            if (on) {
                Dft<R0, true>::run(x);
#pragma unroll
                for (int r = 0; r < R0; ++r) buf[(j * D::PI + r) * WB + line] = x[r];
            }
        }
        __syncthreads();
#pragma unroll
        for (int b = 0; b < PER2; ++b) {
            const int j = (tid + b * NT) / WB;
            C x[RI];
#pragma unroll
            for (int r = 0; r < RI; ++r) x[r] = buf[(r * D::PI + j) * WB + line];
#pragma unroll
            for (int r = 1; r < RI; ++r) x[r] = cmul(x[r], __ldg(a.twF + r * R0 + j));
            if constexpr (OP == OP_UNPAD) {
                DftUnpad<D::R1>::run(x, v[b]);
                if (j == 0) v[b][RO / 2] = mk<T>(0, 0);   // bin N/2
            } else {
                Dft<RI, true>::run(x);
#pragma unroll
                for (int r = 0; r < RI; ++r) v[b][r] = x[r];
            }
        }
        __syncthreads();   // the exchange is read before it is written again
    } else {
#pragma unroll
        for (int b = 0; b < PER2; ++b) {
            const int j = (tid + b * NT) / WB;
#pragma unroll
            for (int r = 0; r < RO; ++r) {
                const int i = j + r * R0;
                C x = act ? gld(i) : mk<T>(0, 0);
                v[b][r] = cscale(x, a.scale);
            }
        }
    }
#pragma unroll
    for (int b = 0; b < PER2; ++b) {
        const int j = (tid + b * NT) / WB;
        if constexpr (OP == OP_PAD) {
            if (j == 0) v[b][RI / 2] = mk<T>(0, 0);   // the source's Nyquist bin
            DftPad<D::R1>::run(v[b], [&](auto ic, C x) { buf[(j * D::PO + decltype(ic)::value) * WB + line] = x; });
        } else {
            if constexpr (OP == OP_DERIV) tp_deriv<T, N, R0, RO>(v[b], a.ktab, j);
            if constexpr (OP == OP_FILT) if (j == 0) v[b][RO / 2] = mk<T>(0, 0);
            Dft<RO, false>::run(v[b]);
#pragma unroll
            for (int r = 0; r < RO; ++r) buf[(j * D::PO + r) * WB + line] = v[b][r];
        }
    }
    __syncthreads();
    constexpr bool addc = OP == OP_PAD || OP == OP_UNPAD;
#pragma unroll 1
    for (int f = tid; f < I3; f += NT) {
        const int j = f / WB;
        C x[R0];
#pragma unroll
        for (int r = 0; r < R0; ++r) x[r] = buf[(r * D::PO + j) * WB + line];
#pragma unroll
        for (int r = 1; r < R0; ++r) x[r] = cmulc(x[r], __ldg(a.twB + r * RO + j));
        Dft<R0, false>::run(x);
        if (act) {
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const int i = j + r * RO;
                C y = x[r];
                if (addc) {
                    y.x += cref.x;
                    y.y += cref.y;
                }
                gst(i, y);
                if constexpr (OP == OP_UNPAD && REAL) {
                    // var(nxt+1:ldx,:) = var(1:2,:) (108_01_padd.f90:195)
                    if (a.pad_copy && gl == 0 && ck_in(a.ncols + 1, a.dst_row, CK_COL_STORE))
                        *reinterpret_cast<C *>(dstz + (long long)i * a.dst_row + a.ncols) = y;
                }
            }
        }
    }
}

// Threads, lines and registers of the column kernels: WB lines (64-byte row segments; 128
// bytes for the short lines of R0 = 8), R0*WB/PER2 threads.  FP32: 24 resident warps with
// one middle butterfly a thread (80 registers) beat 16 warps with two (y-pad of 512 lines,
// 258 levels, as first built: 0.846 against 0.881 ms over four fields; 20 warps spill: 0.949), except
// where all threads load at once in the forward-only transform (0.351 against 0.388 ms for
// three spectra).  FP64 radix-32 butterflies need 8 warps; two middle butterflies a thread
// keep more of them loading (ddy 1.214 against 1.450 ms), which the y-pad's larger exchange
// does not repay (2.63 against 2.34 ms).
// Against the three-radix kernels (ms per step at 512x512x256 levels, before -> now): FP32
// y-pad 1.243 -> 0.888, ddy 0.714 -> 0.566, y-transform 0.393 -> 0.358; FP64 y-pad 3.00 ->
// 2.31, ddy 1.85 -> 1.30; at 128x128 levels the y-pad takes 0.62 and the y-unpad 0.55 of
// their time.
// The L1/shared pipe fell from 69 to 55% busy (y-pad of 64 levels, 91 -> 66 us).  A persistent form
// with the next tile's copies in flight measured slower (1.25 ms): its second tile leaves
// shared memory for 16 warps only.
#ifndef OBL_TP_WARPS_SM
#define OBL_TP_WARPS_SM 24   // resident warps per SM the FP32 column kernels' registers are bounded for
#endif
#ifndef OBL_TP_LINES
#define OBL_TP_LINES 8       // lines per CTA of the FP32 column kernels with R0 > 8
#endif
template <typename T, int N, int OP> struct TpGeo {
    static constexpr int R0 = TwoPass<N>::R0;
    static constexpr int WB = sizeof(T) == 4 ? (R0 == 8 ? 16 : OBL_TP_LINES) : (R0 == 8 ? 8 : 4);
    static constexpr int PER2 = R0 == 32 && (OP == OP_FWD || (sizeof(T) == 8 && OP != OP_PAD)) ? 2 : 1;
    static constexpr int NT = R0 * WB / PER2;
    static constexpr int wsm = sizeof(T) == 4 ? (PER2 == 2 ? 16 : OBL_TP_WARPS_SM) : (R0 == 32 ? 8 : R0 >= 20 ? 12 : 16);
    static constexpr int minb = wsm * 32 / NT > 0 ? wsm * 32 / NT : 1;
};
template <typename T, int N, int OP> inline size_t tp_cols_smem()
{
    using D = TpLine<N, OP>;
    return sizeof(C2<T>) * (size_t)(D::ROWS > D::NI ? D::ROWS : D::NI) * TpGeo<T, N, OP>::WB;
}
template <typename T, int N, int OP, bool REAL>
__global__ void __launch_bounds__(TpGeo<T, N, OP>::NT, TpGeo<T, N, OP>::minb) k_tp_cols(ColArgs<T> a)
{
    using G = TpGeo<T, N, OP>;
    extern __shared__ __align__(128) unsigned char smraw[];
    tp_cols_unit<T, N, OP, REAL, G::NT, G::WB>(a, blockIdx.x, blockIdx.y, reinterpret_cast<C2<T> *>(smraw));
}

// ----------------------------------------------------------------------------- two-pass rows
// The same two passes for contiguous lines: a CTA holds WB row pairs (each one complex
// line) and in every pass deals the pairs (line, butterfly) to consecutive threads with the
// butterfly fastest, so that a warp reads and stores consecutive elements of a row.  The
// exchange of a line is contiguous; line pitches are 8 modulo 16 elements, which keeps the
// lines that share a warp on different banks.  Twiddles come through the read-only path.
// Against the three-radix warp-per-line kernels (us, before -> now, 64 levels of 512x512
// points or as many points): ddx of 512 lines FP32 52 -> 43, x-unpad 81 -> 68; of 384 lines
// 54 -> 39, 91 -> 60; FP64 256 lines 94 -> 60, 189 -> 109.
constexpr int tp_line(int n) { return n + (24 - n % 16) % 16; }

template <typename T, int N, int WB_ = 0> struct TpRows {
    static constexpr int R0 = TwoPass<N>::R0, R1 = TwoPass<N>::R1, RP = 3 * R1 / 2;
    static constexpr int N2 = R0 * RP, LH = N / 2 + 1;
    static constexpr int PF = tp_pitch(R0), PD = tp_pitch(R1), PP = tp_pitch(RP);
    // exchange elements of one line: forward of N and of 3N/2, backward of N and of 3N/2
    static constexpr int LF = tp_line(R1 * PF), LF2 = tp_line(RP * PF), LD = tp_line(R0 * PD), LP = tp_line(R0 * PP);
    static constexpr int WB = WB_ ? WB_ : R0 == 8 ? (sizeof(T) == 4 ? 16 : 8) : R0 == 16 ? (sizeof(T) == 4 ? 8 : 4) : R0 == 20 ? 8 : R0 == 32 && sizeof(T) == 8 ? 2 : 4;
    static constexpr int NT = R0 * WB;                     // one middle-pass butterfly a thread
    // (FP64 radix 32 leaves 8 warps: 4 CTAs of 2 lines against 2 of 4 took the multi-output
    // pass of 512 lines from 2.61 to 2.38 ms and the inverse from 1.34 to 1.26)
    // the inverse's first pass loads: at R0 = 32 its 10..20 butterflies a line are dealt to
    // half as many threads, which then take two middle butterflies each
    static constexpr int PERI = R0 == 32 ? 2 : 1, NTI = NT / PERI;
    // resident warps per SM the registers are bounded for.  FP32: 16 with radices from 20 (20
    // warps spill: the multi-output pass of 512 lines 1.133 instead of 1.108 ms per step), 20
    // below; FP64: 8 with radix 32 (12 spill: 3.6 against 2.4 ms), 16 with 20, else 12.
    static constexpr int wsm = sizeof(T) == 4 ? (R0 >= 20 ? 16 : 20) : (R0 == 32 ? 8 : R0 == 20 ? 16 : 12);
    static constexpr int minb = wsm * 32 / NT > 0 ? wsm * 32 / NT : 1, minbI = wsm * 32 / NTI > 0 ? wsm * 32 / NTI : 1;
    static_assert(NT % 32 == 0, "whole warps: the spectra are split by shuffles");
    template <int OP> static constexpr int line_elems()
    {
        return OP == OP_DERIV ? (LF > LD ? LF : LD) : OP == OP_PAD ? (LF > LP ? LF : LP) : OP == OP_UNPAD ? (LF2 > LD ? LF2 : LD)
                                                                             : OP == OP_FWD ? LF : LF;
    }
    static constexpr int LPF = LP > LF ? LP : LF;
    static constexpr size_t smem_fwd3 = sizeof(C2<T>) * (size_t)WB * (LD + LPF), smem_fwd3_seq = sizeof(C2<T>) * (size_t)WB * LPF;
};

// First forward pass: butterfly f = (line, j) of radix R0 over x[j + r*RI] of rows A, B
template <typename T, int R0, int RI, int WB, int NT, int LS, class ROWS>
__device__ __forceinline__ void tp_rows_first(const ROWS &rows, T scale, C2<T> *buf)
{
    using C = C2<T>;
#pragma unroll 1
    for (int f = threadIdx.x; f < RI * WB; f += NT) {
        const int line = f / RI, j = f % RI;
        const T *A, *B;
        if (!rows(line, A, B)) continue;
        const T ca = A[0], cb = B[0];
        C x[R0];
#pragma unroll
        for (int r = 0; r < R0; ++r) x[r] = mk<T>(A[j + r * RI], B[j + r * RI]);
        const C c = mk<T>(ca, cb);
#pragma unroll
        for (int r = 0; r < R0; ++r) x[r] = cscale(csub(x[r], c), scale);
        Dft<R0, true>::run(x);
#pragma unroll
        for (int r = 0; r < R0; ++r) buf[line * LS + j * tp_pitch(R0) + r] = x[r];
    }
}

// Last backward pass: butterfly (line, j) of radix R0 from the exchange; emit(line, i, x).
// `first` is the thread's first butterfly (two loops of one phase start from opposite ends)
template <typename T, int R0, int RO, int WB, int NT, int LS, class EMIT>
__device__ __forceinline__ void tp_rows_last(int first, const C2<T> *buf, const C2<T> *tw, EMIT &&emit)
{
    using C = C2<T>;
#pragma unroll 1
    for (int f = first; f < RO * WB; f += NT) {
        const int line = f / RO, j = f % RO;
        C x[R0];
#pragma unroll
        for (int r = 0; r < R0; ++r) x[r] = buf[line * LS + r * tp_pitch(RO) + j];
#pragma unroll
        for (int r = 1; r < R0; ++r) x[r] = cmulc(x[r], __ldg(tw + r * RO + j));
        Dft<R0, false>::run(x);
        emit(line, j, x);
    }
}

// Half spectra of the two rows of a line from its spectrum Z (v[r] = bin j + r*R0 in the
// thread of butterfly j): A = (Z[k] + conj Z[N-k])/2, B = (Z[k] - conj Z[N-k])/(2i) for
// k < N/2.  Bin N-k is v[R1-1-r] of butterfly R0-j (of the same one for j = 0), a lane of
// the same warp; emit(k, a, b).  Every lane of the warp calls it.
template <typename T, int R0, int R1, class EMIT>
__device__ __forceinline__ void tp_split_spectra(const C2<T> (&v)[R1], int j, EMIT &&emit)
{
    using C = C2<T>;
    static_assert(32 % R0 == 0, "a line's butterflies lie in one warp");
    const int lane = threadIdx.x & 31, src = (lane & ~(R0 - 1)) + ((R0 - j) & (R0 - 1));
#pragma unroll
    for (int r = 0; r < R1 / 2; ++r) {
        const C p = j == 0 ? v[(R1 - r) % R1] : v[R1 - 1 - r];
        C q;
        q.x = __shfl_sync(0xffffffffu, p.x, src);
        q.y = -__shfl_sync(0xffffffffu, p.y, src);
        const C s = cadd(v[r], q), d = csub(v[r], q);
        emit(j + r * R0, s, mk<T>(d.y, -d.x));
    }
}

// The same from the line's spectrum in shared memory (bin k at z[k]), for R0 not a power of two
template <typename T, int N, int R0, int R1, class EMIT>
__device__ __forceinline__ void tp_split_spectra_smem(const C2<T> (&v)[R1], int j, const C2<T> *z, EMIT &&emit)
{
    using C = C2<T>;
#pragma unroll
    for (int r = 0; r < R1 / 2; ++r) {
        const int k = j + r * R0;
        const C q = cconj(z[k == 0 ? 0 : N - k]);
        const C s = cadd(v[r], q), d = csub(v[r], q);
        emit(k, s, mk<T>(d.y, -d.x));
    }
}


// Inverse of two rows' half spectra A, B (one complex line Z = A + iB on all N bins; Im of
// the DC and Nyquist bins is ignored, as in FFTW's c2r): radix R0 from global memory, one
// exchange, radix R1; op(j, z) may multiply the bins j + r*R1 before the transform, and
// pre(line, j) is called before, emit(line, j, x) with the elements j + r*R0.  tw: the forward table of N = R0*R1
template <typename T, int N, int WB_, class ROWS, class OPF, class PRE, class EMIT>
__device__ __forceinline__ void tp_rows_inv(const ROWS &rows, const OPF &op, C2<T> *buf, const C2<T> *tw, PRE &&pre, EMIT &&emit)
{
    using C = C2<T>;
    using G = TpRows<T, N, WB_>;
    constexpr int R0 = G::R0, R1 = G::R1, WB = G::WB, NT = G::NTI, LS = G::LF;
#pragma unroll 1
    for (int f = threadIdx.x; f < R1 * WB; f += NT) {
        const int line = f / R1, j = f % R1;
        const C *A, *B;
        if (!rows(line, A, B)) continue;
        C x[R0];
#pragma unroll
        for (int r = 0; r < R0; ++r) {
            const int i = j + r * R1;
            const bool lo = r < R0 / 2 || (r == R0 / 2 && j == 0);   // i <= N/2
            const int k = lo ? i : N - i;
            C av = __ldcg(A + k), bv = __ldcg(B + k);
            if (j == 0 && (r == 0 || r == R0 / 2)) { av.y = 0; bv.y = 0; }
            x[r] = lo ? mk<T>(av.x - bv.y, av.y + bv.x) : mk<T>(av.x + bv.y, bv.x - av.y);
        }
        op(j, x);
        Dft<R0, false>::run(x);
#pragma unroll
        for (int r = 0; r < R0; ++r) buf[line * LS + j * G::PF + r] = x[r];
    }
    __syncthreads();
#pragma unroll 1
    for (int b = 0; b < G::PERI; ++b) {
        const int f = threadIdx.x + b * NT, line = f / R0, j = f % R0;
        pre(line, j);
        C x[R1];
#pragma unroll
        for (int r = 0; r < R1; ++r) x[r] = buf[line * LS + r * G::PF + j];
#pragma unroll
        for (int r = 1; r < R1; ++r) x[r] = cmulc(x[r], __ldg(tw + r * R0 + j));
        Dft<R1, false>::run(x);
        emit(line, j, x);
    }
}

template <typename T, int N, int OP>
__device__ __forceinline__ void tp_row_unit(const RowArgs<T> &a, long long base, C2<T> *buf)
{
    using C = C2<T>;
    using G = TpRows<T, N>;
    constexpr int R0 = G::R0, R1 = G::R1, WB = G::WB, NT = G::NT;
    constexpr int RI = OP == OP_UNPAD ? G::RP : R1, RO = OP == OP_PAD ? G::RP : R1, NO = R0 * RO;
    constexpr int LI = OP == OP_UNPAD ? G::LF2 : G::LF, LO = OP == OP_PAD ? G::LP : G::LD;
    const int tid = threadIdx.x;
    auto active = [&](int line) { return base + line < a.npairs; };
    if constexpr (OP != OP_INV) {
        auto src = [&](int line, const T *&A, const T *&B) {
            if (!active(line)) return false;
            A = reinterpret_cast<const T *>(a.src) + 2 * (base + line) * a.src_stride;
            B = A + a.src_stride;
            return true;
        };
        tp_rows_first<T, R0, RI, WB, NT, LI>(src, a.scale, buf);
        __syncthreads();
        const int line = tid / R0, j = tid % R0;
        C v[R1];
        {
            C x[RI];
#pragma unroll
            for (int r = 0; r < RI; ++r) x[r] = buf[line * LI + r * G::PF + j];
#pragma unroll
            for (int r = 1; r < RI; ++r) x[r] = cmul(x[r], __ldg(a.twF + r * R0 + j));
            if constexpr (OP == OP_UNPAD) {
                DftUnpad<R1>::run(x, v);
                if (j == 0) v[R1 / 2] = mk<T>(0, 0);   // bin N/2
            } else {
                Dft<RI, true>::run(x);
#pragma unroll
                for (int r = 0; r < RI; ++r) v[r] = x[r];
            }
        }
        if constexpr (OP == OP_FWD) {
            // both rows' half spectra; the x-Nyquist is zeroed (203_fftn_mpi.f90:25) and the
            // subtracted constants return in the DC bins.  A[0] and B[0] are read by the
            // thread that overwrites them when the call transforms in place
            const bool act = active(line);
            const long long r0 = 2 * (act ? base + line : base);
            C *Ao = reinterpret_cast<C *>(a.dst) + r0 * a.dst_stride, *Bo = Ao + a.dst_stride;
            const T *A = reinterpret_cast<const T *>(a.src) + r0 * a.src_stride;
            auto put = [&](int k, C s, C d) {
                C ao = cscale(s, (T)0.5), bo = cscale(d, (T)0.5);
                if (act) {
                    if (k == 0) {
                        ao.x += A[0] * a.scale * (T)N;
                        bo.x += A[a.src_stride] * a.scale * (T)N;
                    }
                    Ao[k] = ao;
                    Bo[k] = bo;
                }
            };
            if constexpr (32 % R0 == 0) {
                tp_split_spectra<T, R0, R1>(v, j, put);
            } else {
                __syncthreads();
#pragma unroll
                for (int r = 0; r < R1; ++r) buf[line * LI + j + r * R0] = v[r];
                __syncthreads();
                tp_split_spectra_smem<T, N, R0, R1>(v, j, buf + line * LI, put);
            }
            if (act && j == 0) Ao[N / 2] = Bo[N / 2] = mk<T>(0, 0);
            return;
        }
        __syncthreads();   // the exchange is read before it is written again
        if constexpr (OP == OP_PAD) {
            if (j == 0) v[R1 / 2] = mk<T>(0, 0);   // the source's Nyquist bin
            DftPad<R1>::run(v, [&](auto ic, C x) { buf[line * LO + j * tp_pitch(RO) + decltype(ic)::value] = x; });
        } else {
            if constexpr (OP == OP_DERIV) tp_deriv<T, N, R0, R1>(v, a.ktab, j);
            Dft<R1, false>::run(v);
#pragma unroll
            for (int r = 0; r < R1; ++r) buf[line * LO + j * tp_pitch(RO) + r] = v[r];
        }
        __syncthreads();
        constexpr bool addc = OP == OP_PAD || OP == OP_UNPAD;
        tp_rows_last<T, R0, RO, WB, NT, LO>(tid, buf, a.twB, [&](int ln, int jj, const C(&x)[R0]) {
            if (!active(ln)) return;
            const long long r0 = 2 * (base + ln);
            T *A = reinterpret_cast<T *>(a.dst) + r0 * a.dst_stride, *B = A + a.dst_stride;
            T addA = 0, addB = 0;
            if (addc) {
                const T *S = reinterpret_cast<const T *>(a.src) + r0 * a.src_stride;
                addA = S[0];
                addB = S[a.src_stride];
            }
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                A[jj + r * RO] = x[r].x + addA;
                B[jj + r * RO] = x[r].y + addB;
            }
        });
    } else {
        auto src = [&](int line, const C *&A, const C *&B) {
            if (!active(line)) return false;
            A = reinterpret_cast<const C *>(a.src) + 2 * (base + line) * a.src_stride;
            B = A + a.src_stride;
            return true;
        };
        auto same = [](int, C *) {};
        tp_rows_inv<T, N, 0>(src, same, buf, a.twF, [](int, int) {}, [&](int ln, int jj, const C(&x)[R1]) {
            const long long r0 = 2 * (base + ln);
            if (!active(ln)) return;
            T *A = reinterpret_cast<T *>(a.dst) + r0 * a.dst_stride, *B = A + a.dst_stride;
#pragma unroll
            for (int r = 0; r < R1; ++r) {
                A[jj + r * R0] = x[r].x;
                B[jj + r * R0] = x[r].y;
            }
            if (a.pad_mode && jj < 2) {
                A[NO + jj] *= a.pad_scale;
                B[NO + jj] *= a.pad_scale;
            }
        });
    }
}

template <typename T, int N, int OP>
__global__ void __launch_bounds__(OP == OP_INV ? TpRows<T, N>::NTI : TpRows<T, N>::NT, OP == OP_INV ? TpRows<T, N>::minbI : TpRows<T, N>::minb)
    k_tp_rows(RowArgs<T> a)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    tp_row_unit<T, N, OP>(a, (long long)blockIdx.x * TpRows<T, N>::WB, reinterpret_cast<C2<T> *>(smraw));
}

// ----------------------------------------------------------------------------- TMA-fed y-pad
// The FP32 y-pad with its CTA's input tile (NI rows x WB real column pairs of the x-padded
// plane) brought into shared memory by tensor-map copies: one thread issues
// cp.async.bulk.tensor loads of boxes of 2*WB floats x box_rows rows (64-byte row segments,
// landing row after row: element i of line l at tile[i*WB + l], the line-minor layout of
// the exchange scratch), completing on an mbarrier, and the same thread asks L2 for the
// tile pf_ahead planes later (cp.async.bulk.prefetch.tensor).  The tile lands in the
// exchange scratch the CTA already holds, so shared memory per CTA and CTAs per SM stay
// those of k_tp_cols.  The tensor map covers this GPU's own x-padded planes; no multicast.
// The wait is bounded: on timeout wait_err is set (the host reports OBL_ERR_TIMEOUT), the
// CTA waits once more (bounded) for the copy, and its results are not to be used.
template <typename T, int N, int OP, bool REAL>
__global__ void __launch_bounds__(TpGeo<T, N, OP>::NT, TpGeo<T, N, OP>::minb)
    k_tp_cols_tma(ColArgs<T> a, const __grid_constant__ CUtensorMap tm, int box_rows)
{
    using C = C2<T>;
    using D = TpLine<N, OP>;
    constexpr int WB = TpGeo<T, N, OP>::WB;
    extern __shared__ __align__(128) unsigned char smraw[];
    __shared__ __align__(8) unsigned long long bar;
    // tensor copies write 128-byte aligned shared memory (an offset from smraw keeps the
    // pointer in the shared window for the compiler)
    C *buf = reinterpret_cast<C *>(smraw + ((128u - (smem_addr(smraw) & 127u)) & 127u));
    const unsigned sbar = smem_addr(&bar);
    const int x0 = blockIdx.x * 2 * WB, y0 = blockIdx.y * D::NI;
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n\tfence.mbarrier_init.release.cluster;\n\t"
                     "fence.proxy.async.shared::cta;" ::"r"(sbar)
                     : "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sbar),
                     "r"((unsigned)(sizeof(C) * D::NI * WB))
                     : "memory");
        for (int y = 0; y < D::NI; y += box_rows)
            asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
                         "[%0], [%1, {%2, %3}], [%4];" ::"r"(smem_addr(buf + (size_t)y * WB)),
                         "l"(&tm), "r"(x0), "r"(y0 + y), "r"(sbar)
                         : "memory");
        if (a.pf_ahead > 0 && (int)blockIdx.y + a.pf_ahead < a.nlev)
            for (int y = 0; y < D::NI; y += box_rows)
                asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(&tm), "r"(x0),
                             "r"(y0 + a.pf_ahead * D::NI + y)
                             : "memory");
    }
    __syncthreads();   // the barrier is initialised before anyone waits on it
    if (!mbar_wait_bounded(sbar, 0)) {
        if (a.wait_err) atomicExch(a.wait_err, 1);
        mbar_wait_bounded(sbar, 0);   // a late copy lands before the tile is reused
    }
    tp_cols_unit<T, N, OP, REAL, TpGeo<T, N, OP>::NT, WB, true>(a, blockIdx.x, blockIdx.y, buf);
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no libcuda link)
typedef CUresult (*TensorMapEncodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                         const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                         CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                         CUtensorMapFloatOOBfill);
inline TensorMapEncodeTiled tensor_map_encoder()
{
    static TensorMapEncodeTiled fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (TensorMapEncodeTiled)p;
        else
            cudaGetLastError();
    }
    return fn;
}

// rows per tensor copy: NI itself up to 256 rows (the box limit), else the largest divisor
// of NI not above 256; 0 = no such split
constexpr int tma_box_rows(int ni)
{
    if (ni <= 256) return ni;
    for (int b = 256; b >= 8; --b)
        if (ni % b == 0) return b;
    return 0;
}

// ----------------------------------------------------------------------------- launchers
template <typename T, int N, int OP> cudaError_t launch_rows_t(const RowArgs<T> &a, cudaStream_t s)
{
    using G = TpRows<T, N>;
    static bool inits[kMaxDevices] = {};
    constexpr size_t sm = sizeof(C2<T>) * (size_t)G::WB * G::template line_elems<OP>();
    auto kern = k_tp_rows<T, N, OP>;
    const int ds = device_slot();
    if (ds < 0 || !inits[ds]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
        if (ds >= 0) inits[ds] = true;
    }
    const long long grid = (a.npairs + G::WB - 1) / G::WB;
    if (grid < 1) return cudaSuccess;
    kern<<<(unsigned)grid, OP == OP_INV ? G::NTI : G::NT, sm, s>>>(a);
    return cudaGetLastError();
}

template <typename T, int N, int OP, bool REAL> cudaError_t launch_cols_t(const ColArgs<T> &a0, cudaStream_t s)
{
    static bool inits[kMaxDevices] = {};
    constexpr int WB = TpGeo<T, N, OP>::WB, NT = TpGeo<T, N, OP>::NT;
    using D = TpLine<N, OP>;
    const size_t sm = tp_cols_smem<T, N, OP>();
    auto kern = k_tp_cols<T, N, OP, REAL>;
    const int ds = device_slot();
    if (ds < 0 || !inits[ds]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
        if (ds >= 0) inits[ds] = true;
    }
    ColArgs<T> a = a0;
    const int nlines = REAL ? a.ncols / 2 : a.ncols;
    if constexpr (std::is_same<T, float>::value && OP == OP_PAD && REAL && D::RI <= D::R0 && N >= 256 && tma_box_rows(D::NI) > 0) {
        // the x-padded planes as a 2-D map: ncols floats wide (pitch src_row), NI*nlev rows
        const bool fits = a.tma && a.src_plane == a.src_row * (long long)D::NI && (a.src_row * 4) % 16 == 0 &&
                          ((uintptr_t)a.src % 16) == 0 && tensor_map_encoder() != nullptr;
        if (fits) {
            constexpr int BR = tma_box_rows(D::NI);
            CUtensorMap tm;
            const cuuint64_t dims[2] = {(cuuint64_t)a.ncols, (cuuint64_t)D::NI * a.nlev};
            const cuuint64_t strides[1] = {(cuuint64_t)a.src_row * sizeof(T)};
            const cuuint32_t box[2] = {(cuuint32_t)(2 * WB), (cuuint32_t)BR};
            const cuuint32_t estr[2] = {1, 1};
            if (tensor_map_encoder()(&tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void *>(a.src), dims, strides,
                                     box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                     CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return cudaErrorInvalidValue;
            static int tres[kMaxDevices] = {};
            auto tk = k_tp_cols_tma<T, N, OP, REAL>;
            const size_t tsm = sm + 128;
            int tr = ds >= 0 ? tres[ds] : 0;
            if (!tr) {
                cudaError_t e = cudaFuncSetAttribute(tk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsm);
                if (e != cudaSuccess) return e;
                int dev = 0, nsm = 0, per = 0;
                cudaGetDevice(&dev);
                cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, tk, NT, tsm);
                tr = nsm * (per > 0 ? per : 1);
                if (ds >= 0) tres[ds] = tr;
            }
            dim3 grid((nlines + WB - 1) / WB, a.nlev);
            if (grid.x < 1 || grid.y < 1) return cudaSuccess;
            if (OBL_COL_PF) a.pf_ahead = (int)((OBL_COL_PF * (long long)tr + 4LL * grid.x - 1) / (4LL * grid.x));
            tk<<<grid, NT, tsm, s>>>(a, tm, BR);
            return cudaGetLastError();
        }
    }
    dim3 grid((nlines + WB - 1) / WB, a.nlev);
    if (grid.x < 1 || grid.y < 1) return cudaSuccess;
    kern<<<grid, NT, sm, s>>>(a);
    return cudaGetLastError();
}

// Runtime dispatch: n is the base length (the unpadded one for PAD/UNPAD).
template <typename T> cudaError_t launch_rows(int op, int n, const RowArgs<T> &a, cudaStream_t s);
// (The kernels behind them are spread over units of compilation by precision and kind: the
// first call into a unit loads all of it, and nvcc compresses a large one.  The first FP64 ddy
// of a process took 10.8 ms with the complex columns in the same unit, 3.0 without; the first
// press_stag_array 59 to 100 ms with the multi-field, step and inverse kernels of both
// precisions in two units, 12 in units of their own; the first step 49 and 16 ms.)
template <typename T> cudaError_t launch_cols_real(int op, int n, const ColArgs<T> &a, cudaStream_t s);
template <typename T> cudaError_t launch_cols_cplx(int op, int n, const ColArgs<T> &a, cudaStream_t s);
template <typename T> inline cudaError_t launch_cols(int op, bool real, int n, const ColArgs<T> &a, cudaStream_t s)
{
    return real ? launch_cols_real<T>(op, n, a, s) : launch_cols_cplx<T>(op, n, a, s);
}

// The same line ops on up to kMultiFields fields of one shape in one launch: field f
// reads src[f] and writes dst[f]; the args' src/dst are ignored.  Rows: OP_DERIV, OP_PAD,
// OP_UNPAD, OP_FWD; columns: the real-column OP_DERIV, OP_PAD, OP_UNPAD and the complex
// OP_FWD.  For grids whose single-field launches are too small to fill the GPU.
constexpr int kMultiFields = 6;
template <typename T> struct MultiPtr {
    const void *src[kMultiFields];
    void *dst[kMultiFields];
};
template <typename T>
cudaError_t launch_rows_multi_fwd(int n, const RowArgs<T> &a, const MultiPtr<T> &m, int nf, cudaStream_t s);
template <typename T>
cudaError_t launch_cols_multi_fwd(int n, const ColArgs<T> &a, const MultiPtr<T> &m, int nf, cudaStream_t s);
template <typename T>
cudaError_t launch_rows_multi_real(int op, int n, const RowArgs<T> &a, const MultiPtr<T> &m, int nf, cudaStream_t s);
template <typename T>
cudaError_t launch_cols_multi_real(int op, int n, const ColArgs<T> &a, const MultiPtr<T> &m, int nf, cudaStream_t s);
template <typename T>
inline cudaError_t launch_rows_multi(int op, int n, const RowArgs<T> &a, const MultiPtr<T> &m, int nf, cudaStream_t s)
{
    if (nf < 1 || nf > kMultiFields) return cudaErrorInvalidValue;
    return op == OP_FWD ? launch_rows_multi_fwd<T>(n, a, m, nf, s) : launch_rows_multi_real<T>(op, n, a, m, nf, s);
}
template <typename T>
inline cudaError_t launch_cols_multi(int op, int n, const ColArgs<T> &a, const MultiPtr<T> &m, int nf, cudaStream_t s)
{
    if (nf < 1 || nf > kMultiFields) return cudaErrorInvalidValue;
    return op == OP_FWD ? launch_cols_multi_fwd<T>(n, a, m, nf, s) : launch_cols_multi_real<T>(op, n, a, m, nf, s);
}
bool line_length_supported(int n);
// twiddle tables (interleaved re,im in FP64) of the plans of base length n, by role
std::vector<std::vector<double>> plan_tables(int n);

} // namespace obl
