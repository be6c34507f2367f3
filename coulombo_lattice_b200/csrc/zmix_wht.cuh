// z pass of the sub-lattice forms for the two class sets that crystals on the a/4 grid give:
// the 8 zinc-blende classes modulo 4 and a pair of classes modulo 2.
//
// One thread mixes all the classes of R2 frequencies in registers.  A class line of N = 2 H R2
// points, its upper half zero, is transformed as R1 = 2 H points (half of them zero) times R2:
//   phase A  (line, t < R2): loads x[t + R2 j], j < H, from HBM, R1-point DFT over j to q;
//   phase B  (column, q < R1): for every class, twiddles and the R2-point DFT over t (frequencies
//            k = q + R1 s); the classes mixed at each k; the R2-point inverse DFT over s and the
//            conjugate twiddles, back to the same shared-memory words (private to the thread);
//   phase A' (line, n1 < R2): R1-point inverse DFT over q, outputs z = n1 + R2 n2, n2 < H, to HBM.
// Against the pass that mixes through shared memory (k_zmix_rf: its own exchange each way between
// the stages and the mixing, five barriers a density) a point passes shared memory four times
// instead of eight and a density has three barriers.  The block runs several groups of warps, each
// on its own density with its own named barrier, over one copy of the mixing coefficients, so one
// group's barrier and HBM waits are covered by the others.
//
// The stored planes of a group's next density are copied to shared memory with 16-byte cp.async
// while the current one is transformed.
//
// Phases.  Class offsets enter as e^{-i pi k.b/n}.  Within a half (the fcc classes, or those at
// +(1,1,1)) the offsets differ by 0 or +-2 per axis, so relative to the half's class 0 the phases are
// 1, y z, x z, x y with x = e^{-+i pi kx/Px} and so on; class 0's own phase commutes with the
// Walsh-Hadamard mixing, so of the halves' two only the ratio is left: its z part is folded into beta,
// its x y part multiplies the second half's phases.  Everything that depends on the column alone is
// built in FP64 and rounded once (k_zw_columns).
//
// Frequencies above N/2.  The kernel spectrum is even along z, so the coefficients at N - kz are those
// at kz with the characters c and c ^ 3 exchanged, alpha as is and beta conjugated, negated for c = 1, 2
// (alpha_k and beta_k pick up (-i)^rz, rz the z offset of their residue, and beta_k turns into the
// conjugate of beta_{k^3}).  With an even R2 a thread's upper frequencies q + R1 r, r >= R2/2, then read
// the lower half of the table with the names exchanged at compile time: half the table, which is what
// lets two groups of 128-point lines and their staging share an SM.
//
// Bound: instruction issue (78 warp instructions a class point, 60 of them FP32, against 94 for
// k_zmix_rf) at the 16 warps an SM that 128 registers allow.  Measured on a B200, k_zmix_rf -> this
// pass: 128-point lines of the 2,097,152-atom box, 36 densities, 2.47 -> 1.83 ms (2.70 TB/s); 64-point
// lines, 820 densities, 6.93 -> 4.39 ms; 48-point, 78 densities, 0.309 -> 0.217 ms; two classes,
// 54 x 72 x 80 grid, 36 densities, 0.587 -> 0.070 ms (k_zmix_rf keeps 8 classes' threads whatever the
// set).  Without the staging (and with plain constants) 1.88, 5.24 and 0.228 ms on the three zinc-blende shapes.
//
// Error.  The rounding of an FP32 constant is the same in every line, so on smooth densities it adds up
// over the lines and axes: with every constant rounded as it is, integrals of Gaussians over 32 boxes of 12-
// to 128-point axes were off by 5.1e-8 (geometric mean of the root-mean-square error against FP64; k_zmix_rf and
// the whole-plane passes 3.7e-8).  Odd H without twiddles, coprime codelets without twiddles, and the constants of
// turn, dft3 and dft5 as +-1 plus a small part bring it to 2.3e-8, for 0.97 to 1.03 of the pass's time.
// In FP64 (4 columns a block, 256 threads an SM at 255 registers): 48-point lines, 78 densities, 0.571 ->
// 0.362 ms; 64-point, 36 densities, 0.679 -> 0.399; 54 x 72 x 80, two classes, 0.750 -> 0.111.
#pragma once

#include "fft.cuh"
#include "sublattice.cuh"

namespace clk {

// exp(2 pi i m / N), m < N / 2, as in fft.cuh (40-digit values from the Taylor series).
template <> struct WConst<8> {
    static __device__ __forceinline__ double c(int m) {
        switch (m) {
            case 0: return 1.0000000000000000000000000000000000000000;
            case 1: return 0.7071067811865475244008443621048490392848;
            case 2: return 0.0000000000000000000000000000000000000000;
            case 3: return -0.7071067811865475244008443621048490392848;
        }
        return 0.0;
    }
    static __device__ __forceinline__ double s(int m) {
        switch (m) {
            case 0: return 0.0000000000000000000000000000000000000000;
            case 1: return 0.7071067811865475244008443621048490392848;
            case 2: return 1.0000000000000000000000000000000000000000;
            case 3: return 0.7071067811865475244008443621048490392848;
        }
        return 0.0;
    }
};
template <> struct WConst<20> {
    static __device__ __forceinline__ double c(int m) {
        switch (m) {
            case 0: return 1.0000000000000000000000000000000000000000;
            case 1: return 0.9510565162951535721164393333793821434057;
            case 2: return 0.8090169943749474241022934171828190588602;
            case 3: return 0.5877852522924731291687059546390727685977;
            case 4: return 0.3090169943749474241022934171828190588602;
            case 5: return 0.0000000000000000000000000000000000000000;
            case 6: return -0.3090169943749474241022934171828190588602;
            case 7: return -0.5877852522924731291687059546390727685977;
            case 8: return -0.8090169943749474241022934171828190588602;
            case 9: return -0.9510565162951535721164393333793821434057;
        }
        return 0.0;
    }
    static __device__ __forceinline__ double s(int m) {
        switch (m) {
            case 0: return 0.0000000000000000000000000000000000000000;
            case 1: return 0.3090169943749474241022934171828190588602;
            case 2: return 0.5877852522924731291687059546390727685977;
            case 3: return 0.8090169943749474241022934171828190588602;
            case 4: return 0.9510565162951535721164393333793821434057;
            case 5: return 1.0000000000000000000000000000000000000000;
            case 6: return 0.9510565162951535721164393333793821434057;
            case 7: return 0.8090169943749474241022934171828190588602;
            case 8: return 0.5877852522924731291687059546390727685977;
            case 9: return 0.3090169943749474241022934171828190588602;
        }
        return 0.0;
    }
};
template <> struct WConst<24> {
    static __device__ __forceinline__ double c(int m) {
        switch (m) {
            case 0: return 1.0000000000000000000000000000000000000000;
            case 1: return 0.9659258262890682867497431997288973676339;
            case 2: return 0.8660254037844386467637231707529361834714;
            case 3: return 0.7071067811865475244008443621048490392848;
            case 4: return 0.5000000000000000000000000000000000000000;
            case 5: return 0.2588190451025207623488988376240483283491;
            case 6: return 0.0000000000000000000000000000000000000000;
            case 7: return -0.2588190451025207623488988376240483283491;
            case 8: return -0.5000000000000000000000000000000000000000;
            case 9: return -0.7071067811865475244008443621048490392848;
            case 10: return -0.8660254037844386467637231707529361834714;
            case 11: return -0.9659258262890682867497431997288973676339;
        }
        return 0.0;
    }
    static __device__ __forceinline__ double s(int m) {
        switch (m) {
            case 0: return 0.0000000000000000000000000000000000000000;
            case 1: return 0.2588190451025207623488988376240483283491;
            case 2: return 0.5000000000000000000000000000000000000000;
            case 3: return 0.7071067811865475244008443621048490392848;
            case 4: return 0.8660254037844386467637231707529361834714;
            case 5: return 0.9659258262890682867497431997288973676339;
            case 6: return 1.0000000000000000000000000000000000000000;
            case 7: return 0.9659258262890682867497431997288973676339;
            case 8: return 0.8660254037844386467637231707529361834714;
            case 9: return 0.7071067811865475244008443621048490392848;
            case 10: return 0.5000000000000000000000000000000000000000;
            case 11: return 0.2588190451025207623488988376240483283491;
        }
        return 0.0;
    }
};
template <> struct WConst<32> {
    static __device__ __forceinline__ double c(int m) {
        switch (m) {
            case 0: return 1.0000000000000000000000000000000000000000;
            case 1: return 0.9807852804032304491261822361342390369739;
            case 2: return 0.9238795325112867561281831893967882868224;
            case 3: return 0.8314696123025452370787883776179057567386;
            case 4: return 0.7071067811865475244008443621048490392848;
            case 5: return 0.5555702330196022247428308139485328743749;
            case 6: return 0.3826834323650897717284599840303988667613;
            case 7: return 0.1950903220161282678482848684770222409277;
            case 8: return 0.0000000000000000000000000000000000000000;
            case 9: return -0.1950903220161282678482848684770222409277;
            case 10: return -0.3826834323650897717284599840303988667613;
            case 11: return -0.5555702330196022247428308139485328743749;
            case 12: return -0.7071067811865475244008443621048490392848;
            case 13: return -0.8314696123025452370787883776179057567386;
            case 14: return -0.9238795325112867561281831893967882868224;
            case 15: return -0.9807852804032304491261822361342390369739;
        }
        return 0.0;
    }
    static __device__ __forceinline__ double s(int m) {
        switch (m) {
            case 0: return 0.0000000000000000000000000000000000000000;
            case 1: return 0.1950903220161282678482848684770222409277;
            case 2: return 0.3826834323650897717284599840303988667613;
            case 3: return 0.5555702330196022247428308139485328743749;
            case 4: return 0.7071067811865475244008443621048490392848;
            case 5: return 0.8314696123025452370787883776179057567386;
            case 6: return 0.9238795325112867561281831893967882868224;
            case 7: return 0.9807852804032304491261822361342390369739;
            case 8: return 1.0000000000000000000000000000000000000000;
            case 9: return 0.9807852804032304491261822361342390369739;
            case 10: return 0.9238795325112867561281831893967882868224;
            case 11: return 0.8314696123025452370787883776179057567386;
            case 12: return 0.7071067811865475244008443621048490392848;
            case 13: return 0.5555702330196022247428308139485328743749;
            case 14: return 0.3826834323650897717284599840303988667613;
            case 15: return 0.1950903220161282678482848684770222409277;
        }
        return 0.0;
    }
};
template <> struct WConst<36> {
    static __device__ __forceinline__ double c(int m) {
        switch (m) {
            case 0: return 1.0000000000000000000000000000000000000000;
            case 1: return 0.9848077530122080593667430245895230136706;
            case 2: return 0.9396926207859083840541092773247314699362;
            case 3: return 0.8660254037844386467637231707529361834714;
            case 4: return 0.7660444431189780352023926505554166739358;
            case 5: return 0.6427876096865393263226434099072634329076;
            case 6: return 0.5000000000000000000000000000000000000000;
            case 7: return 0.3420201433256687330440996146822595807631;
            case 8: return 0.1736481776669303488517166267693147960004;
            case 9: return 0.0000000000000000000000000000000000000000;
            case 10: return -0.1736481776669303488517166267693147960004;
            case 11: return -0.3420201433256687330440996146822595807631;
            case 12: return -0.5000000000000000000000000000000000000000;
            case 13: return -0.6427876096865393263226434099072634329076;
            case 14: return -0.7660444431189780352023926505554166739358;
            case 15: return -0.8660254037844386467637231707529361834714;
            case 16: return -0.9396926207859083840541092773247314699362;
            case 17: return -0.9848077530122080593667430245895230136706;
        }
        return 0.0;
    }
    static __device__ __forceinline__ double s(int m) {
        switch (m) {
            case 0: return 0.0000000000000000000000000000000000000000;
            case 1: return 0.1736481776669303488517166267693147960004;
            case 2: return 0.3420201433256687330440996146822595807631;
            case 3: return 0.5000000000000000000000000000000000000000;
            case 4: return 0.6427876096865393263226434099072634329076;
            case 5: return 0.7660444431189780352023926505554166739358;
            case 6: return 0.8660254037844386467637231707529361834714;
            case 7: return 0.9396926207859083840541092773247314699362;
            case 8: return 0.9848077530122080593667430245895230136706;
            case 9: return 1.0000000000000000000000000000000000000000;
            case 10: return 0.9848077530122080593667430245895230136706;
            case 11: return 0.9396926207859083840541092773247314699362;
            case 12: return 0.8660254037844386467637231707529361834714;
            case 13: return 0.7660444431189780352023926505554166739358;
            case 14: return 0.6427876096865393263226434099072634329076;
            case 15: return 0.5000000000000000000000000000000000000000;
            case 16: return 0.3420201433256687330440996146822595807631;
            case 17: return 0.1736481776669303488517166267693147960004;
        }
        return 0.0;
    }
};
// H-point DFTs used below: those of fft.cuh and 18 = 2 x 9.
template <int R, int S, typename T>
__device__ __forceinline__ void dft_h(cx<T>* v) {
    if constexpr (R == 18)
        dft_coprime<2, 9, S, true>(v);
    else
        dft<R, S, true>(v);
}

// e + x (c + i S s), c and s compile-time constants of a unit root; ADD false: without e.  In FP32 the larger of
// the two is multiplied as +-x + (c -+ 1) x, whose constant is rounded to a fraction of c's error, and
// sqrt(1/2) as 3/4 x - 0.0429 x (see FINE in fft.cuh).
template <int S, bool ADD, typename T>
__device__ __forceinline__ cx<T> turn(cx<T> e, cx<T> x, double c, double s) {
    const T zero = T(0);
    if (!ADD) e = mk(zero, zero);
    if (c == 0.0) return ADD ? e + mul_is<S>(x) : mul_is<S>(x);  // s = 1
    if (sizeof(T) == 8) {
        const cx<T> w = mk(T(c), T(S * s));
        return ADD ? mk(e.re + w.re * x.re - w.im * x.im, e.im + w.re * x.im + w.im * x.re) : cmul(x, w);
    }
    const T sc = T(c < 0.0 ? -1.0 : 1.0);
    if (c == s || c == -s) {
        const T hi = T(0.75), lo = T(s - 0.75);
        const T re = sc * x.re - S * x.im, im = sc * x.im + S * x.re;
        return ADD ? mk(e.re + hi * re + lo * re, e.im + hi * im + lo * im) : mk(hi * re + lo * re, hi * im + lo * im);
    }
    if (c > s || -c > s) {
        const T cr = T(c - (c < 0.0 ? -1.0 : 1.0)), si = T(S * s);
        const cx<T> u = ADD ? mk(e.re + sc * x.re, e.im + sc * x.im) : mk(sc * x.re, sc * x.im);
        return mk(u.re + cr * x.re - si * x.im, u.im + cr * x.im + si * x.re);
    }
    const T cr = T(c), si = T(S * (s - 1.0));
    const cx<T> u = ADD ? e + mul_is<S>(x) : mul_is<S>(x);
    return mk(u.re - si * x.im + cr * x.re, u.im + si * x.re + cr * x.im);
}

// 2H-point DFT of x[0..H) followed by H zeros: X[2k] = DFT_H(x)[k], X[2k+1] = DFT_H(x w_2H^j)[k].  For odd H
// the odd frequencies are 2m + H modulo 2H, where w_2H^(j (2m + H)) = w_H^(jm) (-1)^j: no twiddles.
template <int H, typename T>
__device__ __forceinline__ void dft_zero_padded(const cx<T>* x, cx<T>* even, cx<T>* odd) {
    if constexpr (H % 2 == 1) {
        cx<T> a[H];
#pragma unroll
        for (int j = 0; j < H; ++j) {
            even[j] = x[j];
            a[j] = j % 2 == 0 ? x[j] : mk(-x[j].re, -x[j].im);
        }
        dft_h<H, -1>(a);
#pragma unroll
        for (int m = 0; m < H; ++m) odd[(m + (H - 1) / 2) % H] = a[m];
    } else {
#pragma unroll
        for (int j = 0; j < H; ++j) {
            even[j] = x[j];
            odd[j] = j == 0 ? x[0] : turn<-1, false>(x[j], x[j], WConst<2 * H>::c(j), WConst<2 * H>::s(j));
        }
        dft_h<H, -1>(odd);
    }
    dft_h<H, -1>(even);
}

// Outputs 0..H-1 of the 2H-point inverse DFT of the interleaved (even, odd) inputs, into even.
template <int H, typename T>
__device__ __forceinline__ void idft_first_half(cx<T>* even, cx<T>* odd) {
    dft_h<H, +1>(even);
    if constexpr (H % 2 == 1) {
        cx<T> a[H];
#pragma unroll
        for (int m = 0; m < H; ++m) a[m] = odd[(m + (H - 1) / 2) % H];
        dft_h<H, +1>(a);
#pragma unroll
        for (int n = 0; n < H; ++n) even[n] = n % 2 == 0 ? even[n] + a[n] : even[n] - a[n];
    } else {
        dft_h<H, +1>(odd);
        even[0] = even[0] + odd[0];
#pragma unroll
        for (int n = 1; n < H; ++n) even[n] = turn<+1, true>(even[n], odd[n], WConst<2 * H>::c(n), WConst<2 * H>::s(n));
    }
}

// Class sets: kZwZb 8 zinc-blende classes modulo 4; kZwPair two classes modulo 2.
enum { kZwZb = 0, kZwPair = 1 };
// Four values of a (column, frequency): 16-byte pieces of the coefficient table.
template <typename T>
struct alignas(16) Quad {
    T x, y, z, w;
};
template <typename T, int SET>
struct ZwSet {
    static constexpr int S = SET == kZwZb ? 8 : 2;      // classes
    static constexpr int C = SET == kZwZb ? 3 : 1;      // quads of coefficients a (column, frequency)
    // columns per block: 64 contiguous bytes a plane and class (zinc-blende; with 32 bytes and twice the
    // groups a block, 36 densities of 128-point lines take 2.03 ms instead of 1.86), 128 (pair)
    static constexpr int L = (SET == kZwZb ? 64 : 128) / (int)sizeof(cx<T>);
};

template <typename T, int SET, int H, int R2>
struct ZwLayout {
    using Z = ZwSet<T, SET>;
    static constexpr int R1 = 2 * H, N = R1 * R2, L = Z::L, LL = Z::S * L;
    static constexpr bool SYM = SET == kZwZb && R2 % 2 == 0;  // coefficients at kz <= N/2 only
    static constexpr int K = SYM ? N / 2 + 1 : N;
    // Row pitch of one q: the lanes of phase B read 64 bytes of columns at consecutive q, so consecutive q
    // start half a 128-byte row apart (a pair's columns fill a row by themselves).
    static constexpr int QP = R2 * LL + (SET == kZwZb ? L : 0);
    static constexpr int NT = (L * R1 + 31) / 32 * 32;  // threads of a group
    static constexpr int NCOL = SET == kZwZb ? 7 : 0;   // column phases
    static constexpr int NPH = SET == kZwZb ? 2 * N : 0;  // z phases of the two halves
    static constexpr size_t table = sizeof(Quad<T>) * (size_t)Z::C * K * L;
    static constexpr size_t shared = table + sizeof(cx<T>) * (size_t)(N + NPH + NCOL * L);
    static constexpr size_t group = sizeof(cx<T>) * ((size_t)R1 * QP + (size_t)(N / 2) * LL);
    static constexpr size_t smem(int groups) { return shared + groups * group; }
    static constexpr int kThreads = sizeof(T) == 4 ? 512 : 256;  // resident threads at 128, 255 registers
    static constexpr int resident(int groups) {  // threads an SM holds with blocks of `groups`
        const int by_regs = kThreads / (NT * groups), by_smem = (int)(228 * 1024 / (smem(groups) + 1024));
        return smem(groups) > 227 * 1024 ? 0 : (by_regs < by_smem ? by_regs : by_smem) * NT * groups;
    }
    // Groups per block: the fewest that let an SM hold the most threads (a block's table is shared by
    // its groups, but a block ends only when its last group does).
    static constexpr int pick() {
        int best = 1;
        for (int g = 2; g <= 15 && g * NT <= kThreads; ++g)  // named barriers 1..15
            if (resident(g) > resident(best)) best = g;
        return best;
    }
    static constexpr int G = pick();
    static_assert(resident(G) > 0, "a block fits an SM");
};

__device__ __forceinline__ void group_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

// The mixing coefficients, packed for the kernel: tab[c][kz][ky][kx] quads with
//   zinc-blende   c = 0: alpha^_0..3 / 4;  c = 1, 2: beta'_0..1 / 4, beta'_2..3 / 4 (re, im)
//   pair          alpha (H_0), beta' (re, im), 0
// from the FP64 class kernels; beta' = beta e^{i pi k.delta/n}, delta = offset(class 0 of the second
// half) - offset(class 0 of the first), its z part only for zinc-blende.
struct ZwBuild {
    int src[8], cj[8];    // raw class kernels of alpha_0.., beta_0.. (conjugated where cj)
    int delta[3], n[3];   // offset difference, grid points per axis
    int p[3];             // transform lengths
    int sgn[2][3];        // +-1: half h's axis phase is e^{-+i pi k/P}
};
template <typename T, int SET>
__global__ void k_zw_table(const cx<double>* __restrict__ raw, ZwBuild b, Quad<T>* __restrict__ tab) {
    const long long nxy = (long long)b.p[0] * b.p[1], nq = nxy * b.p[2];
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < nq;
         q += (long long)gridDim.x * blockDim.x) {
        const int kx = (int)(q % b.p[0]), ky = (int)(q / b.p[0] % b.p[1]), kz = (int)(q / nxy);
        double turn = (double)(kz * b.delta[2]) / b.n[2];
        if (SET == kZwPair) turn += (double)(kx * b.delta[0]) / b.n[0] + (double)(ky * b.delta[1]) / b.n[1];
        cx<double> g;
        sincospi(turn, &g.im, &g.re);
        constexpr int K = SET == kZwZb ? 8 : 2;
        cx<double> v[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            v[k] = raw[b.src[k] * nq + q];
            if (b.cj[k]) v[k].im = -v[k].im;
        }
        if constexpr (SET == kZwZb) {
            cx<double> al[4], be[4];
            wht4(v, al);
            wht4(v + 4, be);
#pragma unroll
            for (int c = 0; c < 4; ++c) be[c] = scale(cmul(be[c], g), 0.25);
            tab[q] = Quad<T>{T(0.25 * al[0].re), T(0.25 * al[1].re), T(0.25 * al[2].re), T(0.25 * al[3].re)};
            tab[nq + q] = Quad<T>{T(be[0].re), T(be[0].im), T(be[1].re), T(be[1].im)};
            tab[2 * nq + q] = Quad<T>{T(be[2].re), T(be[2].im), T(be[3].re), T(be[3].im)};
        } else {
            const cx<double> be = cmul(v[1], g);
            tab[q] = Quad<T>{T(v[0].re), T(be.re), T(be.im), T(0)};
        }
    }
}

// Phases of the zinc-blende mixing that depend on the column, col[i][ky][kx]: x, y, x y of the first
// half; then with the halves' ratio e^{-i pi (kx dx/nx + ky dy/ny)} = r: r, r x, r y, r x y of the second.
// zph[h][kz]: the z phase of half h.
template <typename T>
__global__ void k_zw_columns(ZwBuild b, cx<T>* __restrict__ col, cx<T>* __restrict__ zph) {
    const int nxy = b.p[0] * b.p[1];
    const auto put = [](cx<T>* at, double turn) {
        double s, c;
        sincospi(-turn, &s, &c);
        *at = mk(T(c), T(s));
    };
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nxy; i += gridDim.x * blockDim.x) {
        const int kx = i % b.p[0], ky = i / b.p[0];
        const double x = (double)kx / b.p[0], y = (double)ky / b.p[1];
        const double r = (double)(kx * b.delta[0]) / b.n[0] + (double)(ky * b.delta[1]) / b.n[1];
        const double x0 = b.sgn[0][0] * x, y0 = b.sgn[0][1] * y, x1 = b.sgn[1][0] * x, y1 = b.sgn[1][1] * y;
        put(col + i, x0);
        put(col + nxy + i, y0);
        put(col + 2 * nxy + i, x0 + y0);
        put(col + 3 * nxy + i, r);
        put(col + 4 * nxy + i, r + x1);
        put(col + 5 * nxy + i, r + y1);
        put(col + 6 * nxy + i, r + x1 + y1);
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 2 * b.p[2]; i += gridDim.x * blockDim.x)
        put(zph + i, b.sgn[i / b.p[2]][2] * (double)(i % b.p[2]) / b.p[2]);
}

// Mixes the 8 zinc-blende classes u[0..7] of one frequency in place: phases (tf, to: those of classes
// 1-3 and 5-7; t4: class 4), the Walsh-Hadamard transforms of the halves, the alpha/beta step, and back
// (see sublattice.cuh).  UPPER: the coefficients are those of the mirrored frequency.
template <bool UPPER, typename T>
__device__ __forceinline__ void zw_mix_zb(cx<T>* const (&u)[8], const cx<T>* tf, const cx<T>* to,
                                          cx<T> t4, Quad<T> a, Quad<T> b01, Quad<T> b23) {
    cx<T> f[4] = {*u[0], cmul(*u[1], tf[0]), cmul(*u[2], tf[1]), cmul(*u[3], tf[2])};
    cx<T> o[4] = {cmul(*u[4], t4), cmul(*u[5], to[0]), cmul(*u[6], to[1]), cmul(*u[7], to[2])};
    cx<T> xf[4], xo[4];
    wht4(f, xf);
    wht4(o, xo);
    T al[4] = {a.x, a.y, a.z, a.w};
    cx<T> be[4] = {mk(b01.x, b01.y), mk(b01.z, b01.w), mk(b23.x, b23.y), mk(b23.z, b23.w)};
    if (UPPER) {
        const T t0 = al[0], t1 = al[1];
        al[0] = al[3];
        al[3] = t0;
        al[1] = al[2];
        al[2] = t1;
        const cx<T> s0 = be[0], s1 = be[1];
        be[0] = mk(be[3].re, -be[3].im);
        be[3] = mk(s0.re, -s0.im);
        be[1] = mk(-be[2].re, be[2].im);
        be[2] = mk(-s1.re, s1.im);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        f[c] = mk(al[c] * xf[c].re + be[c].re * xo[c].re + be[c].im * xo[c].im,
                  al[c] * xf[c].im + be[c].re * xo[c].im - be[c].im * xo[c].re);  // + conj(be) xo
        o[c] = mk(al[c] * xo[c].re + be[c].re * xf[c].re - be[c].im * xf[c].im,
                  al[c] * xo[c].im + be[c].re * xf[c].im + be[c].im * xf[c].re);  // + be xf
    }
    wht4(f, xf);
    wht4(o, xo);
    *u[0] = xf[0];
    *u[4] = cmulc(xo[0], t4);
#pragma unroll
    for (int c = 1; c < 4; ++c) {
        *u[c] = cmulc(xf[c], tf[c - 1]);
        *u[4 + c] = cmulc(xo[c], to[c - 1]);
    }
}

template <typename T, int SET, int H, int R2>
__global__ void __launch_bounds__(ZwLayout<T, SET, H, R2>::kThreads, 1)
    k_zw(cx<T>* __restrict__ buf, long long stride, const cx<T>* __restrict__ tw_g,
         const Quad<T>* __restrict__ tab, const cx<T>* __restrict__ col_g, const cx<T>* __restrict__ zph_g,
         long long nxy, int np) {
    using Lay = ZwLayout<T, SET, H, R2>;
    using Z = ZwSet<T, SET>;
    constexpr int R1 = Lay::R1, N = Lay::N, L = Lay::L, LL = Lay::LL, QP = Lay::QP, NT = Lay::NT, S = Z::S,
                  K = Lay::K, NCOL = Lay::NCOL, NPH = Lay::NPH;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int g = threadIdx.x / NT, tid = threadIdx.x - g * NT, groups = blockDim.x / NT;
    Quad<T>* tb = reinterpret_cast<Quad<T>*>(smem_raw);
    cx<T>* ST = reinterpret_cast<cx<T>*>(smem_raw + Lay::table) + (size_t)g * (N / 2) * LL;
    cx<T>* E = reinterpret_cast<cx<T>*>(smem_raw + Lay::table) + (size_t)groups * (N / 2) * LL +
                   (size_t)g * R1 * QP;
    cx<T>* tw = reinterpret_cast<cx<T>*>(smem_raw + Lay::table) +
                    (size_t)groups * ((N / 2) * LL + R1 * QP);
    cx<T>* zph = tw + N;
    cx<T>* colp = zph + NPH;
    const long long c0 = (long long)blockIdx.x * L;
    const int cols = (int)min((long long)L, nxy - c0);  // even: nxy is a multiple of 4
    const int per = (np + gridDim.y - 1) / gridDim.y;
    const int p_end = min(np, (int)(blockIdx.y + 1) * per);
    // stored planes of density p to ST[z][class][column], 16 bytes of columns a copy
    constexpr int W = 16 / (int)sizeof(cx<T>);
    const auto stage_in = [&](int p) {
        const cx<T>* src = buf + (long long)p * stride + c0;
        for (int i = tid; i < (N / 2) * LL / W; i += NT) {
            const int col = W * (i % (L / W)), r = i / (L / W), cls = r % S, z = r / S;
            if (col < cols)
                pd_cp_async16(ST + z * LL + cls * L + col, src + (long long)(cls * (N / 2) + z) * nxy + col);
        }
    };
    int p = blockIdx.y * per + g;
    if (p < p_end) stage_in(p);
    for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = tw_g[i];
    for (int i = threadIdx.x; i < NPH; i += blockDim.x) zph[i] = zph_g[i];
    for (int i = threadIdx.x; i < NCOL * L; i += blockDim.x)
        colp[i] = i % L < cols ? col_g[(long long)(i / L) * nxy + c0 + i % L] : mk(T(0), T(0));
    for (int i = threadIdx.x; i < Z::C * K * L; i += blockDim.x) {
        const int l = i % L, r = i / L, c = r / K, k = r - c * K;
        tb[i] = l < cols ? tab[((long long)c * N + k) * nxy + c0 + l] : Quad<T>{T(0), T(0), T(0), T(0)};
    }
    __syncthreads();
    for (; p < p_end; p += groups) {
        cx<T>* base = buf + (long long)p * stride + c0;
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        group_sync(1 + g, NT);  // ST has landed, and E is free (phase A' of the last density is over)
        // phase A
#pragma unroll 1
        for (int it = tid; it < LL * R2; it += NT) {
            const int line = it % LL, t = it / LL;
            cx<T> x[H], ev[H], od[H];
#pragma unroll
            for (int j = 0; j < H; ++j) x[j] = ST[(t + R2 * j) * LL + line];
            dft_zero_padded<H>(x, ev, od);
            cx<T>* e = E + t * LL + line;
#pragma unroll
            for (int k = 0; k < H; ++k) {
                e[(2 * k) * QP] = ev[k];
                e[(2 * k + 1) * QP] = od[k];
            }
        }
        group_sync(1 + g, NT);
        if (p + groups < p_end) stage_in(p + groups);
        // phase B
        if (tid < L * R1) {
            const int col = tid % L, q = tid / L;
            cx<T>* e = E + q * QP + col;
            cx<T> w[R2];
#pragma unroll
            for (int t = 1; t < R2; ++t) w[t] = tw[t * q];
            cx<T> x[S][R2];
#pragma unroll
            for (int s = 0; s < S; ++s) {
#pragma unroll
                for (int t = 0; t < R2; ++t) {
                    const cx<T> v = e[t * LL + s * L];
                    x[s][t] = t == 0 ? v : cmul(v, w[t]);
                }
                dft<R2, -1, true>(x[s]);
            }
            if constexpr (SET == kZwZb) {
#pragma unroll
                for (int r = 0; r < R2; ++r) {
                    const int k = q + R1 * r;
                    const bool upper = Lay::SYM && r >= R2 / 2;  // compile time
                    const int kt = upper ? N - k : k;
                    const cx<T> zf = zph[k], zo = zph[N + k];
                    const cx<T> tf[3] = {cmul(colp[L + col], zf), cmul(colp[col], zf), colp[2 * L + col]};
                    const cx<T> to[3] = {cmul(colp[5 * L + col], zo), cmul(colp[4 * L + col], zo), colp[6 * L + col]};
                    cx<T>* const u[8] = {&x[0][r], &x[1][r], &x[2][r], &x[3][r],
                                             &x[4][r], &x[5][r], &x[6][r], &x[7][r]};
                    const Quad<T> a = tb[kt * L + col], b01 = tb[(K + kt) * L + col], b23 = tb[(2 * K + kt) * L + col];
                    if (upper)
                        zw_mix_zb<true>(u, tf, to, colp[3 * L + col], a, b01, b23);
                    else
                        zw_mix_zb<false>(u, tf, to, colp[3 * L + col], a, b01, b23);
                }
            } else {
#pragma unroll
                for (int r = 0; r < R2; ++r) {
                    const Quad<T> h = tb[(q + R1 * r) * L + col];
                    const cx<T> a = x[0][r], b = x[1][r];
                    x[0][r] = mk(h.x * a.re + h.y * b.re + h.z * b.im, h.x * a.im + h.y * b.im - h.z * b.re);
                    x[1][r] = mk(h.x * b.re + h.y * a.re - h.z * a.im, h.x * b.im + h.y * a.im + h.z * a.re);
                }
            }
#pragma unroll
            for (int s = 0; s < S; ++s) {
                dft<R2, +1, true>(x[s]);
#pragma unroll
                for (int t = 0; t < R2; ++t) e[t * LL + s * L] = t == 0 ? x[s][0] : cmulc(x[s][t], w[t]);
            }
        }
        group_sync(1 + g, NT);
        // phase A'
#pragma unroll 1
        for (int it = tid; it < LL * R2; it += NT) {
            const int line = it % LL, t = it / LL;
            const int cls = line / L, col = line % L;
            const cx<T>* e = E + t * LL + line;
            cx<T> ev[H], od[H];
#pragma unroll
            for (int k = 0; k < H; ++k) {
                ev[k] = e[(2 * k) * QP];
                od[k] = e[(2 * k + 1) * QP];
            }
            idft_first_half<H>(ev, od);
            if (col < cols) {
                cx<T>* dst = base + (long long)(cls * (N / 2) + t) * nxy + col;
#pragma unroll
                for (int n = 0; n < H; ++n) dst[(long long)(R2 * n) * nxy] = ev[n];
            }
        }
    }
}

// The pass's split N = 2 H R2 of a length; f is called with (H, R2) as SplitTag<H, R2>.
template <int SET, typename F>
bool with_zw_split(int n, F&& f) {
    if constexpr (SET == kZwZb) {
        switch (n) {
#define CLK_ZW(N, A, B)      \
    case N:                  \
        f(SplitTag<A, B>{}); \
        return true;
            CLK_ZW(12, 3, 2)
            CLK_ZW(16, 4, 2)
            CLK_ZW(18, 3, 3)
            CLK_ZW(20, 5, 2)
            CLK_ZW(24, 4, 3)
            CLK_ZW(30, 5, 3)
            CLK_ZW(32, 4, 4)
            CLK_ZW(36, 6, 3)
            CLK_ZW(40, 5, 4)
            CLK_ZW(48, 8, 3)
            CLK_ZW(50, 5, 5)
            CLK_ZW(54, 9, 3)
            CLK_ZW(60, 10, 3)
            CLK_ZW(64, 8, 4)
            CLK_ZW(72, 9, 4)
            CLK_ZW(80, 10, 4)
            CLK_ZW(90, 15, 3)
            CLK_ZW(96, 16, 3)
            CLK_ZW(100, 10, 5)
            CLK_ZW(108, 18, 3)
            CLK_ZW(120, 15, 4)
            CLK_ZW(128, 16, 4)
            default: return false;
        }
    } else {
        switch (n) {
            CLK_ZW(18, 3, 3)
            CLK_ZW(20, 5, 2)
            CLK_ZW(24, 4, 3)
            CLK_ZW(30, 5, 3)
            CLK_ZW(32, 4, 4)
            CLK_ZW(36, 6, 3)
            CLK_ZW(40, 5, 4)
            CLK_ZW(48, 8, 3)
            CLK_ZW(50, 5, 5)
            CLK_ZW(54, 9, 3)
            CLK_ZW(60, 6, 5)
            CLK_ZW(64, 8, 4)
            CLK_ZW(72, 9, 4)
            CLK_ZW(80, 8, 5)
            CLK_ZW(90, 9, 5)
            CLK_ZW(96, 8, 6)
            CLK_ZW(100, 10, 5)
            CLK_ZW(108, 9, 6)
            CLK_ZW(120, 12, 5)
            CLK_ZW(128, 8, 8)
            CLK_ZW(144, 9, 8)
            CLK_ZW(150, 15, 5)
            CLK_ZW(160, 10, 8)
            CLK_ZW(180, 15, 6)
            CLK_ZW(192, 12, 8)
            CLK_ZW(240, 15, 8)
            CLK_ZW(256, 16, 8)
#undef CLK_ZW
            default: return false;
        }
    }
}

}  // namespace clk
