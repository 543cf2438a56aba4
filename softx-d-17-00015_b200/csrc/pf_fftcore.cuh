// Row transforms with the length known at compile time: every radix and all
// index arithmetic are constants, and each butterfly lives in registers.
//
// tw[t] = exp(+2 pi i t / L).  SIGN=+1 is FFTW's unnormalised backward
// transform, SIGN=-1 the forward one.
#pragma once
#include <cuda_runtime.h>

template <typename C> struct CTraits;
template <> struct CTraits<double2> {
    using R = double;
    static __device__ __forceinline__ double2 make(double x, double y) { return make_double2(x, y); }
};
template <> struct CTraits<float2> {
    using R = float;
    static __device__ __forceinline__ float2 make(float x, float y) { return make_float2(x, y); }
};

template <typename C> __device__ __forceinline__ C c_add(C a, C b) { return CTraits<C>::make(a.x + b.x, a.y + b.y); }
template <typename C> __device__ __forceinline__ C c_sub(C a, C b) { return CTraits<C>::make(a.x - b.x, a.y - b.y); }
// fixed contraction, so a product rounds alike in every kernel and with
// twiddles from tables or constants
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
template <typename C> __device__ __forceinline__ C c_mul(C a, C b) {
    return CTraits<C>::make(fma(a.x, b.x, -mul_rn(a.y, b.y)), fma(a.y, b.x, mul_rn(a.x, b.y)));
}
// a * (SIGN * i)
template <int SIGN, typename C> __device__ __forceinline__ C c_muli(C a) {
    return SIGN > 0 ? CTraits<C>::make(-a.y, a.x) : CTraits<C>::make(a.y, -a.x);
}
template <int SIGN, typename C> __device__ __forceinline__ C c_tw(C w) {
    return SIGN > 0 ? w : CTraits<C>::make(w.x, -w.y);
}

// cos(2 pi k/720), k = 0 .. 180, correctly rounded: the roots of unity of
// every codelet length (divisors of 720) as compile-time constants.  Read from
// the shared-memory twiddle table instead, each cost a load, and the trivial
// ones (1, i, (1+i)/sqrt 2) a full complex product.
static __device__ constexpr double kCos720[181] = {
    1.0, 0.9999619230641713, 0.9998476951563913, 0.9996573249755573,
    0.9993908270190958, 0.9990482215818578, 0.9986295347545738, 0.9981347984218669,
    0.9975640502598242, 0.996917333733128, 0.9961946980917455, 0.9953961983671789,
    0.9945218953682733, 0.9935718556765875, 0.992546151641322, 0.9914448613738104,
    0.9902680687415704, 0.9890158633619168, 0.9876883405951378, 0.9862856015372314,
    0.984807753012208, 0.9832549075639546, 0.981627183447664, 0.9799247046208296,
    0.9781476007338057, 0.9762960071199334, 0.9743700647852352, 0.9723699203976766,
    0.9702957262759965, 0.9681476403781077, 0.9659258262890683, 0.963630453208623,
    0.9612616959383189, 0.958819734868193, 0.9563047559630354, 0.9537169507482269,
    0.9510565162951535, 0.9483236552061993, 0.9455185755993168, 0.9426414910921784,
    0.9396926207859084, 0.9366721892483976, 0.9335804264972017, 0.9304175679820246,
    0.9271838545667874, 0.9238795325112867, 0.9205048534524404, 0.917060074385124,
    0.9135454576426009, 0.9099612708765432, 0.9063077870366499, 0.9025852843498606,
    0.898794046299167, 0.8949343616020251, 0.8910065241883679, 0.8870108331782217,
    0.882947592858927, 0.8788171126619654, 0.8746197071393959, 0.8703556959398997,
    0.8660254037844386, 0.8616291604415257, 0.8571673007021123, 0.8526401643540922,
    0.848048096156426, 0.8433914458128857, 0.838670567945424, 0.8338858220671682,
    0.8290375725550417, 0.8241261886220157, 0.8191520442889918, 0.8141155183563192,
    0.8090169943749475, 0.8038568606172173, 0.7986355100472928, 0.7933533402912352,
    0.7880107536067219, 0.7826081568524139, 0.7771459614569709, 0.77162458338772,
    0.766044443118978, 0.7604059656000309, 0.754709580222772, 0.7489557207890022,
    0.7431448254773942, 0.7372773368101241, 0.7313537016191705, 0.7253743710122876,
    0.7193398003386512, 0.7132504491541816, 0.7071067811865476, 0.7009092642998509,
    0.6946583704589973, 0.688354575693754, 0.6819983600624985, 0.6755902076156602,
    0.6691306063588582, 0.6626200482157375, 0.6560590289905073, 0.6494480483301837,
    0.6427876096865394, 0.636078220277764, 0.6293203910498375, 0.6225146366376195,
    0.6156614753256583, 0.6087614290087207, 0.6018150231520483, 0.5948227867513413,
    0.5877852522924731, 0.5807029557109398, 0.573576436351046, 0.5664062369248328,
    0.5591929034707468, 0.5519369853120581, 0.5446390350150271, 0.5372996083468239,
    0.5299192642332049, 0.5224985647159489, 0.5150380749100542, 0.5075383629607042,
    0.5, 0.4924235601034671, 0.484809620246337, 0.4771587602596084,
    0.46947156278589075, 0.4617486132350339, 0.4539904997395468, 0.44619781310980877,
    0.4383711467890774, 0.43051109680829514, 0.42261826174069944, 0.414693242656239,
    0.4067366430758002, 0.3987490689252462, 0.39073112848927377, 0.3826834323650898,
    0.374606593415912, 0.3665012267242973, 0.35836794954530027, 0.3502073812594675,
    0.3420201433256687, 0.3338068592337709, 0.32556815445715664, 0.31730465640509214,
    0.30901699437494745, 0.3007057995042731, 0.2923717047227367, 0.2840153447039226,
    0.27563735581699916, 0.2672383760782569, 0.25881904510252074, 0.25038000405444144,
    0.24192189559966773, 0.23344536385590542, 0.224951054343865, 0.21643961393810288,
    0.20791169081775934, 0.1993679344171972, 0.1908089953765448, 0.18223552549214744,
    0.17364817766693036, 0.16504760586067765, 0.15643446504023087, 0.14780941112961063,
    0.13917310096006544, 0.1305261922200516, 0.12186934340514748, 0.11320321376790672,
    0.10452846326765347, 0.095845752520224, 0.08715574274765818, 0.07845909572784494,
    0.0697564737441253, 0.06104853953485687, 0.052335956242943835, 0.043619387365336,
    0.03489949670250097, 0.026176948307873153, 0.01745240643728351, 0.008726535498373935,
    0.0,
};
// cos and sin of 2 pi e/R, e >= 0, R a divisor of 720
__device__ __forceinline__ constexpr double cos_720(int t) {
    t %= 720;
    if (t > 360) t = 720 - t;
    return t <= 180 ? kCos720[t] : -kCos720[360 - t];
}
__device__ __forceinline__ constexpr double cos_root(int e, int R) { return cos_720(e * (720 / R)); }
__device__ __forceinline__ constexpr double sin_root(int e, int R) { return cos_720(e * (720 / R) + 540); }
// a times exp(SIGN 2 pi i e/R); e and R are constants once the caller's loops
// are unrolled
template <int SIGN, typename C> __device__ __forceinline__ C c_root(C a, int e, int R) {
    using T = typename CTraits<C>::R;
    e %= R;
    if (e == 0) return a;
    if (2 * e == R) return CTraits<C>::make(-a.x, -a.y);
    if (4 * e == R) return c_muli<SIGN>(a);
    if (4 * e == 3 * R) return c_muli<-SIGN>(a);
    const T c = (T)cos_root(e, R), s = SIGN > 0 ? (T)sin_root(e, R) : (T)-sin_root(e, R);
    return c_mul(a, CTraits<C>::make(c, s));
}

__host__ __device__ constexpr int fft_first_radix(int L) {
    return L % 4 == 0 ? 4 : L % 2 == 0 ? 2 : L % 3 == 0 ? 3 : L % 5 == 0 ? 5 : L % 7 == 0 ? 7 : L;
}
template <int R, int SIGN, typename C>
__device__ __forceinline__ void fft_dft(C (&v)[R]) {
    if constexpr (R == 2) {
        const C a = v[0];
        v[0] = c_add(a, v[1]);
        v[1] = c_sub(a, v[1]);
    } else if constexpr (R == 4) {
        const C a = c_add(v[0], v[2]), b = c_sub(v[0], v[2]);
        const C c = c_add(v[1], v[3]), d = c_muli<SIGN>(c_sub(v[1], v[3]));
        v[0] = c_add(a, c);
        v[1] = c_add(b, d);
        v[2] = c_sub(a, c);
        v[3] = c_sub(b, d);
    } else if constexpr (R == 3) {
        using T = typename CTraits<C>::R;
        const T s3 = (T)0.86602540378443864676;  // sin(2 pi / 3)
        const C t = c_add(v[1], v[2]);
        const C u = CTraits<C>::make(v[0].x - (T)0.5 * t.x, v[0].y - (T)0.5 * t.y);
        const C w = c_muli<SIGN>(CTraits<C>::make(s3 * (v[1].x - v[2].x), s3 * (v[1].y - v[2].y)));
        v[0] = c_add(v[0], t);
        v[1] = c_add(u, w);
        v[2] = c_sub(u, w);
    } else {  // small prime: direct DFT
        C o[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            C acc = v[0];
#pragma unroll
            for (int p = 1; p < R; ++p) acc = c_add(acc, c_root<SIGN>(v[p], p * q, R));
            o[q] = acc;
        }
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = o[q];
    }
}

// ---------------------------------------------------------------------------
// Register codelets and the four-step transform.
//
// rfft_run<R>: an R-point FFT (R <= 32) of v[R] held in registers; every index
// is a compile-time constant so nothing spills to local memory, and so are
// the internal twiddles W_R^e.
template <int R, int REM, int NS, int SIGN, typename C>
__device__ __forceinline__ void rfft_stage(const C (&src)[R], C (&dst)[R]) {
    constexpr int RR = fft_first_radix(REM);
    constexpr int NB = R / RR;
    constexpr int STRIDE = R / (NS * RR);
#pragma unroll
    for (int j = 0; j < NB; ++j) {
        const int k = j % NS;
        C v[RR];
#pragma unroll
        for (int q = 0; q < RR; ++q) {
            C x = src[j + q * NB];
            if (NS > 1 && q > 0 && k > 0) x = c_root<SIGN>(x, q * k * STRIDE, R);
            v[q] = x;
        }
        fft_dft<RR, SIGN>(v);
        const int base = (j / NS) * NS * RR + k;
#pragma unroll
        for (int q = 0; q < RR; ++q) dst[base + q * NS] = v[q];
    }
}

template <int R, int REM, int NS, int SIGN, typename C>
__device__ __forceinline__ void rfft_run(C (&a)[R]) {
    if constexpr (REM > 1) {
        constexpr int RR = fft_first_radix(REM);
        C b[R];
        rfft_stage<R, REM, NS, SIGN>(a, b);
#pragma unroll
        for (int i = 0; i < R; ++i) a[i] = b[i];
        rfft_run<R, REM / RR, NS * RR, SIGN>(a);
    }
}

// L = L1 * L2 with both factors <= 32 and L1 as close to sqrt(L) as allowed
__host__ __device__ constexpr int fft4_l1(int L) {
    if (L <= 32) return L;
    int best = 0;
    for (int d = 1; d <= 32; ++d)
        if (L % d == 0 && L / d <= 32 && (best == 0 || (d * d <= L && d > best) || (best * best > L && d < best)))
            best = d;
    return best;
}
// padded row pitch of the transposed intermediate (odd, so 16-byte accesses
// of consecutive threads fall in distinct bank groups)
__host__ __device__ constexpr int fft4_yp(int L1) { return (L1 % 2 == 0) ? L1 + 1 : L1 + 2; }
// elements one row occupies in shared memory
__host__ __device__ constexpr int fft4_pitch(int L) {
    return fft4_l1(L) == L ? L : ((L / fft4_l1(L)) * fft4_yp(fft4_l1(L)) > L ? (L / fft4_l1(L)) * fft4_yp(fft4_l1(L)) : L);
}

// The split of the z passes.  FP64: always two codelets, so that a row's short
// transform is still shared by several threads; in FP32 lengths up to 32 keep
// their one codelet, whose roundings the results are held to.
template <typename C> __host__ __device__ constexpr int fftz_l1(int L) {
    if (L > 32 || sizeof(C) == 8) return fft4_l1(L);
    int best = 1;
    for (int d = 1; d * d <= L; ++d)
        if (L % d == 0) best = d;
    return best;
}
__host__ __device__ constexpr int fft_pitch_of(int L, int L1) {
    return (L / L1) * fft4_yp(L1) > L ? (L / L1) * fft4_yp(L1) : L;
}

// In-place FFT of B rows (row r at rows + r*RS, natural order in and out).
// tw2[k1*L2 + n2] = W_L^(n2*k1) (the four-step twiddles, laid out so
// consecutive threads read consecutive entries).
// All threads of the block must call it; it synchronises internally.
template <int L, int SIGN, typename C>
__device__ __forceinline__ void fft4_rows(C *rows, int B, int RS, const C *tw2) {
    constexpr int L1 = fft4_l1(L);
    constexpr int L2 = L / L1;
    if constexpr (L2 == 1) {
        for (int b = threadIdx.x; b < B; b += blockDim.x) {
            C v[L];
#pragma unroll
            for (int i = 0; i < L; ++i) v[i] = rows[b * RS + i];
            rfft_run<L, L, 1, SIGN>(v);
#pragma unroll
            for (int i = 0; i < L; ++i) rows[b * RS + i] = v[i];
        }
        __syncthreads();
    } else {
        constexpr int YP = fft4_yp(L1);
        // each pass of these loops covers whole rows, because a row is read
        // in one layout and rewritten in the other (blockDim.x >= 32 >= L1, L2)
        const int rp1 = blockDim.x / L2;
        // step 1: L1-point transforms over n1 of x[L2*n1 + n2], twiddle, transpose
        for (int b0 = 0; b0 < B; b0 += rp1) {
            const int b = b0 + (int)threadIdx.x / L2, n2 = (int)threadIdx.x % L2;
            const bool act = (int)threadIdx.x < rp1 * L2 && b < B;
            C v[L1];
            if (act) {
#pragma unroll
                for (int i = 0; i < L1; ++i) v[i] = rows[b * RS + L2 * i + n2];
            }
            __syncthreads();
            if (act) {
                rfft_run<L1, L1, 1, SIGN>(v);
#pragma unroll
                for (int k1 = 0; k1 < L1; ++k1) {
                    C w = v[k1];
                    if (k1 > 0 && n2 > 0) w = c_mul(w, c_tw<SIGN>(tw2[k1 * L2 + n2]));
                    rows[b * RS + n2 * YP + k1] = w;
                }
            }
        }
        __syncthreads();
        // step 2: L2-point transforms over n2, output X[k1 + L1*k2]
        const int rp2 = blockDim.x / L1;
        for (int b0 = 0; b0 < B; b0 += rp2) {
            const int b = b0 + (int)threadIdx.x / L1, k1 = (int)threadIdx.x % L1;
            const bool act = (int)threadIdx.x < rp2 * L1 && b < B;
            C v[L2];
            if (act) {
#pragma unroll
                for (int i = 0; i < L2; ++i) v[i] = rows[b * RS + i * YP + k1];
            }
            __syncthreads();
            if (act) {
                rfft_run<L2, L2, 1, SIGN>(v);
#pragma unroll
                for (int k2 = 0; k2 < L2; ++k2) rows[b * RS + k1 + L1 * k2] = v[k2];
            }
        }
        __syncthreads();
    }
}

// Fill the tables a four-step transform of length L needs (in shared memory).
template <int L, typename C>
__device__ __forceinline__ void fft4_tables(C *tw, C *tw2, const C *__restrict__ gtw) {
    constexpr int L1 = fft4_l1(L);
    constexpr int L2 = L / L1;
    for (int i = threadIdx.x; i < L; i += blockDim.x) tw[i] = gtw[i];
    for (int i = threadIdx.x; i < L; i += blockDim.x) {
        const int k1 = i / L2, n2 = i - k1 * L2;
        tw2[i] = gtw[(k1 * n2) % L];
    }
}

// ---------------------------------------------------------------------------
// Stockham passes of radix 8 or 6 where the length allows (else 4, 2, 3, 5,
// 7), each butterfly an in-register codelet (rfft_run): a length-384 row takes
// three passes (8, 8, 6) instead of five (4, 4, 4, 2, 3), so three barriers
// and shared-memory round trips instead of five.  B rows of length L sit
// contiguously in `src`, `dst` is the ping-pong buffer; the pass with radix R
// maps butterfly j (k = j mod NS) to outputs (j/NS)*NS*R + k + q*NS after
// twiddling input q by W^(SIGN q k L/(NS R)).
__host__ __device__ constexpr int fft_big_radix(int L) {
    return L % 8 == 0 ? 8 : L % 6 == 0 ? 6 : fft_first_radix(L);
}

template <int L, int R, int NS, int SIGN, typename C>
__device__ __forceinline__ void fft_pass_big(const C *__restrict__ src, C *__restrict__ dst, int B, const C *tw) {
    constexpr int NB = L / R;
    constexpr int STRIDE = L / (NS * R);
    for (int idx = threadIdx.x; idx < NB * B; idx += blockDim.x) {
        const int b = idx / NB, j = idx - b * NB;
        const int k = j % NS;
        const C *sp = src + b * L;
        C *dp = dst + b * L;
        C v[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            C x = sp[j + q * NB];
            if (NS > 1 && q > 0) x = c_mul(x, c_tw<SIGN>(tw[q * k * STRIDE]));
            v[q] = x;
        }
        if constexpr (R == 8 || R == 6) rfft_run<R, R, 1, SIGN>(v);
        else fft_dft<R, SIGN>(v);
        const int base = (j / NS) * NS * R + k;
#pragma unroll
        for (int q = 0; q < R; ++q) dp[base + q * NS] = v[q];
    }
}

template <int L, int REM, int NS, int SIGN, typename C>
__device__ __forceinline__ C *fft_run_big(C *src, C *dst, int B, const C *tw) {
    if constexpr (REM == 1) {
        return src;
    } else {
        constexpr int R = fft_big_radix(REM);
        fft_pass_big<L, R, NS, SIGN>(src, dst, B, tw);
        __syncthreads();
        return fft_run_big<L, REM / R, NS * R, SIGN>(dst, src, B, tw);
    }
}

// ---------------------------------------------------------------------------
// Per-length choice between the four-step transform (one shared-memory
// transpose, codelets in registers) and the multi-pass Stockham transform
// (a ping-pong buffer of B*L, radix-8/6 register codelets, low register use).  FP64 lengths above 192
// need ~165 registers per thread in the four-step form, which caps occupancy
// at one 256-thread block per SM; they use Stockham.
template <int L, typename C> struct FFTRows {
    static constexpr bool four = (sizeof(C) == 8) || (L <= 192);
    static constexpr int pitch = four ? fft4_pitch(L) : L;
    // shared-memory elements for B rows plus the two tables
    static __host__ __device__ constexpr int smem_elems(int B) { return (four ? B * pitch : 2 * B * L) + 2 * L; }
    // rows at `rows` (B rows, pitch `pitch`); `scratch` = rows + B*pitch
    template <int SIGN>
    static __device__ __forceinline__ void run(C *rows, int B, const C *tw, const C *tw2) {
        if constexpr (four) {
            fft4_rows<L, SIGN>(rows, B, pitch, tw2);
        } else {
            C *res = fft_run_big<L, L, 1, SIGN>(rows, rows + B * L, B, tw);
            if (res != rows) {
                for (int i = threadIdx.x; i < B * L; i += blockDim.x) rows[i] = res[i];
                __syncthreads();
            }
        }
    }
};

// ---------------------------------------------------------------------------
// The transform of B rows between a source and a destination outside shared
// memory: ld(b, j) gives element j of row b to the first codelet in registers
// (it must not branch around its load, or the codelet's loads wait for one
// another), st(b, j, step, v) takes the last codelet's elements j + step*q =
// v[q], and only what passes between the
// codelets goes through shared memory: once for the four-step lengths (one
// barrier), twice for the three-pass Stockham ones.  Staged whole through
// shared memory on both sides, the z passes were bound by it (73% of its
// bandwidth at FP64 length 384, with the first Stockham pass's stores, 128
// bytes apart, eight to a bank): rows are now padded by one in eight.
template <int L, typename C> struct RowsIO {
    static constexpr bool four = FFTRows<L, C>::four;
    static constexpr int L1 = fftz_l1<C>(L), L2 = L / L1;
    static constexpr int pitch = !four ? L + L / 8 : L2 > 1 ? fft_pitch_of(L, L1) : 0;
    // shared-memory elements for B rows and the table
    static __host__ __device__ constexpr int smem_elems(int B) { return (four ? B * pitch : 2 * B * pitch) + L; }
    // the table of this length in shared memory (a barrier follows in run)
    static __device__ __forceinline__ void table(C *tw, const C *__restrict__ gtw) {
        for (int i = threadIdx.x; i < L; i += blockDim.x) {
            if constexpr (four) tw[i] = gtw[(i / L2) * (i % L2)];
            else tw[i] = gtw[i];
        }
    }
    static __device__ __forceinline__ int pad(int i) { return i + i / 8; }

    template <int SIGN, typename Ld, typename St>
    static __device__ __forceinline__ void run(C *sm, int B, const C *tw, Ld ld, St st) {
        if constexpr (four && L2 == 1) {
            for (int b = threadIdx.x; b < B; b += blockDim.x) {
                C v[L];
#pragma unroll
                for (int i = 0; i < L; ++i) v[i] = ld(b, i);
                rfft_run<L, L, 1, SIGN>(v);
                st(b, 0, 1, v);
            }
        } else if constexpr (four) {
            constexpr int YP = fft4_yp(L1);
            __syncthreads();  // the table
            const int rp1 = blockDim.x / L2, n2 = (int)threadIdx.x % L2;
            if ((int)threadIdx.x < rp1 * L2)
                for (int b = (int)threadIdx.x / L2; b < B; b += rp1) {
                    C v[L1];
#pragma unroll
                    for (int i = 0; i < L1; ++i) v[i] = ld(b, L2 * i + n2);
                    rfft_run<L1, L1, 1, SIGN>(v);
#pragma unroll
                    for (int k1 = 0; k1 < L1; ++k1) {
                        C w = v[k1];
                        if (k1 > 0 && n2 > 0) w = c_mul(w, c_tw<SIGN>(tw[k1 * L2 + n2]));
                        sm[b * pitch + n2 * YP + k1] = w;
                    }
                }
            __syncthreads();
            const int rp2 = blockDim.x / L1, k1 = (int)threadIdx.x % L1;
            if ((int)threadIdx.x < rp2 * L1)
                for (int b = (int)threadIdx.x / L1; b < B; b += rp2) {
                    C v[L2];
#pragma unroll
                    for (int i = 0; i < L2; ++i) v[i] = sm[b * pitch + i * YP + k1];
                    rfft_run<L2, L2, 1, SIGN>(v);
                    st(b, k1, L1, v);
                }
        } else {
            constexpr int R1 = fft_big_radix(L), R2 = fft_big_radix(L / R1), R3 = L / R1 / R2;
            static_assert(R3 <= 8 && (R3 == 8 || R3 == 6 || R3 <= 4), "three passes");
            C *s1 = sm, *s2 = sm + B * pitch;
            for (int idx = threadIdx.x; idx < L / R1 * B; idx += blockDim.x) {
                const int b = idx / (L / R1), j = idx - b * (L / R1);
                C v[R1];
#pragma unroll
                for (int q = 0; q < R1; ++q) v[q] = ld(b, j + q * (L / R1));
                rfft_run<R1, R1, 1, SIGN>(v);
#pragma unroll
                for (int q = 0; q < R1; ++q) s1[b * pitch + pad(j * R1 + q)] = v[q];
            }
            __syncthreads();
            for (int idx = threadIdx.x; idx < L / R2 * B; idx += blockDim.x) {
                const int b = idx / (L / R2), j = idx - b * (L / R2), k = j % R1;
                C v[R2];
#pragma unroll
                for (int q = 0; q < R2; ++q) {
                    v[q] = s1[b * pitch + pad(j + q * (L / R2))];
                    if (q > 0) v[q] = c_mul(v[q], c_tw<SIGN>(tw[q * k * R3]));
                }
                rfft_run<R2, R2, 1, SIGN>(v);
                const int base = (j / R1) * R1 * R2 + k;
#pragma unroll
                for (int q = 0; q < R2; ++q) s2[b * pitch + pad(base + q * R1)] = v[q];
            }
            __syncthreads();
            for (int idx = threadIdx.x; idx < L / R3 * B; idx += blockDim.x) {
                const int b = idx / (L / R3), j = idx - b * (L / R3);  // j < R1*R2: one block of the last pass
                C v[R3];
#pragma unroll
                for (int q = 0; q < R3; ++q) {
                    v[q] = s2[b * pitch + pad(j + q * (L / R3))];
                    if (q > 0) v[q] = c_mul(v[q], c_tw<SIGN>(tw[q * j]));
                }
                rfft_run<R3, R3, 1, SIGN>(v);
                st(b, j, L / R3, v);
            }
        }
    }
};
