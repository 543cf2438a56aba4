// 3/2-dealiased Fourier transforms between spectral (coll) and physical space
// (transform.fftw3.f90:35-147) as batched mixed-radix Stockham FFTs staged
// through shared memory:
//   coll -> phys : z pass  (c2c length 3K, sign +1) over the M columns of each
//                  radial point, Hermitian fill of m=0 (transform.fftw3.f90:72-74);
//                  theta pass (c2r length 3M; two real rows packed per complex FFT)
//   phys -> coll : theta pass (r2c, scaled by 1/(9KM)), z pass (c2c, sign -1),
//                  truncation to |k|<K, m<M.
// FFTW's sign conventions are kept: +1 is the unnormalised backward transform;
// the c2r transform ignores the imaginary part of the theta DC bin.
#include <algorithm>
#include <cmath>
#include "pf_internal.cuh"
#include "pf_fftcore.cuh"

static constexpr int FFT_THREADS = 256;

// the lengths 3K, 3M whose row transforms are compiled (codelets in registers);
// others take the mixed-radix passes of smem_fft
#define PF_FFT_LENGTHS(X) X(12) X(15) X(18) X(24) X(36) X(48) X(72) X(96) X(144) X(192) X(288) X(384)

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// multiply by sign*i
__device__ __forceinline__ double2 cmuli(double2 a, int sign) {
    return sign > 0 ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

// An R-point transform of v in registers.  w[p] = exp(2 pi i p/R), 1 <= p <=
// (R-1)/2, for the odd radices above 3, whose outputs q and R-q share the
// real sums of v[p] + v[R-p] and v[p] - v[R-p].
template <int R> __device__ __forceinline__ void gen_dft(double2 (&v)[R], const double2 (&w)[(R + 1) / 2], int sign) {
    if constexpr (R == 2) {
        const double2 a = v[0];
        v[0] = cadd(a, v[1]);
        v[1] = csub(a, v[1]);
    } else if constexpr (R == 4) {
        const double2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]);
        const double2 c = cadd(v[1], v[3]), d = cmuli(csub(v[1], v[3]), sign);
        v[0] = cadd(a, c);
        v[1] = cadd(b, d);
        v[2] = csub(a, c);
        v[3] = csub(b, d);
    } else if constexpr (R == 3) {
        const double s3 = 0.86602540378443864676;  // sin(2 pi/3)
        const double2 t = cadd(v[1], v[2]);
        const double2 u = make_double2(v[0].x - 0.5 * t.x, v[0].y - 0.5 * t.y);
        const double2 x = cmuli(make_double2(s3 * (v[1].x - v[2].x), s3 * (v[1].y - v[2].y)), sign);
        v[0] = cadd(v[0], t);
        v[1] = cadd(u, x);
        v[2] = csub(u, x);
    } else {
        constexpr int H = (R - 1) / 2;
        double2 a[H], b[H], o = v[0];
#pragma unroll
        for (int p = 1; p <= H; ++p) {
            a[p - 1] = cadd(v[p], v[R - p]);
            b[p - 1] = cmuli(csub(v[p], v[R - p]), sign);
            o = cadd(o, a[p - 1]);
        }
        const double2 v0 = v[0];
        v[0] = o;
#pragma unroll
        for (int q = 1; q <= H; ++q) {
            double2 c = v0, d = make_double2(0.0, 0.0);
#pragma unroll
            for (int p = 1; p <= H; ++p) {
                const int e = p * q % R;
                const double2 x = w[e <= H ? e : R - e];
                const double sn = e <= H ? x.y : -x.y;
                c = make_double2(fma(x.x, a[p - 1].x, c.x), fma(x.x, a[p - 1].y, c.y));
                d = make_double2(fma(sn, b[p - 1].x, d.x), fma(sn, b[p - 1].y, d.y));
            }
            v[q] = cadd(c, d);
            v[R - q] = csub(c, d);
        }
    }
}

// One Stockham pass of radix R over B batches of length L: butterfly j
// (k = j mod Ns) goes to outputs (j/Ns)*Ns*R + k + q*Ns with twiddles
// W^(sign q k L/(Ns R)).
template <int R>
__device__ __forceinline__ void smem_pass(const double2 *src, double2 *dst, int B, int L, int Ns, const double2 *tw,
                                          int sign) {
    const int nb = L / R, stride = nb / Ns;
    const float inb = 1.0f / nb, ins = 1.0f / Ns;
    double2 w[(R + 1) / 2];
#pragma unroll
    for (int p = 1; p <= (R - 1) / 2; ++p) w[p] = tw[p * nb];
    for (int idx = threadIdx.x; idx < nb * B; idx += blockDim.x) {
        const int b = fdiv(idx, nb, inb), j = idx - b * nb;
        const int jn = fdiv(j, Ns, ins), k = j - jn * Ns;
        const double2 *sp = src + b * L + j;
        double2 *dp = dst + b * L + jn * Ns * R + k;
        double2 v[R];
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = sp[q * nb];
        if (Ns > 1) {
            const int t = k * stride;
#pragma unroll
            for (int q = 1; q < R; ++q) {
                double2 x = tw[q * t];
                if (sign < 0) x.y = -x.y;
                v[q] = cmul(v[q], x);
            }
        }
        gen_dft<R>(v, w, sign);
#pragma unroll
        for (int q = 0; q < R; ++q) dp[q * Ns] = v[q];
    }
}

// B batches of length L (batch stride L) in `buf`; `tmp` is the ping-pong
// buffer; tw[t] = exp(+2 pi i t/L).  Returns the buffer holding the result.
// Stockham autosort.  Each radix has its own code with the butterfly in
// registers: with the radix a variable the butterfly lived in local memory and
// the primes took a table product per term (N=37, 3K=60, 3M=33, six fields: z
// 9.8, theta 23.2 us; now 9.0, 8.2).
__device__ __forceinline__ double2 *smem_fft(double2 *buf, double2 *tmp, int B, const FFTPlan &pl, const double2 *tw,
                                             int sign) {
    double2 *src = buf, *dst = tmp;
    int Ns = 1;
    for (int s = 0; s < pl.nf; ++s) {
        switch (pl.f[s]) {
        case 2: smem_pass<2>(src, dst, B, pl.L, Ns, tw, sign); break;
        case 3: smem_pass<3>(src, dst, B, pl.L, Ns, tw, sign); break;
        case 4: smem_pass<4>(src, dst, B, pl.L, Ns, tw, sign); break;
        case 5: smem_pass<5>(src, dst, B, pl.L, Ns, tw, sign); break;
        case 7: smem_pass<7>(src, dst, B, pl.L, Ns, tw, sign); break;
        case 11: smem_pass<11>(src, dst, B, pl.L, Ns, tw, sign); break;
        default: smem_pass<13>(src, dst, B, pl.L, Ns, tw, sign); break;
        }
        __syncthreads();
        double2 *t = src;
        src = dst;
        dst = t;
        Ns *= pl.f[s];
    }
    return src;
}

struct SrcPtrs {
    const double2 *p[6];
};
struct PhysPtrs {
    double *p[6];
};
struct CPhysPtrs {
    const double *p[6];
};
struct DstPtrs {
    double2 *p[6];
};

// z pass, spectral -> (m, z) columns: grid (m-chunk, n, comp)
__global__ void __launch_bounds__(FFT_THREADS, 2) k_zinv(SrcPtrs src, double2 *__restrict__ T, Geo g, FFTPlan pz, const double2 *__restrict__ twz,
                       int MC) {
    extern __shared__ double2 sm[];
    const int Z = g.Z, K = g.K;
    double2 *buf = sm, *tmp = sm + MC * Z, *tw = sm + 2 * MC * Z;
    const int comp = blockIdx.z, n = blockIdx.y, m0 = blockIdx.x * MC;
    const int mc = min(MC, g.M - m0);
    const double2 *f = src.p[comp] + (size_t)n * g.Hp;
    for (int i = threadIdx.x; i < Z; i += blockDim.x) tw[i] = twz[i];
    const float iZ = 1.0f / Z;
#pragma unroll 4
    for (int idx = threadIdx.x; idx < mc * Z; idx += blockDim.x) {
        const int c = fdiv(idx, Z, iZ), j = idx - c * Z, m = m0 + c;
        // zero-padded in k, the Hermitian fill at m = 0
        const int kk = j < K ? j : j - Z;
        const bool zero = j >= K && j <= 2 * K, conj = m == 0 && kk < 0;
        double2 v = make_double2(0.0, 0.0);
        if (!zero) v = f[conj ? -kk : m * (2 * K - 1) + kk];
        v.y = conj ? -v.y : v.y;
        buf[idx] = v;
    }
    __syncthreads();
    const double2 *res = smem_fft(buf, tmp, mc, pz, tw, +1);
    double2 *out = T + ((size_t)(comp * g.N + n) * g.M + m0) * Z;
    for (int idx = threadIdx.x; idx < mc * Z; idx += blockDim.x) out[idx] = res[idx];
}

// theta pass, (m, z) columns -> physical: grid (z-chunk, n); ncomp comps,
// ZC rows per block, two rows per complex FFT
__global__ void __launch_bounds__(FFT_THREADS, 2) k_thinv(const double2 *__restrict__ T, PhysPtrs dst, int ncomp, Geo g, FFTPlan pt,
                        const double2 *__restrict__ twt, int ZC) {
    extern __shared__ double2 sm[];
    const int Th = g.Th, M = g.M, Z = g.Z;
    const int np = ZC / 2, B = ncomp * np;
    double2 *buf = sm, *tmp = sm + B * Th, *tw = sm + 2 * B * Th;
    const int n = blockIdx.y, z0 = blockIdx.x * ZC;
    for (int i = threadIdx.x; i < Th; i += blockDim.x) tw[i] = twt[i];
    const float inp = 1.0f / np, iM = 1.0f / M;
    // Th = 3M: mode m's thread also clears X[M + m] of the zero band (m = 0 X[2M])
#pragma unroll 4
    for (int idx = threadIdx.x; idx < ncomp * M * np; idx += blockDim.x) {
        const int rest = fdiv(idx, np, inp), zp = idx - rest * np;
        const int comp = fdiv(rest, M, iM), m = rest - comp * M;
        const int za = z0 + 2 * zp, zb = za + 1;
        const double2 *col = T + ((size_t)(comp * g.N + n) * M + m) * Z;
        double2 a = (za < Z) ? col[za] : make_double2(0.0, 0.0);
        double2 b = (zb < Z) ? col[zb] : make_double2(0.0, 0.0);
        double2 *X = buf + (comp * np + zp) * Th;
        X[M + m] = make_double2(0.0, 0.0);
        if (m == 0) {
            X[0] = make_double2(a.x, b.x);  // c2r: DC imaginary parts ignored
            X[2 * M] = make_double2(0.0, 0.0);
        } else {
            X[m] = make_double2(a.x - b.y, a.y + b.x);            // a + i b
            X[Th - m] = make_double2(a.x + b.y, -a.y + b.x);      // conj(a) + i conj(b)
        }
    }
    __syncthreads();
    const double2 *res = smem_fft(buf, tmp, B, pt, tw, +1);
    const float iC = 1.0f / ZC, iT = 1.0f / Th;
    for (int idx = threadIdx.x; idx < ncomp * Th * ZC; idx += blockDim.x) {
        const int rest = fdiv(idx, ZC, iC), zz = idx - rest * ZC;
        const int comp = fdiv(rest, Th, iT), t = rest - comp * Th;
        const int z = z0 + zz;
        if (z >= Z) continue;
        const double2 v = res[(comp * np + zz / 2) * Th + t];
        dst.p[comp][((size_t)n * Th + t) * Z + z] = (zz & 1) ? v.y : v.x;
    }
}

// theta pass, physical -> (m, z) columns (scaled): grid (z-chunk, n).
// cross != 0: inputs are (r,t,z,curlr,curlt,curlz) and the three outputs are
// the components of u x curl(u) (velocity.f90:325-330).
__global__ void __launch_bounds__(FFT_THREADS, 2) k_thfwd(CPhysPtrs src, int ncomp, int cross, double2 *__restrict__ T, Geo g, FFTPlan pt,
                        const double2 *__restrict__ twt, int ZC, double scale) {
    extern __shared__ double2 sm[];
    const int Th = g.Th, M = g.M, Z = g.Z;
    const int np = ZC / 2, B = ncomp * np;
    double2 *buf = sm, *tmp = sm + B * Th, *tw = sm + 2 * B * Th;
    const int n = blockIdx.y, z0 = blockIdx.x * ZC;
    for (int i = threadIdx.x; i < Th; i += blockDim.x) tw[i] = twt[i];
    double *bre = reinterpret_cast<double *>(buf);
    const float iC = 1.0f / ZC, iT = 1.0f / Th, inp = 1.0f / np, iM = 1.0f / M;
    if (cross) {  // a grid point's three components together
#pragma unroll 2
        for (int idx = threadIdx.x; idx < Th * ZC; idx += blockDim.x) {
            const int t = fdiv(idx, ZC, iC), zz = idx - t * ZC, z = z0 + zz;
            const size_t at = ((size_t)n * Th + t) * Z + min(z, Z - 1);
            const double ur = src.p[0][at], ut = src.p[1][at], uz = src.p[2][at];
            const double cr = src.p[3][at], ct = src.p[4][at], cz = src.p[5][at];
            double *o = bre + 2 * (zz / 2 * Th + t) + (zz & 1);
            o[0] = z < Z ? scale * (ut * cz - uz * ct) : 0.0;
            o[2 * np * Th] = z < Z ? scale * (uz * cr - ur * cz) : 0.0;
            o[4 * np * Th] = z < Z ? scale * (ur * ct - ut * cr) : 0.0;
        }
    } else {
#pragma unroll 4
        for (int idx = threadIdx.x; idx < ncomp * Th * ZC; idx += blockDim.x) {
            const int rest = fdiv(idx, ZC, iC), zz = idx - rest * ZC, z = z0 + zz;
            const int comp = fdiv(rest, Th, iT), t = rest - comp * Th;
            const double v = src.p[comp][((size_t)n * Th + t) * Z + min(z, Z - 1)];
            bre[2 * ((comp * np + zz / 2) * Th + t) + (zz & 1)] = z < Z ? scale * v : 0.0;
        }
    }
    __syncthreads();
    const double2 *res = smem_fft(buf, tmp, B, pt, tw, -1);
    for (int idx = threadIdx.x; idx < ncomp * M * np; idx += blockDim.x) {
        const int rest = fdiv(idx, np, inp), zp = idx - rest * np;
        const int comp = fdiv(rest, M, iM), m = rest - comp * M;
        const double2 *X = res + (comp * np + zp) * Th;
        const double2 A = X[m], Bv = X[m ? Th - m : 0];
        // separate the two packed real transforms
        const double2 a = make_double2(0.5 * (A.x + Bv.x), 0.5 * (A.y - Bv.y));
        const double2 b = make_double2(0.5 * (A.y + Bv.y), -0.5 * (A.x - Bv.x));
        double2 *col = T + ((size_t)(comp * g.N + n) * M + m) * Z;
        const int za = z0 + 2 * zp, zb = za + 1;
        if (za < Z) col[za] = a;
        if (zb < Z) col[zb] = b;
    }
}

// z pass, (m, z) columns -> spectral with truncation: grid (m-chunk, n, comp)
__global__ void __launch_bounds__(FFT_THREADS, 2) k_zfwd(const double2 *__restrict__ T, DstPtrs dst, Geo g, FFTPlan pz,
                       const double2 *__restrict__ twz, int MC) {
    extern __shared__ double2 sm[];
    const int Z = g.Z, K = g.K;
    double2 *buf = sm, *tmp = sm + MC * Z, *tw = sm + 2 * MC * Z;
    const int comp = blockIdx.z, n = blockIdx.y, m0 = blockIdx.x * MC;
    const int mc = min(MC, g.M - m0);
    for (int i = threadIdx.x; i < Z; i += blockDim.x) tw[i] = twz[i];
    const double2 *in = T + ((size_t)(comp * g.N + n) * g.M + m0) * Z;
#pragma unroll 4
    for (int idx = threadIdx.x; idx < mc * Z; idx += blockDim.x) buf[idx] = in[idx];
    __syncthreads();
    const double2 *res = smem_fft(buf, tmp, mc, pz, tw, -1);
    double2 *f = dst.p[comp] + (size_t)n * g.Hp;
    const float iK = 1.0f / (2 * K - 1);
    for (int idx = threadIdx.x; idx < mc * (2 * K - 1); idx += blockDim.x) {
        const int c = fdiv(idx, 2 * K - 1, iK), kk = idx - c * (2 * K - 1) - (K - 1);
        const int m = m0 + c;
        if (m == 0) {
            if (kk >= 0) f[kk] = res[c * Z + kk];
        } else {
            f[m * (2 * K - 1) + kk] = res[c * Z + (kk >= 0 ? kk : Z + kk)];
        }
    }
}

// ------------------------------------------------ the compiled lengths
// The same four passes with the row transform known at compile time: a z pass
// keeps its columns' rows in registers on both sides (RowsIO), a theta pass
// takes one field (or the three components of the product) of ROW_ZC z rows.
// Bound by latency at these sizes: N=40, M=16, 3K=72, 3M=48, three fields,
// z 10.6 -> 3.1, theta 13.5 -> 6.1 us inverse, z 9.5 -> 3.4, theta 11.3 -> 5.2
// forward against the mixed-radix passes.
static constexpr int ROW_ZC = 16;
// the product of a long (two-buffer) length: half the rows, to fit in shared memory
__host__ __device__ constexpr int thfwd_zc(int L, int nc) { return nc == 3 && L > 192 ? ROW_ZC / 2 : ROW_ZC; }

template <int ZL>
__global__ void __launch_bounds__(FFT_THREADS) k_zinv_rows(SrcPtrs src, double2 *__restrict__ T, Geo g,
                                                           const double2 *__restrict__ twz, int MC) {
    extern __shared__ double2 sm[];
    using FR = RowsIO<ZL, double2>;
    constexpr int K = ZL / 3;
    double2 *tw = sm + (FR::smem_elems(MC) - ZL);
    const int comp = blockIdx.z, n = blockIdx.y, m0 = blockIdx.x * MC;
    const int mc = min(MC, g.M - m0);
    const double2 *__restrict__ f = src.p[comp] + (size_t)n * g.Hp;
    double2 *out = T + ((size_t)(comp * g.N + n) * g.M + m0) * ZL;
    FR::table(tw, twz);
    FR::template run<+1>(
        sm, mc, tw,
        [&](int c, int j) -> double2 {  // zero-padded in k, the Hermitian fill at m = 0
            const int m = m0 + c, kk = j < K ? j : j - ZL;
            const bool zero = j >= K && j <= 2 * K, conj = m == 0 && kk < 0;
            double2 v = make_double2(0.0, 0.0);
            if (!zero) v = f[conj ? -kk : m * (2 * K - 1) + kk];
            v.y = conj ? -v.y : v.y;
            return v;
        },
        [&](int c, int j, int step, auto &v) {
#pragma unroll
            for (int q = 0; q < (int)(sizeof(v) / sizeof(double2)); ++q) out[c * ZL + j + step * q] = v[q];
        });
}

template <int TL>
__global__ void __launch_bounds__(FFT_THREADS) k_thinv_rows(const double2 *__restrict__ T, PhysPtrs dst, Geo g,
                                                            const double2 *__restrict__ twt) {
    extern __shared__ double2 sm[];
    using FR = FFTRows<TL, double2>;
    constexpr int M = TL / 3, np = ROW_ZC / 2, RS = FR::pitch;
    double2 *tw = sm + (FR::smem_elems(np) - 2 * TL), *tw2 = tw + TL;
    const int Z = g.Z, n = blockIdx.y, z0 = blockIdx.x * ROW_ZC, comp = blockIdx.z;
    fft4_tables<TL>(tw, tw2, twt);
    const double2 *in = T + (size_t)(comp * g.N + n) * M * Z;
    // mode m's thread also clears X[M + m] of the zero band (m = 0 X[2M])
#pragma unroll 4
    for (int idx = threadIdx.x; idx < M * np; idx += blockDim.x) {
        const int zp = idx % np, m = idx / np;
        const int za = z0 + 2 * zp, zb = za + 1;
        const double2 a = (za < Z) ? in[m * Z + za] : make_double2(0.0, 0.0);
        const double2 b = (zb < Z) ? in[m * Z + zb] : make_double2(0.0, 0.0);
        double2 *X = sm + zp * RS;
        X[M + m] = make_double2(0.0, 0.0);
        if (m == 0) {
            X[0] = make_double2(a.x, b.x);  // c2r: DC imaginary parts ignored
            X[2 * M] = make_double2(0.0, 0.0);
        } else {
            X[m] = make_double2(a.x - b.y, a.y + b.x);
            X[TL - m] = make_double2(a.x + b.y, -a.y + b.x);
        }
    }
    __syncthreads();
    FR::template run<+1>(sm, np, tw, tw2);
    double *__restrict__ out = dst.p[comp] + (size_t)n * TL * Z;
    for (int idx = threadIdx.x; idx < TL * ROW_ZC; idx += blockDim.x) {
        const int zz = idx % ROW_ZC, t = idx / ROW_ZC, z = z0 + zz;
        const double2 v = sm[(zz / 2) * RS + t];
        if (z < Z) out[t * Z + z] = (zz & 1) ? v.y : v.x;
    }
}

// NC = 3: the components of u x curl(u) from six fields; 1: field blockIdx.z
template <int TL, int NC>
__global__ void __launch_bounds__(FFT_THREADS) k_thfwd_rows(CPhysPtrs src, double2 *__restrict__ T, Geo g,
                                                            const double2 *__restrict__ twt, double scale) {
    extern __shared__ double2 sm[];
    using FR = FFTRows<TL, double2>;
    constexpr int ZC = thfwd_zc(TL, NC), M = TL / 3, np = ZC / 2, RS = FR::pitch;
    double2 *tw = sm + (FR::smem_elems(NC * np) - 2 * TL), *tw2 = tw + TL;
    const int Z = g.Z, n = blockIdx.y, z0 = blockIdx.x * ZC;
    fft4_tables<TL>(tw, tw2, twt);
    double *re = reinterpret_cast<double *>(sm);
#pragma unroll 4
    for (int idx = threadIdx.x; idx < TL * ZC; idx += blockDim.x) {
        const int zz = idx % ZC, t = idx / ZC, z = z0 + zz;
        const size_t at = ((size_t)n * TL + t) * Z + min(z, Z - 1);
        double *o = re + 2 * (zz / 2 * RS + t) + (zz & 1);
        if (NC == 3) {
            const double ur = src.p[0][at], ut = src.p[1][at], uz = src.p[2][at];
            const double cr = src.p[3][at], ct = src.p[4][at], cz = src.p[5][at];
            o[0] = z < Z ? scale * (ut * cz - uz * ct) : 0.0;
            o[2 * np * RS] = z < Z ? scale * (uz * cr - ur * cz) : 0.0;
            o[4 * np * RS] = z < Z ? scale * (ur * ct - ut * cr) : 0.0;
        } else {
            const double v = src.p[blockIdx.z][at];
            o[0] = z < Z ? scale * v : 0.0;
        }
    }
    __syncthreads();
    FR::template run<-1>(sm, NC * np, tw, tw2);
    for (int idx = threadIdx.x; idx < NC * M * np; idx += blockDim.x) {
        const int zp = idx % np, m = idx / np % M, c = idx / (np * M);
        const double2 *X = sm + (c * np + zp) * RS;
        const double2 A = X[m], B = X[m ? TL - m : 0];
        // separate the two packed real transforms
        const int za = z0 + 2 * zp, zb = za + 1;
        double2 *col = T + ((size_t)((NC == 3 ? c : blockIdx.z) * g.N + n) * M + m) * Z;
        if (za < Z) col[za] = make_double2(0.5 * (A.x + B.x), 0.5 * (A.y - B.y));
        if (zb < Z) col[zb] = make_double2(0.5 * (A.y + B.y), -0.5 * (A.x - B.x));
    }
}

template <int ZL>
__global__ void __launch_bounds__(FFT_THREADS) k_zfwd_rows(const double2 *__restrict__ T, DstPtrs dst, Geo g,
                                                           const double2 *__restrict__ twz, int MC) {
    extern __shared__ double2 sm[];
    using FR = RowsIO<ZL, double2>;
    constexpr int K = ZL / 3;
    double2 *tw = sm + (FR::smem_elems(MC) - ZL);
    const int comp = blockIdx.z, n = blockIdx.y, m0 = blockIdx.x * MC;
    const int mc = min(MC, g.M - m0);
    const double2 *__restrict__ in = T + ((size_t)(comp * g.N + n) * g.M + m0) * ZL;
    double2 *__restrict__ f = dst.p[comp] + (size_t)n * g.Hp;
    FR::table(tw, twz);
    FR::template run<-1>(
        sm, mc, tw, [&](int c, int j) -> double2 { return in[c * ZL + j]; },
        [&](int c, int j, int step, auto &v) {  // the kept |k| < K, k >= 0 only at m = 0
            const int m = m0 + c;
#pragma unroll
            for (int q = 0; q < (int)(sizeof(v) / sizeof(double2)); ++q) {
                const int t = j + step * q, kk = t < K ? t : t - ZL;
                if (!(t >= K && t <= 2 * K) && !(m == 0 && kk < 0)) f[m * (2 * K - 1) + kk] = v[q];
            }
        });
}

// columns and threads of a z pass's block
struct RowsLaunch {
    int MC, threads;
    size_t smem;
};
template <int L> static RowsLaunch zrows_plan(const Geo &g) {
    using FR = RowsIO<L, double2>;
    const int per = FR::four ? FR::L2 : L / 8;  // threads that work on a row
    RowsLaunch r;
    r.MC = std::min(g.M, std::max(1, FFT_THREADS / per));
    r.threads = std::min(FFT_THREADS, std::max(32, (r.MC * per + 31) / 32 * 32));
    r.smem = FR::smem_elems(r.MC) * sizeof(double2);
    return r;
}

static size_t zpass_smem(const pf_ctx *ctx, int MC) { return (size_t)(2 * MC + 1) * ctx->g.Z * sizeof(double2); }
static size_t thpass_smem(const pf_ctx *ctx, int ncomp, int ZC) {
    return ((size_t)2 * ncomp * (ZC / 2) + 1) * ctx->g.Th * sizeof(double2);
}

static const size_t kSmemBudget = 200 * 1024;

static int pick_mc(const pf_ctx *ctx) {
    int MC = ctx->g.M;
    while (MC > 1 && zpass_smem(ctx, MC) > 96 * 1024) --MC;
    return MC;
}
static int pick_zc(const pf_ctx *ctx, int ncomp) {
    int ZC = 16;
    while (ZC > 2 && thpass_smem(ctx, ncomp, ZC) > kSmemBudget) ZC -= 2;
    return ZC;
}

static int set_smem(const void *fn, size_t bytes) { return pf_raise_smem(fn, bytes); }

int pf_launch_coll2phys(pf_ctx *ctx, int ncomp, const double2 *const *src, double *const *dst) {
    const Geo &g = ctx->g;
    SrcPtrs sp{};
    PhysPtrs pp{};
    for (int c = 0; c < ncomp; ++c) {
        sp.p[c] = src[c];
        pp.p[c] = dst[c];
    }
    double2 *T = (double2 *)ctx->T;
    switch (g.Z) {
#define PF_CASE(L)                                                                                               \
    case L: {                                                                                                    \
        const RowsLaunch r = zrows_plan<L>(g);                                                                   \
        PF_TRY(set_smem((const void *)k_zinv_rows<L>, r.smem));                                                  \
        ProfScope ps_(ctx, PF_K_ZINV);                                                                           \
        k_zinv_rows<L><<<dim3((g.M + r.MC - 1) / r.MC, g.N, ncomp), r.threads, r.smem, ctx->stream>>>(sp, T, g,  \
                                                                                          ctx->twZ, r.MC);       \
    } break;
        PF_FFT_LENGTHS(PF_CASE)
#undef PF_CASE
    default: {
        const int MC = pick_mc(ctx);
        const size_t sz = zpass_smem(ctx, MC);
        PF_TRY(set_smem((const void *)k_zinv, sz));
        ProfScope ps_(ctx, PF_K_ZINV);
        k_zinv<<<dim3((g.M + MC - 1) / MC, g.N, ncomp), FFT_THREADS, sz, ctx->stream>>>(sp, T, g, ctx->planZ, ctx->twZ,
                                                                                         MC);
    }
    }
    PF_LAUNCHED(ctx);
    switch (g.Th) {
#define PF_CASE(L)                                                                                               \
    case L: {                                                                                                    \
        const size_t sz = FFTRows<L, double2>::smem_elems(ROW_ZC / 2) * sizeof(double2);                         \
        PF_TRY(set_smem((const void *)k_thinv_rows<L>, sz));                                                     \
        ProfScope ps_(ctx, PF_K_THINV);                                                                          \
        k_thinv_rows<L><<<dim3((g.Z + ROW_ZC - 1) / ROW_ZC, g.N, ncomp), 128, sz, ctx->stream>>>(T, pp, g,       \
                                                                                                  ctx->twT);     \
    } break;
        PF_FFT_LENGTHS(PF_CASE)
#undef PF_CASE
    default: {
        const int ZC = pick_zc(ctx, ncomp);
        const size_t sz = thpass_smem(ctx, ncomp, ZC);
        PF_TRY(set_smem((const void *)k_thinv, sz));
        ProfScope ps_(ctx, PF_K_THINV);
        k_thinv<<<dim3((g.Z + ZC - 1) / ZC, g.N), FFT_THREADS, sz, ctx->stream>>>(T, pp, ncomp, g, ctx->planT, ctx->twT,
                                                                                   ZC);
    }
    }
    PF_LAUNCHED(ctx);
    return PF_OK;
}

int pf_launch_phys2coll(pf_ctx *ctx, int ncomp, const double *const *src, double2 *const *dst, bool cross) {
    const Geo &g = ctx->g;
    CPhysPtrs sp{};
    DstPtrs dp{};
    const int nin = cross ? 6 : ncomp;
    for (int c = 0; c < nin; ++c) sp.p[c] = src[c];
    for (int c = 0; c < ncomp; ++c) dp.p[c] = dst[c];
    double2 *T = (double2 *)ctx->T;
    const double scale = 1.0 / (double)(g.Z * g.Th);  // transform.fftw3.f90:114
    switch (g.Th) {
#define PF_CASE(L)                                                                                               \
    case L: {                                                                                                    \
        const auto k = cross ? k_thfwd_rows<L, 3> : k_thfwd_rows<L, 1>;                                          \
        const int zc = thfwd_zc(L, cross ? 3 : 1);                                                               \
        const size_t sz = FFTRows<L, double2>::smem_elems((cross ? 3 : 1) * zc / 2) * sizeof(double2);           \
        PF_TRY(set_smem((const void *)k, sz));                                                                   \
        ProfScope ps_(ctx, PF_K_THFWD);                                                                          \
        k<<<dim3((g.Z + zc - 1) / zc, g.N, cross ? 1 : ncomp), cross ? 256 : 128, sz, ctx->stream>>>(    \
            sp, T, g, ctx->twT, scale);                                                                          \
    } break;
        PF_FFT_LENGTHS(PF_CASE)
#undef PF_CASE
    default: {
        const int ZC = pick_zc(ctx, ncomp);
        const size_t sz = thpass_smem(ctx, ncomp, ZC);
        PF_TRY(set_smem((const void *)k_thfwd, sz));
        ProfScope ps_(ctx, PF_K_THFWD);
        k_thfwd<<<dim3((g.Z + ZC - 1) / ZC, g.N), FFT_THREADS, sz, ctx->stream>>>(sp, ncomp, cross ? 1 : 0, T, g,
                                                                                   ctx->planT, ctx->twT, ZC, scale);
    }
    }
    PF_LAUNCHED(ctx);
    switch (g.Z) {
#define PF_CASE(L)                                                                                               \
    case L: {                                                                                                    \
        const RowsLaunch r = zrows_plan<L>(g);                                                                   \
        PF_TRY(set_smem((const void *)k_zfwd_rows<L>, r.smem));                                                  \
        ProfScope ps_(ctx, PF_K_ZFWD);                                                                           \
        k_zfwd_rows<L><<<dim3((g.M + r.MC - 1) / r.MC, g.N, ncomp), r.threads, r.smem, ctx->stream>>>(T, dp, g,  \
                                                                                          ctx->twZ, r.MC);       \
    } break;
        PF_FFT_LENGTHS(PF_CASE)
#undef PF_CASE
    default: {
        const int MC = pick_mc(ctx);
        const size_t sz = zpass_smem(ctx, MC);
        PF_TRY(set_smem((const void *)k_zfwd, sz));
        ProfScope ps_(ctx, PF_K_ZFWD);
        k_zfwd<<<dim3((g.M + MC - 1) / MC, g.N, ncomp), FFT_THREADS, sz, ctx->stream>>>(T, dp, g, ctx->planZ, ctx->twZ,
                                                                                         MC);
    }
    }
    PF_LAUNCHED(ctx);
    return PF_OK;
}

// ------------------------------------------------------------ CFL maxima
// per radial point: max|u_r|, max|u_t|, max|u_z + 1 - r^2| (velocity.f90:459-467)
__global__ void k_maxphys(const double *__restrict__ pr, const double *__restrict__ pt,
                          const double *__restrict__ pz, double *out, DevMesh dm, Geo g) {
    const int n = blockIdx.x;
    const size_t plane = (size_t)g.Th * g.Z;
    const double base = 1.0 - dm.rp[4 * g.N + n] * dm.rp[4 * g.N + n];
    double a = 0.0, b = 0.0, c = 0.0;
    for (size_t i = threadIdx.x; i < plane; i += blockDim.x) {
        const size_t at = (size_t)n * plane + i;
        a = fmax(a, fabs(pr[at]));
        b = fmax(b, fabs(pt[at]));
        c = fmax(c, fabs(pz[at] + base));
    }
    __shared__ double s[3][32];
    for (int o = 16; o > 0; o >>= 1) {
        a = fmax(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = fmax(b, __shfl_xor_sync(0xffffffffu, b, o));
        c = fmax(c, __shfl_xor_sync(0xffffffffu, c, o));
    }
    const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        s[0][w] = a;
        s[1][w] = b;
        s[2][w] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < nw; ++i) {
            a = fmax(a, s[0][i]);
            b = fmax(b, s[1][i]);
            c = fmax(c, s[2][i]);
        }
        out[3 * n + 0] = a;
        out[3 * n + 1] = b;
        out[3 * n + 2] = c;
    }
}

int pf_launch_maxtstep(pf_ctx *ctx, double *dt3) {
    const Geo &g = ctx->g;
    std::vector<double> mx(3 * g.N);
    if (ctx->cfl_fused) {  // maxima left by the fused theta pass
        std::vector<unsigned long long> bits(3 * g.N);
        PF_CUDA(cudaMemcpyAsync(bits.data(), ctx->cflmax, bits.size() * sizeof(unsigned long long),
                                cudaMemcpyDeviceToHost, ctx->stream));
        PF_CUDA(cudaStreamSynchronize(ctx->stream));
        for (int i = 0; i < 3 * g.N; ++i) mx[i] = bits_to_double(bits[i]);
    } else {
    {
        ProfScope ps_(ctx, PF_K_EW);
        k_maxphys<<<g.N, 256, 0, ctx->stream>>>(ctx->phys[0].d, ctx->phys[1].d, ctx->phys[2].d, ctx->red, ctx->dm, g);
    }
    PF_LAUNCHED(ctx);
    PF_CUDA(cudaMemcpyAsync(mx.data(), ctx->red, mx.size() * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    PF_CUDA(cudaStreamSynchronize(ctx->stream));
    }
    const double PI = 3.1415926535897931;
    const std::vector<double> &r = ctx->hm.r;
    const int N = g.N;
    double dt[3] = {1e99, 1e99, 1e99};
    for (int n = 0; n < N; ++n) {
        double d;
        if (n == 0) d = r[1] - r[0];
        else if (n == N - 1) d = r[N - 1] - r[N - 2];
        else d = std::min(r[n] - r[n - 1], r[n + 1] - r[n]);
        if (mx[3 * n] != 0.0) dt[0] = std::min(dt[0], d / mx[3 * n]);
        d = 2.0 * PI / (double)(g.Th * g.Mp);
        if (mx[3 * n + 1] != 0.0) dt[1] = std::min(dt[1], d / mx[3 * n + 1]);
        d = 2.0 * PI / (g.alpha * g.Z);
        if (mx[3 * n + 2] != 0.0) dt[2] = std::min(dt[2], d / mx[3 * n + 2]);
    }
    for (int i = 0; i < 3; ++i) dt3[i] = dt[i];
    return PF_OK;
}

// ------------------------------------------------------------------ C ABI
extern "C" int pf_tra_coll2phys(const pf_coll *c, pf_phys *p) {
    PF_ARG(c && p && c->ctx == p->ctx, "pf_tra_coll2phys: bad argument");
    const double2 *src[1] = {c->d};
    double *dst[1] = {p->d};
    return pf_launch_coll2phys(c->ctx, 1, src, dst);
}

extern "C" int pf_tra_phys2coll(const pf_phys *p, pf_coll *c) {
    PF_ARG(c && p && c->ctx == p->ctx, "pf_tra_phys2coll: bad argument");
    const double *src[1] = {p->d};
    double2 *dst[1] = {c->d};
    return pf_launch_phys2coll(c->ctx, 1, src, dst, false);
}
