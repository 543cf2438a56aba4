// Spectral -> physical transform of one coll field that allocates no device
// memory: the variant of var_coll2spec + tra_spec2phys for callers that
// cannot call cudaMalloc (for example a host code whose device memory is
// owned by another allocator or pool, a loop that must not allocate while a
// stream is being captured elsewhere, or a Fortran driver that only hands
// over device pointers it allocated itself).
//
// Its scratch is the file-scope array below, PF_NOALLOC_SCRATCH_BYTES
// (24 MiB) in size; every GPU that loads this library holds it until the
// process exits.  The first 64 KiB hold the twiddle tables of every built
// transform length, written once per device at set-up; the rest holds the
// (m, z) intermediate of the z pass.  All calls share the intermediate and it
// keeps the previous call's contents (nothing in it has to start at zero:
// every call writes every entry it later reads).  Calls that overlap on the
// GPU -- on different streams, or from different host threads without
// ordering -- race on it.
//
// Host code must not hand the array's name to a kernel: in host code the name
// denotes a host-side stand-in.  The first call made on a device, with that
// device current, does the set-up: it looks up the device address with
// cudaGetSymbolAddress and writes the twiddle tables with a synchronous copy.
// Make that first call before any stream capture.  Every later call only
// queues its two kernels on the caller's stream.  The address and the tables
// are kept per device ordinal for the life of the process; a cudaDeviceReset
// in the caller discards the tables, and this entry point is not usable on
// that device after one.
#include <algorithm>
#include <cmath>
#include <mutex>
#include "pf_internal.cuh"
#include "pf_fftcore.cuh"

static __device__ __align__(256) unsigned char g_noalloc_scratch[PF_NOALLOC_SCRATCH_BYTES];

static constexpr size_t kTwiddleBytes = 64 * 1024;  // tables of all built lengths (21 KiB used)
static std::mutex g_noalloc_mu;
static void *g_noalloc_addr[256];

#define PF_NA_LENGTHS(X) X(12) X(15) X(18) X(24) X(36) X(48) X(72) X(96) X(144) X(192) X(288) X(384)
static const int kLengths[] = {
#define PF_CASE(L) L,
    PF_NA_LENGTHS(PF_CASE)
#undef PF_CASE
};
static constexpr int kNumLengths = (int)(sizeof(kLengths) / sizeof(kLengths[0]));

// offset (in double2 entries) of length L's table exp(+2 pi i t/L), t < L,
// in the twiddle region; -1 if L is not built
static int twiddle_offset(int L) {
    int off = 0;
    for (int i = 0; i < kNumLengths; ++i) {
        if (kLengths[i] == L) return off;
        off += kLengths[i];
    }
    return -1;
}

// Set-up, once per device: the scratch address, and the twiddle tables of
// every built length (rounded once from long double) written into its first
// kTwiddleBytes with a synchronous copy from host memory.
static int scratch_address(int dev, unsigned char **out) {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (dev < 0 || dev >= 256) {
        pf_set_error("pf_tra_coll2phys_noalloc: device index %d out of range", dev);
        return PF_ERR_ARG;
    }
    if (!g_noalloc_addr[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            pf_set_error("pf_tra_coll2phys_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
            return PF_ERR_CUDA;
        }
        std::vector<double2> tw;
        for (int i = 0; i < kNumLengths; ++i) {
            const int L = kLengths[i];
            for (int t = 0; t < L; ++t) {
                const long double a = 2.0L * 3.14159265358979323846264338327950288L * (long double)t / (long double)L;
                tw.push_back(make_double2((double)cosl(a), (double)sinl(a)));
            }
        }
        static_assert(kTwiddleBytes >= 1329 * sizeof(double2), "twiddle region too small");
        e = cudaMemcpy(p, tw.data(), tw.size() * sizeof(double2), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            pf_set_error("pf_tra_coll2phys_noalloc: twiddle set-up copy failed: %s", cudaGetErrorString(e));
            return PF_ERR_CUDA;
        }
        g_noalloc_addr[dev] = p;
    }
    *out = static_cast<unsigned char *>(g_noalloc_addr[dev]);
    return PF_OK;
}

// z pass: reference coll layout in (re[nh*N+n], im[...]), (m, z) columns out.
// A block takes MC columns of four consecutive radial points, since n is the
// fastest index of the input: a 32-byte sector then serves four rows of the
// block (one radial point per block read each sector four times: 9.2 us a
// field at N=64, K=64, M=32, now 6.3).
static constexpr int NA_NR = 4;
template <int ZL>
__global__ void __launch_bounds__(256) k_na_zinv(const double *__restrict__ re, const double *__restrict__ im,
                                                 double2 *__restrict__ T, const double2 *__restrict__ twz, int N,
                                                 int M, int MC) {
    extern __shared__ __align__(16) unsigned char smraw[];
    using FR = RowsIO<ZL, double2>;
    constexpr int K = ZL / 3;
    double2 *rows = reinterpret_cast<double2 *>(smraw);
    double2 *tw = rows + (FR::smem_elems(MC * NA_NR) - ZL);
    const int n0 = blockIdx.y * NA_NR, m0 = blockIdx.x * MC;
    const int mc = min(MC, M - m0);
    FR::table(tw, twz);
    FR::template run<+1>(
        rows, mc * NA_NR, tw,
        [&](int b, int j) -> double2 {  // zero-padded in k, the Hermitian fill at m = 0
            const int m = m0 + b / NA_NR, n = min(n0 + b % NA_NR, N - 1);
            const int kk = j < K ? j : j - ZL;
            const bool zero = j >= K && j <= 2 * K, conj = m == 0 && kk < 0;
            double2 v = make_double2(0.0, 0.0);
            if (!zero) {
                const size_t at = (size_t)(conj ? -kk : m * (2 * K - 1) + kk) * N + n;
                v = make_double2(re[at], im[at]);
            }
            v.y = conj ? -v.y : v.y;
            return v;
        },
        [&](int b, int j, int step, auto &v) {
            const int m = m0 + b / NA_NR, n = n0 + b % NA_NR;
            if (n >= N) return;
            double2 *out = T + ((size_t)n * M + m) * ZL + j;
#pragma unroll
            for (int q = 0; q < (int)(sizeof(v) / sizeof(double2)); ++q) out[step * q] = v[q];
        });
}

// theta pass (c2r, two real rows per complex FFT) into the phys layout:
// NA_ZC rows of one radial point per block, four warps, which is what eight
// packed rows of the row transform keep busy (256 threads and the radix-4
// passes: 12.1 us a field, now 7.1)
static constexpr int NA_ZC = 16, NA_TH_THREADS = 128;
template <int TL>
__global__ void __launch_bounds__(NA_TH_THREADS) k_na_thinv(const double2 *__restrict__ T, double *__restrict__ phys,
                                                            const double2 *__restrict__ twt, int Z) {
    extern __shared__ __align__(16) unsigned char smraw[];
    using FR = FFTRows<TL, double2>;
    constexpr int M = TL / 3, np = NA_ZC / 2, RS = FR::pitch;
    double2 *buf = reinterpret_cast<double2 *>(smraw);
    double2 *tw = buf + (FR::smem_elems(np) - 2 * TL), *tw2 = tw + TL;
    const int n = blockIdx.y, z0 = blockIdx.x * NA_ZC;
    fft4_tables<TL>(tw, tw2, twt);
    // mode m's thread also clears X[M + m] of the zero band (m = 0 X[2M])
#pragma unroll 4
    for (int idx = threadIdx.x; idx < M * np; idx += blockDim.x) {
        const int zp = idx % np, m = idx / np;
        const int za = z0 + 2 * zp, zb = za + 1;
        const double2 *col = T + ((size_t)n * M + m) * Z;
        const double2 a = (za < Z) ? col[za] : make_double2(0.0, 0.0);
        const double2 b = (zb < Z) ? col[zb] : make_double2(0.0, 0.0);
        double2 *X = buf + zp * RS;
        X[M + m] = make_double2(0.0, 0.0);
        if (m == 0) {
            X[0] = make_double2(a.x, b.x);
            X[2 * M] = make_double2(0.0, 0.0);
        } else {
            X[m] = make_double2(a.x - b.y, a.y + b.x);
            X[TL - m] = make_double2(a.x + b.y, -a.y + b.x);
        }
    }
    __syncthreads();
    FR::template run<+1>(buf, np, tw, tw2);
    for (int idx = threadIdx.x; idx < TL * NA_ZC; idx += blockDim.x) {
        const int zz = idx % NA_ZC, t = idx / NA_ZC;
        const int z = z0 + zz;
        if (z >= Z) continue;
        const double2 v = buf[(zz / 2) * RS + t];
        phys[((size_t)n * TL + t) * Z + z] = (zz & 1) ? v.y : v.x;
    }
}

template <int L>
static int na_zinv(const double *re, const double *im, double2 *T, const double2 *tw, int N, int M, cudaStream_t st) {
    using FR = RowsIO<L, double2>;
    // threads a row keeps busy; enough columns for a block, and blocks for the GPU
    const int per = FR::four ? FR::L2 : L / 8, nb = (N + NA_NR - 1) / NA_NR;
    int MC = std::min(M, std::max(1, 256 / (per * NA_NR)));
    while (MC > 1 && (M + MC - 1) / MC * nb < 2 * B200_SMS) MC = (MC + 1) / 2;
    const int threads = std::min(256, (MC * NA_NR * per + 31) / 32 * 32);
    const size_t sm = FR::smem_elems(MC * NA_NR) * sizeof(double2);
    PF_TRY(pf_raise_smem((const void *)k_na_zinv<L>, sm));
    k_na_zinv<L><<<dim3((M + MC - 1) / MC, nb), std::max(threads, 32), sm, st>>>(re, im, T, tw, N, M, MC);
    PF_CHECK_LAUNCH();
    return PF_OK;
}

template <int L> static int na_thinv(const double2 *T, double *phys, const double2 *tw, int N, int Z, cudaStream_t st) {
    const size_t sm = FFTRows<L, double2>::smem_elems(NA_ZC / 2) * sizeof(double2);
    PF_TRY(pf_raise_smem((const void *)k_na_thinv<L>, sm));
    k_na_thinv<L><<<dim3((Z + NA_ZC - 1) / NA_ZC, N), NA_TH_THREADS, sm, st>>>(T, phys, tw, Z);
    PF_CHECK_LAUNCH();
    return PF_OK;
}

static bool na_length_ok(int L) {
    switch (L) {
#define PF_CASE(L) case L:
        PF_NA_LENGTHS(PF_CASE)
#undef PF_CASE
        return true;
    default:
        return false;
    }
}

extern "C" int pf_tra_coll2phys_noalloc(int N, int K, int M, const double *re, const double *im, double *phys,
                                        void *cuda_stream) {
    PF_ARG(re && im && phys, "pf_tra_coll2phys_noalloc: null pointer");
    PF_ARG(N >= 1 && K >= 1 && M >= 1, "pf_tra_coll2phys_noalloc: N, K, M must be >= 1");
    const int Z = 3 * K, Th = 3 * M;
    if (!na_length_ok(Z) || !na_length_ok(Th)) {
        pf_set_error("pf_tra_coll2phys_noalloc: transform lengths 3K=%d, 3M=%d are not among the built ones "
                     "(12 15 18 24 36 48 72 96 144 192 288 384)", Z, Th);
        return PF_ERR_ARG;
    }
    const size_t need = kTwiddleBytes + (size_t)N * M * Z * sizeof(double2);
    if (need > PF_NOALLOC_SCRATCH_BYTES) {
        pf_set_error("pf_tra_coll2phys_noalloc: N*M*3K*16 + 64 KiB = %zu bytes exceeds the %u-byte static scratch",
                     need, (unsigned)PF_NOALLOC_SCRATCH_BYTES);
        return PF_ERR_ARG;
    }
    int dev = 0;
    PF_CUDA(cudaGetDevice(&dev));
    unsigned char *scratch = nullptr;
    PF_TRY(scratch_address(dev, &scratch));
    cudaStream_t st = (cudaStream_t)cuda_stream;
    const double2 *tables = reinterpret_cast<const double2 *>(scratch);
    const double2 *twz = tables + twiddle_offset(Z);
    const double2 *twt = tables + twiddle_offset(Th);
    double2 *T = reinterpret_cast<double2 *>(scratch + kTwiddleBytes);
    switch (Z) {
#define PF_CASE(L)                                          \
    case L:                                                 \
        PF_TRY((na_zinv<L>(re, im, T, twz, N, M, st)));     \
        break;
        PF_NA_LENGTHS(PF_CASE)
#undef PF_CASE
    }
    switch (Th) {
#define PF_CASE(L)                                          \
    case L:                                                 \
        PF_TRY((na_thinv<L>(T, phys, twt, N, Z, st)));      \
        break;
        PF_NA_LENGTHS(PF_CASE)
#undef PF_CASE
    }
    return PF_OK;
}
