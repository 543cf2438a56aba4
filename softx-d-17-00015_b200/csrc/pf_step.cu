// Fused vel_step (velocity.f90:367-394): one launch per predictor or corrector.
//
// Every stage of the step is independent between Fourier modes, so a block
// takes a tile of 16 modes through all of them with the tile's fields in
// shared memory:
//   rhs    : optional nlincorr (timestep.f90:174-184) or N_ := N copy, rhs =
//            Lt u_ + N in the u+-/uz variables (velocity.f90:369-373)
//   div    : PPE right-hand side div(pm2rt(rhs)), zero boundary rows
//            (velocity.f90:228-230)
//   PPE    : pressure Poisson solve with LNp (timestep.f90:102-123)
//   proj   : rhs - rt2pm(grad p), zero boundary rows (velocity.f90:232-236)
//   solves : the u+, u-, uz Helmholtz systems (LDp, LDm, LDz)
//   final  : influence-matrix correction (velocity.f90:238-256), pm2rt,
//            constant-flux adjustment of k=m=0 (velocity.f90:170-175),
//            mean-mode symmetry zeros, and the corrector error
//            max |u_old - u_new|^2 (timestep.f90:190-207)
// From HBM it reads u_, N (and N_, the old u in the corrector), the factors
// and the influence vectors, and writes N (or N_) and u: no stage's result
// leaves the SM.
#include <cmath>
#include "pf_internal.cuh"

struct StepArgs {
    const double2 *u_[3];  // previous state (ur_, ut_, uz_)
    double2 *Nl[3];        // vel_N (read; rewritten by nlincorr)
    double2 *N_[3];        // saved N_ (read in the corrector, written in the predictor)
    double2 *u[3];         // vel_u (read as u_old by the corrector, written)
    const double *lnp, *ld[3];  // factor tiles of LNp, LDp, LDm, LDz
    int ldpiv[3];          // 1 if that Helmholtz factorisation pivoted
    const double *U, *Ainv, *Ui;
    void *curl[3];         // curl(u) for the nonlinear terms that follow a predictor (null: not wanted),
    int mixed;             // FP32 (mixed precision) or FP64,
    double *mpart;         // and in mixed precision the mean mode's partial sums [tile][N][3]
    DevMesh dm;
    Geo g;
    double c1, c2;         // Lt coefficients: 1/dt and (1-implicit) nu/Re
    double implicit;
    int mode;              // 0 predictor, 1 corrector
    int const_flux;
    DevScalars *sc;
};

// --------------------------------------------------------- banded solves
// A warp solves one system of its tile's 16 modes: lane = 2*slot + (re, im),
// and the right-hand side sits in shared memory as rows of 32 doubles, solved
// in place.  The factors are streamed from the set's tile (pf_internal.cuh)
// through a ring of chunks that another warp keeps filled with bulk copies:
// asking for a copy takes some 200 cycles, as long as five columns of the
// solve.  Modes k and -k of a paired tile (W = 8) read the same factor values.
// Column j costs one multiply-add on the dependent chain going forward and
// three going back: the division by U(j, j) is a product with its reciprocal
// held as a sum of two doubles, as accurate as the division.  With the
// factors at hand and the code fetched a column takes 42 cycles forward and 54
// back, 73 and 83 with pivots and wide rows (N = 40, W = 8); in a block's one
// run of the sweeps, with both waited for, 89 and 145 on average.
__device__ __forceinline__ void cp_async16(unsigned saddr, const void *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(saddr), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// w[0] and w[p] exchanged, p = 0 .. KL
__device__ __forceinline__ void pivot_swap(double (&w)[KL + 1], int p) {
    static_assert(KL == 4, "select tree of five entries");
    const double t = w[0];
    const double lo = (p & 1) ? w[1] : t, hi = (p & 1) ? w[3] : w[2];
    const double mid = (p & 2) ? hi : lo;
    w[0] = (p & 4) ? w[4] : mid;
#pragma unroll
    for (int r = 1; r <= KL; ++r) w[r] = p == r ? t : w[r];
}

// Accesses to a lane's own column of a field under a uniform condition, as
// predicated instructions (a branch each costs the solves a third of their time).
__device__ __forceinline__ double lds_if(unsigned addr, bool on) {
    double v;
    asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %2, 0;\nmov.f64 %0, 0d0000000000000000;\n@p ld.shared.f64 %0, [%1];\n}\n"
                 : "=d"(v) : "r"(addr), "r"((int)on));
    return v;
}
__device__ __forceinline__ void sts_if(unsigned addr, double v, bool on) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %2, 0;\n@p st.shared.f64 [%0], %1;\n}\n" ::"r"(addr), "d"(v), "r"((int)on));
}

// Bulk copy of `bytes` (a multiple of 16) into shared memory; the mbarrier's
// phase completes when they have landed.  One lane calls it.
__device__ __forceinline__ void bulk_copy(unsigned dst, const void *src, unsigned bytes, unsigned mbar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(mbar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(mbar) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p)); }
__device__ __forceinline__ void mbar_arrive(unsigned mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(mbar) : "memory");
}

// The stream of one system's factors through its ring.  flags bit 0: the set
// has pivots; bit 1: its U has entries beyond KL columns (pivots in the last
// KL+1 columns alone, the wall row's, leave U narrow).  A chunk is `g` groups
// of 1920 bytes (W = 8) or twice that: five columns of the forward sweep, one
// turn of its register window, then five narrow or three wide columns of the
// back substitution.
static constexpr int RING = 4;      // chunks, or two where four of a group each do not fit
static constexpr int GROUP = 1920;  // bytes for W = 8
static constexpr int GF = KL + 1;   // forward columns of a group
__host__ __device__ constexpr int group_back(bool wide) { return wide ? 3 : 5; }
__host__ __device__ constexpr int group_bytes(int W) { return GROUP / 8 * W; }
// a stream's mbarriers: a chunk has landed in its place, its place is free again
struct StreamBars {
    unsigned long long full[RING], empty[RING];
    long long asked;  // chunks asked for so far
};
__device__ __forceinline__ unsigned bar_full(unsigned bars, int place) { return bars + place * 8; }
__device__ __forceinline__ unsigned bar_empty(unsigned bars, int place) { return bars + (RING + place) * 8; }
struct FactorStream {
    const double *ft;   // the tile
    int N, W, flags;
    int g, places;      // groups a chunk, chunks of the ring
    unsigned ring, bars;  // shared addresses: the chunks, the StreamBars
};
// Ask for chunks from .. to-1 of the stream, each once its place is free; by
// one lane.  False if a place was not free within the second of MBAR_TRIES: no
// more are asked for then.
__device__ __noinline__ bool stream_fill(const FactorStream s, int from, int to) {
    if (s.g < 1) return false;  // a ring too small for a chunk
    const double *src = s.ft;
    int q = 0, place = 0, turn = 0, tries = MBAR_TRIES;
#pragma unroll 1
    for (int back = 0; back < 2; ++back) {
        const int cols = s.g * (back ? group_back(s.flags & 2) : GF);
        const int row = (back ? ft_back_rows(s.flags & 2) : ft_fwd_rows(s.flags & 1)) * s.W;
#pragma unroll 1
        for (int j0 = 0; j0 < s.N; j0 += cols, ++q) {
            const int words = min(cols, s.N - j0) * row;
            if (q >= to) return true;
            if (q >= from) {
                // (a solve that has given up hands places back with their copies still on the way)
                if (turn > 0 && !(mbar_wait(bar_empty(s.bars, place), (turn - 1) & 1, tries) &&
                                  mbar_wait(bar_full(s.bars, place), (turn - 1) & 1, tries)))
                    return false;
                bulk_copy(s.ring + place * s.g * group_bytes(s.W), src, words * 8, bar_full(s.bars, place));
                asm volatile("st.shared.u64 [%0], %1;\n" ::"r"(s.bars + 2 * RING * 8), "l"(q + 1ll) : "memory");
            }
            src += words;
            if (++place == s.places) {
                place = 0;
                ++turn;
            }
        }
    }
    return true;
}

// A group's factors are read into registers before any of its results is
// stored, which would order the reads behind the chain.  f: the field's byte
// offset into the block's dynamic shared memory.  Returns false if a copy
// did not come within the second of MBAR_TRIES; it then waits for no other, and
// what it leaves in the field is of no use.
template <bool PIV, bool WIDE, int W>
__device__ __noinline__ bool tile_solve(const FactorStream s, int f) {
    extern __shared__ __align__(128) unsigned char step_sm[];
    constexpr int FR = ft_fwd_rows(PIV), BR = ft_back_rows(WIDE), KU = BR - 2, GB = group_back(WIDE);
    static_assert(GF * FR * W * 8 <= group_bytes(W) && GB * BR * W * 8 <= group_bytes(W) && (KU + 1) % GB == 0, "group size");
    const int lane = threadIdx.x & 31, N = s.N;
    const unsigned base = (unsigned)__cvta_generic_to_shared(step_sm);
    const double *rd = reinterpret_cast<const double *>(step_sm + (s.ring - base)) + (W == 16 ? lane >> 1 : lane >> 2);
    const unsigned fl = base + f + lane * 8;
    int place = 0, left = 0;
    unsigned par = 0;
    int tries = MBAR_TRIES;
    if (s.g < 1) return false;
    const double *col = rd;
    auto next = [&](int group) {  // the next group's factors
        if (left == 0) {
            mbar_wait(bar_full(s.bars, place), par, tries);
            col = rd + place * s.g * (group_bytes(W) / 8);
            left = s.g;
        } else {
            col += group;
        }
    };
    // they have been used; at a chunk's end its place is handed back to the
    // asynchronous copies, which only the proxy fence orders after the reads
    // (handed back with the reads still in flight, a refill overtook them)
    auto done = [&](bool sweep_over) {
        if (--left == 0 || sweep_over) {
            left = 0;
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_empty(s.bars, place));
            if (++place == s.places) {
                place = 0;
                par ^= 1;
            }
        }
    };
    {
        double w[KL + 1];
#pragma unroll
        for (int r = 0; r <= KL; ++r) w[r] = lds_if(fl + r * 256, true);
        unsigned fj = fl;
#pragma unroll 1
        for (int j0 = 0; j0 < N; j0 += GF, fj += GF * 256) {
            next(GF * FR * W);
            double L[GF][FR];
#pragma unroll
            for (int c = 0; c < GF; ++c)
#pragma unroll
                for (int r = 0; r < FR; ++r) L[c][r] = col[(c * FR + r) * W];
#pragma unroll
            for (int c = 0; c < GF; ++c) {  // columns past N-1: nothing of them is stored
                const double ahead = lds_if(fj + (c + KL + 1) * 256, j0 + c + KL + 1 < N);
                if (PIV) pivot_swap(w, __double2loint(L[c][FR - 1]));
                const double b = w[0];
                sts_if(fj + c * 256, b, j0 + c < N);
#pragma unroll
                for (int r = 1; r <= KL; ++r) w[r - 1] = fma(-L[c][r - 1], b, w[r]);  // L zero beyond row N-1
                w[KL] = ahead;
            }
            done(j0 + GF >= N);
        }
    }
    {
        double v[KU + 1];
        unsigned fj = fl + (N - 1) * 256;
#pragma unroll
        for (int r = 0; r <= KU; ++r) v[r] = lds_if(fj - r * 256, true);
#pragma unroll 1
        for (int j0 = N - 1; j0 >= 0; j0 -= KU + 1, fj -= (KU + 1) * 256) {
#pragma unroll
            for (int h = 0; h < (KU + 1) / GB; ++h) {
                if (h > 0 && j0 - h * GB < 0) break;
                next(GB * BR * W);
                double U[GB][BR];
#pragma unroll
                for (int c = 0; c < GB; ++c)
#pragma unroll
                    for (int r = 0; r < BR; ++r) U[c][r] = col[(c * BR + r) * W];
#pragma unroll
                for (int cc = 0; cc < GB; ++cc) {
                    const int c = h * GB + cc;
                    const double ahead = lds_if(fj - (c + KU + 1) * 256, j0 - c - KU - 1 >= 0);
                    const double x = fma(v[0], U[cc][0], v[0] * U[cc][1]);
                    sts_if(fj - c * 256, x, j0 - c >= 0);
#pragma unroll
                    for (int r = 1; r <= KU; ++r) v[r - 1] = fma(-x, U[cc][r + 1], v[r]);  // U zero above row 0
                    v[KU] = ahead;
                }
                done(j0 - (h + 1) * GB < 0);
            }
        }
    }
    __syncwarp();
    return tries > 0;
}

// ------------------------------------------------------------------ tiles
// The mode of a slot of a tile: the pipe's first tiles (wide) hold 16
// consecutive k of m = 0, the others k and -k of 8 consecutive (m, k >= 0),
// m >= 1, in slots 2i and 2i+1.  Returns false for an idle slot.
__device__ __forceinline__ bool tile_mode(const Geo &g, int tile, int slot, int &nh, int &k, int &m) {
    const int nz = pf_mean_tiles(g);
    if (tile < nz) {
        m = 0;
        nh = k = tile * 16 + slot;
        return k < g.K;
    }
    const int it = (tile - nz) * 8 + (slot >> 1);
    m = 1 + it / g.K;
    k = it - (m - 1) * g.K;
    const bool twin = slot & 1;
    if (twin) k = -k;
    nh = m * (2 * g.K - 1) + k;
    return m < g.M && !(twin && k == 0);
}

__device__ __forceinline__ double sq(double2 a) { return fma(a.x, a.x, __dmul_rn(a.y, a.y)); }
// max that keeps a NaN (fmax drops it): a state gone non-finite shows as a
// NaN corrector error instead of a converged one
__device__ __forceinline__ double nanmax(double a, double b) { return (b > a || b != b) ? b : a; }

// A radial band in shared memory, ten doubles a row: the nine weights of rows
// js .. js+8, js = row_start(n), zeros outside the band, and a power of r.
// The window never leaves the field, so a product has no bounds to test, and a
// row is five 16-byte reads that half a warp shares; read from global memory
// (L2: the blocks' shared memory leaves little L1) with the bounds of each
// entry, the rows were most of the instructions of the stages and what they
// waited for (N=64, 12113 modes: 176 -> 163 us).
static constexpr int STEP_ROW = 2 * 10 * 8;  // bytes a radial point of the two tables
__device__ __forceinline__ int row_start(int n, int N) { return min(max(n - KL, 0), N - NBAND); }
struct BandRow {
    double w[NBAND + 1];
    __device__ __forceinline__ explicit BandRow(const double *tab, int n) {
        const double2 *t = reinterpret_cast<const double2 *>(tab + n * 10);
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            const double2 v = t[i];
            w[2 * i] = v.x;
            w[2 * i + 1] = v.y;
        }
    }
    __device__ __forceinline__ double power() const { return w[NBAND]; }
    // sum_j band(n, j) x(j), j ascending, x a field at this thread's slot
    __device__ __forceinline__ double2 apply(int js, const double2 *x) const {
        double2 acc = make_double2(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < NBAND; ++i) {
            const double2 v = x[js * 16 + i * 16];
            acc.x = fma(w[i], v.x, acc.x);
            acc.y = fma(w[i], v.y, acc.y);
        }
        return acc;
    }
};
static_assert(NBAND == 9, "rows of ten doubles");

// Dynamic shared memory of a block: StepHead, the rows of the radial Laplacian
// (with r^-2) and derivative (r^-1), four fields b0..b3 of [N][16]
// double2, the pressure ring of `ppe` bytes, then three Helmholtz rings of
// `ld` bytes each if there is room for them (`apart`); else these share b3
// and the pressure ring, once both are done with.
struct StepHead {
    StreamBars bars[4];    // LNp, LDp, LDm, LDz
    double ainv[16][17];   // 4x4 inverse per slot
    double coef[8][16];    // aR(1..4), aI(1..4) per slot
    double flux;           // 2 int uz r dr of the mean mode
    double wmax[8];
};
static constexpr int STEP_HEAD = 3584;
static_assert(sizeof(StepHead) <= STEP_HEAD, "block header");
struct StepSmem {
    int ppe, ld, apart;
    int far;  // the launch's own tiles work on more than L2 holds (a batch's other groups, beside it, not counted)
};

// 16 slots by NT/16 row groups; W = 16: a tile of m = 0.  Products that feed
// sums are written as fma or rounded products, so every instantiation rounds
// alike and a pipe steps bit for bit the same alone and in a batch.  Each stage reads
// the rows it needs of other threads from fields nobody writes in that stage,
// so a stage is one short loop over the thread's rows and one barrier; fully
// unrolled rows held in registers took twice as long, waiting for instructions.
// CHAIN: launched behind the transforms (chain_wait), whose output and u are
// asked for after the parts that only the matrices decide.
template <int NT, int W, bool CHAIN>
__device__ __forceinline__ void step_tile(const StepArgs &a, int tile, const StepSmem lay) {
    extern __shared__ __align__(128) unsigned char step_sm[];
    StepHead &hd = *reinterpret_cast<StepHead *>(step_sm);
    constexpr int NR = NT / 16;
    const Geo &g = a.g;
    const int N = g.N, nz = pf_mean_tiles(g);
    const size_t Hp = g.Hp;
    const int slot = threadIdx.x & 15, ty = threadIdx.x >> 4, warp = threadIdx.x >> 5;
    // six of the warps take turns, tile by tile, at solving a system (roles 0
    // to 2, and 0 the pressure) and at filling its ring (3 to 5): a warp's
    // number decides the scheduler it runs on
    static_assert(NT >= 192, "a solving and a filling warp for each system");
    const int role = warp < 6 ? (warp + tile) % 6 : 6;
    const bool lane0 = (threadIdx.x & 31) == 0;
    const int fields = STEP_HEAD + N * STEP_ROW;
    double *const lap = reinterpret_cast<double *>(step_sm + STEP_HEAD), *const der = lap + N * 10;
    double2 *const b0 = reinterpret_cast<double2 *>(step_sm + fields) + slot;
    double2 *const b1 = b0 + N * 16, *const b2 = b1 + N * 16, *const b3 = b2 + N * 16;
    const unsigned sbase = (unsigned)__cvta_generic_to_shared(step_sm);
    int nh, k, m;
    const bool live = tile_mode(g, tile, slot, nh, k, m);
    if (!live) nh = 0;
    if (threadIdx.x == 0) {
        for (int s = 0; s < 4; ++s) {
            hd.bars[s].asked = 0;
            for (int i = 0; i < 2 * RING; ++i)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(sbase + s * (int)sizeof(StreamBars) + i * 8) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    // u_r, u_theta, u_z of the tile into b0, b3, b1
    auto load_u = [&]() {
        for (int n = ty; n < N; n += NR) {
            const int e = n * 16;
            if (live) {
                const size_t at = (size_t)n * Hp + nh;
                cp_async16((unsigned)__cvta_generic_to_shared(b0 + e), a.u_[0] + at);
                cp_async16((unsigned)__cvta_generic_to_shared(b3 + e), a.u_[1] + at);
                cp_async16((unsigned)__cvta_generic_to_shared(b1 + e), a.u_[2] + at);
            } else {
                b0[e] = b1[e] = b3[e] = make_double2(0.0, 0.0);
            }
        }
    };
    if (!CHAIN) load_u();
    // the factor streams; those whose rings are free now are started
    const size_t ftile = (size_t)(W == 16 ? 16 * tile : 8 * (tile + nz)) * N * FT_ROWS;
    auto stream = [&](int sys) {  // 0: LNp, 1..3: LDp, LDm, LDz
        FactorStream s;
        s.N = N;
        s.W = W;
        s.ft = (sys == 0 ? a.lnp : pick3(a.ld, sys - 1)) + ftile;
        s.flags = sys == 0 ? 3 : pick3(a.ldpiv, sys - 1);
        const int bytes = sys == 0 ? lay.ppe : lay.ld;
        s.ring = sbase + fields + N * 1024;
        if (sys > 0) s.ring += (lay.apart ? lay.ppe : -N * 256) + (sys - 1) * lay.ld;
        s.places = bytes >= RING * group_bytes(W) ? RING : 2;
        s.g = bytes / (s.places * group_bytes(W));
        s.bars = sbase + sys * (int)sizeof(StreamBars);
        return s;
    };
    bool ok = true;
    __syncthreads();  // the barriers are there
    if (lane0 && (role == 0 || (lay.apart && role >= 3 && role < 6))) {
        const FactorStream s = stream(role == 0 ? 0 : role - 2);
        ok = stream_fill(s, 0, s.places);
    }
    for (int i = threadIdx.x; i < 256; i += NT) {
        int h, kk, mm;
        if (tile_mode(g, tile, i & 15, h, kk, mm)) hd.ainv[i & 15][i >> 4] = h != 0 ? a.Ainv[(size_t)(i >> 4) * Hp + h] : 0.0;
    }
    const double *__restrict__ rp = a.dm.rp;
    for (int i = threadIdx.x; i < 20 * N; i += NT) {  // the rows, column by column
        const int c = i / N, n = i - c * N, t = c >= 10, j = row_start(n, N) + c - 10 * t;
        const bool in = j >= n - KL && j <= n + KL;
        const double *__restrict__ src = c == 9 || c == 19 ? rp + (t ? 2 : 1) * N + n : (t ? a.dm.dr : a.dm.radLap) + (in ? (KL + n - j) * N + j : 0);
        lap[(t * N + n) * 10 + c - 10 * t] = in || c == 9 || c == 19 ? __ldg(src) : 0.0;
    }
    const double mMp = (double)(m * g.Mp), kal = g.alpha * k, c2 = a.c2;
    // diagonal of Lt for the uz system at row n: c1 - c2 ((m Mp)^2/r^2 + (alpha k)^2)
    const double mm2 = __dmul_rn(mMp, mMp), kk2 = __dmul_rn(kal, kal);
    auto diag0 = [&](double r2) { return fma(-c2, fma(mm2, r2, kk2), a.c1); };
    // N of one component at one row, and N_ in the corrector: the loads of the
    // next row (of the next component after the last) are in flight while one
    // is worked on; each value is read once: streamed past L1
    double2 vN = make_double2(0.0, 0.0), vP = vN;
    auto load_N = [&](int c, int n) {
        if (!live || n >= N) return;
        const size_t at = (size_t)n * Hp + nh;
        vN = __ldcs(pick3(a.Nl, c) + at);
        if (a.mode == 1) vP = __ldcs(pick3(a.N_, c) + at);
    };
    if (CHAIN) {
        chain_wait();
        load_u();
    }
    load_N(2, ty);
    cp_async_wait_all();
    __syncthreads();
    // st 0: rhs of uz, b1 -> b2; st 1: the off-diagonal part of Lt u_r plus
    // N_r, b0 -> b1; st 2: the same of u_theta (b3), then the u+ and u-
    // right-hand sides b0, b1
#pragma unroll 1
    for (int st = 0; st < 3; ++st) {
        const int comp = st == 0 ? 2 : st - 1;
        const double2 *src = st == 0 ? b1 : st == 1 ? b0 : b3;
#pragma unroll 1
        for (int n = ty; n < N; n += NR) {
            double2 v = vN;
            const double2 P = vP;
            const bool last = n + NR >= N;
            if (!last || st < 2) load_N(last ? st : comp, last ? ty : n + NR);
            const BandRow row(lap, n);
            const double2 s = row.apply(row_start(n, N), src);
            const double r2 = row.power(), d = diag0(r2);
            if (a.mode == 1) {  // N = c N + (1-c) N_
                const double d1 = a.implicit, d2 = 1.0 - a.implicit;
                v = make_double2(fma(d1, v.x, __dmul_rn(d2, P.x)), fma(d1, v.y, __dmul_rn(d2, P.y)));
            }
            if (live) (a.mode == 1 ? pick3(a.Nl, comp) : pick3(a.N_, comp))[(size_t)n * Hp + nh] = v;
            v = make_double2(fma(c2, s.x, v.x), fma(c2, s.y, v.y));
            if (st == 0) {
                const double2 x = b1[n * 16];
                b2[n * 16] = make_double2(fma(d, x.x, v.x), fma(d, x.y, v.y));
            } else if (st == 1) {
                b1[n * 16] = v;
            } else {
                const double2 ar = b1[n * 16], x = b0[n * 16], y = b3[n * 16];
                // the u+- systems' diagonals: -1/r^2 -+ 2 m Mp/r^2 beyond that of uz
                const double t = __dmul_rn(2.0 * mMp, r2);
                const double dp = fma(-c2, __dadd_rn(r2, t), d), dm = fma(-c2, __dsub_rn(r2, t), d);
                b0[n * 16] = make_double2(fma(dp, x.x - y.y, ar.x - v.y), fma(dp, x.y + y.x, ar.y + v.x));
                b1[n * 16] = make_double2(fma(dm, x.x + y.y, ar.x + v.y), fma(dm, x.y - y.x, ar.y - v.x));
            }
        }
        __syncthreads();
    }
    // the last stage's reads, brought to L2 under the solves where they come
    // from DRAM (64 pipes, N=64: 254 -> 247 us, N=32: 190 -> 181); from L2 they
    // are quick enough, and asking costs more (N=48, 2985 modes: 40 -> 43).
    // The slots at the ends of a row's runs cover its lines.
    if (lay.far && live && nh != 0 && (slot < 2 || slot >= 14 || (W == 16 && slot == 8)))
        for (int n = ty; n < N; n += NR) {
            const size_t at = (size_t)n * Hp + nh;
            if (k >= 0)
#pragma unroll
                for (int i = 0; i < 6; ++i) prefetch_l2(a.U + (size_t)i * N * Hp + at);
            if (a.mode == 1)
#pragma unroll
                for (int c = 0; c < 3; ++c) prefetch_l2(a.u[c] + at);
        }
    // div(pm2rt(rhs)) (velocity.f90:98-114; variables.f90:472-477) with
    // tim_zerobc: b0, b1, b2 -> b3
#pragma unroll 1
    for (int n = ty; n < N; n += NR) {
        const BandRow row(der, n);
        double2 dv = make_double2(0.0, 0.0);
        if (n != 0 && n != N - 1) {
            double2 s = make_double2(0.0, 0.0);
#pragma unroll 1
            for (int f = 0; f < 2; ++f) {
                const double2 e = row.apply(row_start(n, N), f ? b1 : b0);
                s.x += e.x;
                s.y += e.y;
            }
            const double rm1 = row.power(), m1r1 = rm1 * mMp;
            const double2 p = b0[n * 16], q = b1[n * 16], z = b2[n * 16];
            const double tx = 0.5 * (p.y - q.y), ty_ = -0.5 * (p.x - q.x);
            dv.x = fma(-z.y, kal, fma(-ty_, m1r1, fma(0.5 * (p.x + q.x), rm1, 0.5 * s.x)));
            dv.y = fma(z.x, kal, fma(tx, m1r1, fma(0.5 * (p.y + q.y), rm1, 0.5 * s.y)));
        }
        b3[n * 16] = dv;
    }
    __syncthreads();
    // LNp of k = m = 0 is held as zeros, so its pressure is zero (timestep.f90:110-113)
    if (role == 0) {
        ok &= tile_solve<true, true, W>(stream(0), fields + 3 * N * 256);
    } else if (role == 3 && lane0) {
        ok &= stream_fill(stream(0), stream(0).places, 1 << 30);
    }
    ok = !__syncthreads_or(!ok);
    // rhs - rt2pm(grad p), grad p = (dr p, i m/r p, i alpha k p); zero boundary rows
#pragma unroll 1
    for (int n = ty; n < N; n += NR) {
        const int e = n * 16;
        const BandRow row(der, n);
        if (n == 0 || n == N - 1) {
            b0[e] = b1[e] = b2[e] = make_double2(0.0, 0.0);
            continue;
        }
        const double2 s = row.apply(row_start(n, N), b3);
        const double2 pv = b3[e];
        const double m1r1 = row.power() * mMp;
        const double2 vp = b0[e], vm = b1[e], vz = b2[e];
        b0[e] = make_double2(vp.x - fma(-pv.x, m1r1, s.x), vp.y - fma(-pv.y, m1r1, s.y));
        b1[e] = make_double2(vm.x - fma(pv.x, m1r1, s.x), vm.y - fma(pv.y, m1r1, s.y));
        b2[e] = make_double2(fma(pv.y, kal, vz.x), fma(-pv.x, kal, vz.y));
    }
    // b3 and the pressure ring, written by ordinary stores and read by loads
    // so far, may now take asynchronous copies
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    if (!ok) {
        // no more waits
    } else if (role < 3) {
        const FactorStream s = stream(1 + role);
        const int f = fields + role * N * 256;
        if (s.flags == 0) ok &= tile_solve<false, false, W>(s, f);
        else if (s.flags == 1) ok &= tile_solve<true, false, W>(s, f);
        else ok &= tile_solve<true, true, W>(s, f);  // low Re, small dt or very clustered meshes
    } else if (role < 6 && lane0) {
        const FactorStream s = stream(role - 2);
        ok &= stream_fill(s, lay.apart ? s.places : 0, 1 << 30);
    }
    if (__syncthreads_or(!ok)) {
        // reported to the host; the copies still on their way must not land in
        // the shared memory of a block after this one
        if (threadIdx.x == 0) {
            atomicCAS(&a.sc->info, 0, PF_STEP_STUCK);
            int tries = MBAR_TRIES;
#pragma unroll 1
            for (int sys = 0; sys < 4; ++sys) {
                const FactorStream s = stream(sys);
                const int n = (int)*(volatile long long *)&hd.bars[sys].asked;
#pragma unroll 1
                for (int q = max(0, n - s.places); q < n; ++q)
                    mbar_wait(bar_full(s.bars, q % s.places), q / s.places & 1, tries);
            }
        }
        __syncthreads();
    }
    if (threadIdx.x < 16 && live) {
        // vel_evalBC + a = -A^-1 B (velocity.f90:239-243, 262-298)
        const int e = (N - 1) * 16;
        const double2 pw = b0[e], qw = b1[e], zw = b2[e];
        const double urRe = 0.5 * (pw.x + qw.x), urIm = 0.5 * (pw.y + qw.y);
        const double utRe = 0.5 * (pw.y - qw.y), utIm = -0.5 * (pw.x - qw.x);
        double drRe = 0.0, drIm = 0.0;
#pragma unroll
        for (int j = 0; j <= KL; ++j) {
            const int ej = (N - 1 - KL + j) * 16;
            const double w = a.dm.dr1[1 * (KL + 1) + j];
            const double2 x = b0[ej], y = b1[ej];
            drRe = fma(w, x.x + y.x, drRe);
            drIm = fma(w, x.y + y.y, drIm);
        }
        drRe = 0.5 * drRe;
        drIm = 0.5 * drIm;
        const double d = rp[2 * N + (N - 1)];
        const double dm_ = __dmul_rn(d, mMp);
        const double BRe[4] = {pw.x, qw.x, -zw.y, fma(-kal, zw.y, fma(-dm_, utIm, fma(urRe, d, drRe)))};
        const double BIm[4] = {pw.y, qw.y, zw.x, fma(kal, zw.x, fma(dm_, utRe, fma(urIm, d, drIm)))};
        for (int i = 0; i < 4; ++i) {
            double sr = 0.0, si = 0.0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                sr = fma(hd.ainv[slot][i * 4 + j], BRe[j], sr);
                si = fma(hd.ainv[slot][i * 4 + j], BIm[j], si);
            }
            hd.coef[i][slot] = -sr;
            hd.coef[4 + i][slot] = -si;
        }
    }
    if (W == 16 && tile == 0 && warp == 1) {  // the tile of k = m = 0 (slot 0)
        const double2 *z = reinterpret_cast<const double2 *>(step_sm + fields) + 2 * N * 16;
        double s = 0.0;
        for (int n = threadIdx.x & 31; n < N; n += 32) s = fma(z[n * 16].x, a.dm.intrdr[n], s);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((threadIdx.x & 31) == 0) hd.flux = 2.0 * s;
    }
    __syncthreads();
    double err = 0.0;
    if (live) {
        double cf[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) cf[i] = hd.coef[i][slot];
        // U of (k, m) and (-k, m): equal but for the sign of the last vector,
        // which the gradient's i alpha k gives; both read the k >= 0 column
        const double *__restrict__ Uc = a.U + (k < 0 ? nh - 2 * k : nh);
        const double sg = k < 0 ? -1.0 : 1.0;
        double2 *__restrict__ u0 = a.u[0] + nh;
        double2 *__restrict__ u1 = a.u[1] + nh;
        double2 *__restrict__ u2 = a.u[2] + nh;
        const size_t NH = (size_t)N * Hp;
        const bool zero = nh == 0;
        const double d3 = (zero && a.const_flux) ? -hd.flux / a.sc->flux_d1 : 0.0;
#pragma unroll 2
        for (int n = ty; n < N; n += NR) {
            const size_t at = (size_t)n * Hp;
            double Uv[6];
#pragma unroll
            for (int i = 0; i < 6; ++i) Uv[i] = zero ? 0.0 : Uc[i * NH + at];
            double2 o[3];
            if (a.mode == 1) {  // read once, overwritten below: stream past L1
                o[0] = __ldcs(u0 + at);
                o[1] = __ldcs(u1 + at);
                o[2] = __ldcs(u2 + at);
            }
            double2 rr = b0[n * 16], tt = b1[n * 16], zz = b2[n * 16];
            Uv[5] = sg * Uv[5];
            rr.x = fma(cf[0], Uv[0], rr.x); rr.y = fma(cf[4], Uv[0], rr.y);
            tt.x = fma(cf[1], Uv[1], tt.x); tt.y = fma(cf[5], Uv[1], tt.y);
            zz.x = fma(-cf[6], Uv[2], zz.x); zz.y = fma(cf[2], Uv[2], zz.y);
            rr.x = fma(cf[3], Uv[3], rr.x); rr.y = fma(cf[7], Uv[3], rr.y);
            tt.x = fma(cf[3], Uv[4], tt.x); tt.y = fma(cf[7], Uv[4], tt.y);
            zz.x = fma(-cf[7], Uv[5], zz.x); zz.y = fma(cf[3], Uv[5], zz.y);
            double2 ur = make_double2(0.5 * (rr.x + tt.x), 0.5 * (rr.y + tt.y));
            double2 ut = make_double2(0.5 * (rr.y - tt.y), -0.5 * (rr.x - tt.x));
            if (zero) {  // flux adjustment and symmetry zeros of the mean mode
                ur = make_double2(0.0, 0.0);
                ut.y = 0.0;
                zz = make_double2(a.const_flux ? fma(d3, a.Ui[n], zz.x) : zz.x, 0.0);
            }
            if (a.mode == 1) {
                err = nanmax(err, sq(make_double2(o[0].x - ur.x, o[0].y - ur.y)));
                err = nanmax(err, sq(make_double2(o[1].x - ut.x, o[1].y - ut.y)));
                err = nanmax(err, sq(make_double2(o[2].x - zz.x, o[2].y - zz.y)));
            }
            u0[at] = ur;
            u1[at] = ut;
            u2[at] = zz;
            b0[n * 16] = ur;
            b1[n * 16] = ut;
            b2[n * 16] = zz;
        }
        if (zero && ty == 0 && a.const_flux) a.sc->Pr0 = a.sc->Pr0 + d3 * g.Re / 4.0;
    }
    if (a.mode == 0 && a.curl[0]) {
        // curl(u) and the mean mode's sums over this tile (k_nl_prep's, while
        // u is still on the chip)
        __syncthreads();
#pragma unroll 1
        for (int n = ty; n < ((N + 1) & ~1); n += NR) {  // whole warps: the half-warps sum together
            const BandRow row(der, min(n, N - 1));
            double s[3] = {0.0, 0.0, 0.0};
            if (live && n < N) {
                const size_t at = (size_t)n * Hp + nh;
                const int js = row_start(n, N);
                const double2 dt = row.apply(js, b1), dz = row.apply(js, b2);
                const double2 ur = b0[n * 16], ut = b1[n * 16], uz = b2[n * 16];
                const double rm1 = row.power();
                const Curl c = mode_curl(ur, ut, uz, dt, dz, rm1, rm1 * mMp, kal);
                if (a.mixed) {
                    reinterpret_cast<float2 *>(a.curl[0])[at] = make_float2((float)c.r.x, (float)c.r.y);
                    reinterpret_cast<float2 *>(a.curl[1])[at] = make_float2((float)c.t.x, (float)c.t.y);
                    reinterpret_cast<float2 *>(a.curl[2])[at] = make_float2((float)c.z.x, (float)c.z.y);
                    mean_terms(nh == 0, ur, ut, uz, c, s);
                } else {
                    reinterpret_cast<double2 *>(a.curl[0])[at] = c.r;
                    reinterpret_cast<double2 *>(a.curl[1])[at] = c.t;
                    reinterpret_cast<double2 *>(a.curl[2])[at] = c.z;
                }
            }
            if (a.mixed) {
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    for (int o = 8; o > 0; o >>= 1) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
                if (slot == 0 && n < N)
                    for (int q = 0; q < 3; ++q) a.mpart[((size_t)tile * N + n) * 3 + q] = s[q];
            }
        }
    }
    if (a.mode == 1) {
        // one atomic per block; the pipe's last block publishes the maximum
        // and clears the accumulator for the next corrector
        for (int o = 16; o > 0; o >>= 1) err = nanmax(err, __shfl_xor_sync(0xffffffffu, err, o));
        if ((threadIdx.x & 31) == 0) hd.wmax[warp] = err;
        __syncthreads();
        if (threadIdx.x == 0) {
            double e = hd.wmax[0];
            for (int i = 1; i < NT / 32; ++i) e = nanmax(e, hd.wmax[i]);
            atomicMax(&a.sc->dterr2_acc, (unsigned long long)__double_as_longlong(e));
            __threadfence();
            if (atomicAdd(&a.sc->tiles_done, 1) == pf_step_tiles(g) - 1) {
                a.sc->dterr2_bits = atomicExch(&a.sc->dterr2_acc, 0ull);
                a.sc->tiles_done = 0;
            }
        }
    }
}

// ------------------------------------------------------------- kernels
// Lone pipe: the m = 0 tiles and the paired tiles in one launch.  Batch: one
// launch per kind of tile and radial size over the tiles of every such pipe,
// blk[b] = (pipe, tile).  MINB: resident blocks per SM that shared memory
// allows at that size and the registers are capped for.
template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_step(const __grid_constant__ StepArgs a, const StepSmem lay) {
    if ((int)blockIdx.x < pf_mean_tiles(a.g)) step_tile<NT, 16, true>(a, blockIdx.x, lay);
    else step_tile<NT, 8, true>(a, blockIdx.x, lay);
}

template <int NT, int MINB, int W>
__global__ void __launch_bounds__(NT, MINB) k_step_batch(const StepArgs *__restrict__ args, const int2 *__restrict__ blk,
                                                         const StepSmem lay, const int *__restrict__ act) {
    const int2 pb = blk[blockIdx.x];
    if (act && !act[pb.x]) return;
    const StepArgs a = args[pb.x];  // by value: stores through its pointers cannot alias it
    step_tile<NT, W, false>(a, pb.y, lay);
}

// ------------------------------------------------------------------ host
// (N limit, threads, resident blocks): shared memory, 1.2 KB a radial point
// plus the rings, allows that many blocks
#define PF_STEP_SHAPES(X) X(32, 192, 4) X(64, 256, 2) X(128, 256, 1)

// The rings when `blocks` blocks are to share an SM: what their fields leave
// free, at least two groups of 16 matrices.  The Helmholtz rings lie apart
// from the fields where each then has two groups a chunk, or half a sweep:
// a block alone on its SM has its whole factors in flight from the start.
static constexpr size_t SM_SMEM = 228 * 1024;
// `tiles` of 16 modes read and write about 470 bytes a mode and radial point.
static StepSmem step_rings(int N, int blocks, size_t tiles) {
    const int room = (int)std::min(SM_SMEM / blocks - 1024, (size_t)227 * 1024) - STEP_HEAD - N * (1024 + STEP_ROW);
    const int unit = RING * group_bytes(8);  // one group a chunk for W = 8
    const int half = 2 * ((N + 19) / 20);    // groups of half a forward sweep, an even number
    StepSmem l{};
    l.far = tiles * 16 * N * 470 > ((size_t)126 << 20);
    const int each = std::min(room / 4 / unit, half);
    l.apart = each >= std::min(2, half);
    l.ppe = std::max(l.apart ? each : room / unit, 1) * unit;
    // a stream needs two chunks of a group of 16 matrices: fewer blocks then fit
    if (!l.apart) l.ppe = std::max(l.ppe, (3 * (2 * group_bytes(16) + 128) - N * 256 + 127) & ~127);
    l.ld = l.apart ? l.ppe : ((N * 256 + l.ppe) / 3) & ~127;
    return l;
}
static size_t step_smem(int N, const StepSmem &l) {
    return (size_t)STEP_HEAD + N * (1024 + STEP_ROW) + l.ppe + (l.apart ? 3 * l.ld : 0);
}

// leave_curl: the fused transforms follow and read curl(u)
static StepArgs make_step_args(const pf_ctx *ctx, int corrector, bool leave_curl) {
    StepArgs a;
    for (int i = 0; i < 3; ++i) {
        a.u_[i] = ctx->prev[i].d;
        a.Nl[i] = ctx->vel[3 + i].d;
        a.N_[i] = ctx->prev[3 + i].d;
        a.u[i] = ctx->vel[i].d;
    }
    const pf_lumesh *ld[3] = {&ctx->LDp, &ctx->LDm, &ctx->LDz};
    a.lnp = ctx->LNp.tiles;
    for (int i = 0; i < 3; ++i) {
        a.ld[i] = ld[i]->tiles;
        a.ldpiv[i] = ld[i]->pivoted;
    }
    leave_curl = leave_curl && pf_nl_fused_supported(ctx);
    for (int i = 0; i < 3; ++i) a.curl[i] = leave_curl ? pf_curl_field(ctx, i) : nullptr;
    a.mixed = ctx->cfg.precision == PF_PREC_MIXED;
    a.mpart = ctx->mpart;
    a.U = ctx->U;
    a.Ainv = ctx->Ainv;
    a.Ui = ctx->Ui;
    a.dm = ctx->dm;
    a.g = ctx->g;
    a.c1 = ctx->Ltz.c1;
    a.c2 = ctx->Ltz.c2;
    a.implicit = ctx->cfg.implicit;
    a.mode = corrector;
    a.const_flux = ctx->cfg.const_flux;
    a.sc = ctx->dsc;
    return a;
}

bool pf_fused_step_ok(const pf_ctx *ctx) { return ctx->g.N <= STEP_MAX_N; }

// One predictor (corrector=0) or corrector (corrector=1) vel_step.  The
// predictor's u_ := u copy is a pointer swap of vel[0..2] and prev[0..2]; what
// it was given to leave is noted for pf_next_nonlinear.
int pf_vel_step_fused(pf_ctx *ctx, int corrector, bool leave_curl) {
    const Geo &g = ctx->g;
    if (!pf_fused_step_ok(ctx)) {
        pf_set_error("fused step supports N <= %d", STEP_MAX_N);
        return PF_ERR_ARG;
    }
    if (!corrector) {
        for (int i = 0; i < 3; ++i) std::swap(ctx->vel[i].d, ctx->prev[i].d);
        ctx->parity ^= 1;
    }
    const StepArgs a = make_step_args(ctx, corrector, leave_curl);
    ctx->curl_left = !corrector && a.curl[0];
    const int blocks = pf_step_tiles(g);
    {
        ProfScope ps_(ctx, PF_K_STEP);
#define PF_CASE(NMAX, NT, MINB)                                             \
    else if (g.N <= NMAX) {                                                 \
        const StepSmem lay = step_rings(g.N, MINB, blocks);                         \
        const size_t sm = step_smem(g.N, lay);                              \
        PF_TRY(pf_raise_smem((const void *)k_step<NT, MINB>, sm));          \
        PF_CUDA(launch_chained(k_step<NT, MINB>, dim3(blocks), NT, sm, ctx->stream, a, lay)); \
    }
        if (blocks <= ctx->sms) {  // a block to an SM: all its threads and shared memory for latency
            const StepSmem lay = step_rings(g.N, 1, blocks);
            const size_t sm = step_smem(g.N, lay);
            PF_TRY(pf_raise_smem((const void *)k_step<256, 1>, sm));
            PF_CUDA(launch_chained(k_step<256, 1>, dim3(blocks), 256, sm, ctx->stream, a, lay));
        }
        PF_STEP_SHAPES(PF_CASE)
#undef PF_CASE
    }
    PF_LAUNCHED(ctx);
    return PF_OK;
}

// ---------------------------------------------------------------- batched
// Step arguments of every pipe for both pointer parities and both modes,
// and one (pipe, tile) map per radial size and kind of tile.  The m = 0 tiles
// launch by themselves: they hold sixteen factor columns instead of eight.  The launches are
// independent and run concurrently, forked onto auxiliary streams.
namespace {
struct StepGroup {
    int N, W;  // radial points; 16: m = 0 tiles, 8: paired tiles
    int2 *blk;
    int nblk;
};
}  // namespace
struct pf_step_batch {
    void *mem;               // the argument records, then the maps
    StepArgs *d_args[2][2];  // [pointer state after the predictor's swap][mode]
    std::vector<StepGroup> groups;
    pf_aux *aux;
};

void pf_step_batch_free(pf_step_batch *b) {
    if (!b) return;
    cudaFree(b->mem);
    delete b;
}

static int step_batch_fill(pf_step_batch *b, pf_ctx *const *pipes, int n) {
    std::vector<StepArgs> args;
    for (int s = 0; s < 2; ++s)
        for (int m = 0; m < 2; ++m)
            for (int i = 0; i < n; ++i) {
                pf_ctx *c = pipes[i];
                if (s) for (int k = 0; k < 3; ++k) std::swap(c->vel[k].d, c->prev[k].d);
                args.push_back(make_step_args(c, m, true));
                if (s) for (int k = 0; k < 3; ++k) std::swap(c->vel[k].d, c->prev[k].d);
            }
    std::vector<int> sizes;
    for (int i = 0; i < n; ++i) sizes.push_back(pipes[i]->g.N);
    std::sort(sizes.begin(), sizes.end(), std::greater<int>());  // the longest blocks first
    sizes.erase(std::unique(sizes.begin(), sizes.end()), sizes.end());
    std::vector<int2> maps;
    std::vector<size_t> at;
    for (const int W : {16, 8})
        for (const int N : sizes) {
            const size_t from = maps.size();
            for (int i = 0; i < n; ++i) {
                const Geo &g = pipes[i]->g;
                if (g.N != N) continue;
                const int nz = pf_mean_tiles(g), all = pf_step_tiles(g);
                for (int t = W == 16 ? 0 : nz; t < (W == 16 ? nz : all); ++t) maps.push_back(make_int2(i, t));
            }
            if (maps.size() == from) continue;
            b->groups.push_back(StepGroup{N, W, nullptr, (int)(maps.size() - from)});
            at.push_back(from);
        }
    const size_t abytes = args.size() * sizeof(StepArgs);  // a multiple of 8, as the maps need
    std::vector<unsigned char> host(abytes + maps.size() * sizeof(int2));
    std::memcpy(host.data(), args.data(), abytes);
    std::memcpy(host.data() + abytes, maps.data(), maps.size() * sizeof(int2));
    PF_CUDA(cudaMalloc(&b->mem, host.size()));
    PF_CUDA(cudaMemcpy(b->mem, host.data(), host.size(), cudaMemcpyHostToDevice));
    for (int q = 0; q < 4; ++q) b->d_args[q / 2][q % 2] = reinterpret_cast<StepArgs *>(b->mem) + (size_t)q * n;
    int2 *blk = reinterpret_cast<int2 *>(reinterpret_cast<unsigned char *>(b->mem) + abytes);
    for (size_t k = 0; k < at.size(); ++k) b->groups[k].blk = blk + at[k];
    return b->aux->reserve(b->groups.size());
}

// state 0: the pointers as the pipes hold them now; state 1: vel/prev swapped
int pf_step_batch_build(pf_ctx *const *pipes, int n, pf_aux *aux, pf_step_batch **out) {
    *out = nullptr;
    for (int i = 0; i < n; ++i)
        if (!pf_fused_step_ok(pipes[i])) {
            pf_set_error("batched step supports N <= %d", STEP_MAX_N);
            return PF_ERR_ARG;
        }
    pf_step_batch *b = new pf_step_batch();
    b->aux = aux;
    const int s = step_batch_fill(b, pipes, n);
    if (s != PF_OK) {
        pf_step_batch_free(b);
        return s;
    }
    *out = b;
    return PF_OK;
}

static int step_group_launch(const StepGroup &gr, const StepArgs *a, const int *act, cudaStream_t st) {
#define PF_CASE(NMAX, NT, MINB)                                                \
    else if (gr.N <= NMAX) {                                                   \
        const StepSmem lay = step_rings(gr.N, MINB, gr.nblk);                           \
        const size_t sm = step_smem(gr.N, lay);                                \
        if (gr.W == 16) {                                                      \
            PF_TRY(pf_raise_smem((const void *)k_step_batch<NT, MINB, 16>, sm)); \
            k_step_batch<NT, MINB, 16><<<gr.nblk, NT, sm, st>>>(a, gr.blk, lay, act); \
        } else {                                                               \
            PF_TRY(pf_raise_smem((const void *)k_step_batch<NT, MINB, 8>, sm));  \
            k_step_batch<NT, MINB, 8><<<gr.nblk, NT, sm, st>>>(a, gr.blk, lay, act);  \
        }                                                                      \
    }
    if (false) {
    }
    PF_STEP_SHAPES(PF_CASE)
#undef PF_CASE
    PF_CHECK_LAUNCH();
    return PF_OK;
}

// One predictor or corrector vel_step of every pipe, one launch per group;
// the caller tracks the pointer state (the predictor's swap is the caller's).
// act: null, or the mask of the pipes to step.
int pf_step_batch_launch(pf_step_batch *b, int state, int corrector, const int *act, cudaStream_t st,
                         pf_stage_prof *prof, unsigned long long *nk) {
    const StepArgs *a = b->d_args[state][corrector ? 1 : 0];
    StageScope ss_(prof, PF_K_STEP, st);
    const size_t more = b->groups.size() - 1;
    if (more > 0) PF_CUDA(cudaEventRecord(b->aux->fork, st));
    for (size_t k = 0; k < more; ++k) PF_CUDA(cudaStreamWaitEvent(b->aux->st[k], b->aux->fork, 0));
    for (size_t k = 0; k <= more; ++k) {
        PF_TRY(step_group_launch(b->groups[k], a, act, k ? b->aux->st[k - 1] : st));
        ++*nk;
    }
    for (size_t k = 0; k < more; ++k) {
        PF_CUDA(cudaEventRecord(b->aux->join[k], b->aux->st[k]));
        PF_CUDA(cudaStreamWaitEvent(st, b->aux->join[k], 0));
    }
    return PF_OK;
}
