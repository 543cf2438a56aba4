// Per-Fourier-mode banded Helmholtz / pressure-Poisson systems on the device:
// matrix assembly with axis-parity and wall rows, banded LU with partial
// pivoting (LAPACK dgbtrf == dgbtf2 for KL=4 < block size), banded solves
// (dgbtrs), the influence-matrix precompute and correction, and the
// constant-flux adjustment (timestep.f90:46-123; velocity.f90:120-298).
//
// Storage: lu[(row*N + col)*Hp + nh] with `row` the 0-based LAPACK band row
// (diagonal at row KV), so one thread per mode reads column-major bands and
// consecutive modes are consecutive in memory.
#include <cmath>
#include "pf_internal.cuh"

#define LU(row, col) lu[((size_t)(row) * N + (col)) * Hp + nh]

// What a factorisation leaves for the host (ctx->lustat).
struct LUStat {
    int info[4];   // per set: first singular pivot (1-based column), 0 = ok
    int piv[4];    // per set: bit 0 some row was swapped, bit 1 a row of U reaches beyond KL columns
    int inv;       // influence matrices: -(nh + 1) of a singular one
};

// The sets of one launch.
struct LUJob {
    struct Set {
        double *lu;
        unsigned char *piv;
        double *tiles;
        int PM, BC;
        double c1, c2;
    } s[4];
    int n;
    LUStat *st;
};

// Assemble A = c1 I + c2 Lap(PM) with the axis-parity first row and the wall
// row, and factor it (timestep.f90:75-93; dgbtf2).  Thread = the matrix of
// (k >= 0, m) of set blockIdx.y, stored for (-k, m) as well, which has the
// same bits.  Bound by the chain of one column (pivot search, reciprocal,
// multipliers, update: about 300 cycles), so the columns the elimination can
// reach, 5 rows by 9, stay in registers, each band entry is made as its row
// enters and every element is stored once.  N = 40, the three Helmholtz sets
// of 729 modes: 49 us, 670 instructions a column in 36 warps (on the band in
// memory, one launch and one host wait per set: about 150 us each).
__global__ void __launch_bounds__(32) k_lu_factor(const LUJob job, const DevMesh dm, const Geo g) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= g.M * g.K) return;
    const LUJob::Set &A = job.s[blockIdx.y];
    const int N = g.N, Hp = g.Hp, PM = A.PM, BC = A.BC;
    const double c1 = A.c1, c2 = A.c2;
    const int m = q / g.K, k = q % g.K;
    const int S = (m * g.Mp + abs(PM)) % 2;  // axis parity (timestep.f90:82)
    const size_t at = (size_t)m * (2 * g.K - 1) + k;
    const int twin = m > 0 ? -2 * k : 0;  // from (k, m) to (-k, m)
    double *lu = A.lu + at;
    unsigned char *piv = A.piv + at;
    auto put = [&](int row, int col, double v) {
        double *o = lu + ((size_t)row * N + col) * Hp;
        *o = v;
        o[twin] = v;
    };
    double w[KL + 1][KV + 1];  // rows j.. j+KL, columns j .. j+KV
    auto entry = [&](int r, int c) {
        return lumesh_entry(dm, N, g.Mp, g.alpha, PM, BC, c1, c2, k, m, S, r, c);
    };
#pragma unroll
    for (int i = 0; i <= KL; ++i)
#pragma unroll
        for (int c = 0; c <= KV; ++c) w[i][c] = c <= i + KL ? entry(i, c) : 0.0;
    // row r > KL; loads that no branch waits for
    auto row_in = [&](int r, double (&x)[KV + 1]) {
        const int rr = min(r, N - 1);
#pragma unroll
        for (int i = 0; i <= KV; ++i) x[i] = dm.radLap[(KV - i) * N + min(rr - KL + i, N - 1)];
#pragma unroll
        for (int i = 0; i <= KV; ++i) x[i] = r - KL + i < N ? __dmul_rn(c2, x[i]) : 0.0;
        if (r < N - 1) {
            x[KL] = entry(r, r);
        } else {
#pragma unroll
            for (int i = 0; i <= KV; ++i) x[i] = r == N - 1 && i <= KL ? dm.dr1[BC * (KL + 1) + i] : 0.0;
        }
    };
    for (int c = 0; c < KV; ++c)  // storage above the first row
        for (int row = 0; row < KV - c; ++row)
            put(row, c, row >= KL ? __dmul_rn(c2, dm.radLap[(row - KL) * N + c]) : 0.0);
    const bool factor = !(BC == 1 && q == 0);  // the singular Neumann mean mode is left as it is
    int ju = 0, flags = 0;
    for (int j = 0; j < N; ++j) {
        double nx[KV + 1];
        row_in(j + KL + 1, nx);
        if (factor) {
            int jp = 0;
            double amax = fabs(w[0][0]), pv = w[0][0];
#pragma unroll
            for (int i = 1; i <= KL; ++i) {
                const double x = fabs(w[i][0]);
                if (x > amax) {
                    amax = x;
                    pv = w[i][0];
                    jp = i;
                }
            }
            piv[(size_t)j * Hp] = (unsigned char)jp;
            piv[(long long)j * Hp + twin] = (unsigned char)jp;
            if (pv != 0.0) {
                ju = max(ju, min(j + KL + jp, N - 1));
                if (jp != 0) {
                    flags |= ju > j + KL ? 3 : 1;
#pragma unroll
                    for (int i = 1; i <= KL; ++i)
                        if (jp == i)
#pragma unroll
                            for (int c = 0; c <= KV; ++c) {
                                const double t = w[0][c];
                                w[0][c] = w[i][c];
                                w[i][c] = t;
                            }
                }
                const double rp = 1.0 / pv;
#pragma unroll
                for (int i = 1; i <= KL; ++i)
                    w[i][0] *= rp;  // rows and columns beyond the last hold zeros
#pragma unroll
                for (int c = 1; c <= KV; ++c) {
                    const double y = -w[0][c];
#pragma unroll
                    for (int i = 1; i <= KL; ++i)
                        w[i][c] = fma(w[i][0], y, w[i][c]);
                }
            } else {
                flags |= jp != 0;
                atomicCAS(&job.st->info[blockIdx.y], 0, j + 1);
            }
        }
#pragma unroll
        for (int c = 0; c <= KV; ++c)
            if (j + c < N) put(KV - c, j + c, w[0][c]);
#pragma unroll
        for (int i = 1; i <= KL; ++i)
            put(KV + i, j, j + i < N ? w[i][0] : __dmul_rn(c2, dm.radLap[(KL + i) * N + j]));
#pragma unroll
        for (int i = 0; i < KL; ++i)
#pragma unroll
            for (int c = 0; c <= KV; ++c) w[i][c] = c < KV ? w[i + 1][c + 1] : 0.0;
#pragma unroll
        for (int c = 0; c <= KV; ++c) w[KL][c] = nx[c];
    }
    if (flags) atomicOr(&job.st->piv[blockIdx.y], flags);
}

// One banded solve (dgbtrs 'N' with one right-hand side): forward sweep with
// the row interchanges and unit-lower multipliers, then the upper-triangular
// band back substitution (dtbsv).  b(n) is at b[n*stride] and is zero before
// row j0 (there it is only written); the active part of the vector is held in
// registers, and the factors of the next PRE columns are read while these are
// worked on.
__device__ __forceinline__ void lu_solve_one(const double *__restrict__ lu, const unsigned char *__restrict__ piv,
                                             int N, int Hp, int nh, double *b, size_t stride, int j0) {
    constexpr int PRE = 4;
    {
        double w[KL + 1];
#pragma unroll
        for (int i = 0; i <= KL; ++i) w[i] = j0 + i < N ? b[(size_t)(j0 + i) * stride] : 0.0;
        double l[PRE][KL], bn[PRE], ln[PRE][KL], bnn[PRE];
        int p[PRE], pn[PRE];
        auto get = [&](int jb, double (&lo)[PRE][KL], int (&po)[PRE], double (&bo)[PRE]) {
#pragma unroll
            for (int s = 0; s < PRE; ++s) {
                const int j = jb + s;
                po[s] = j < N - 1 ? piv[(size_t)j * Hp + nh] : 0;
#pragma unroll
                for (int i = 1; i <= KL; ++i) lo[s][i - 1] = j + i < N ? LU(KV + i, j) : 0.0;
                bo[s] = j + KL + 1 < N ? b[(size_t)(j + KL + 1) * stride] : 0.0;
            }
        };
        get(j0, l, p, bn);
        for (int jb = j0; jb < N; jb += PRE) {
            get(jb + PRE, ln, pn, bnn);
#pragma unroll
            for (int s = 0; s < PRE; ++s) {
                const int j = jb + s;
                if (j < N) {
#pragma unroll
                    for (int i = 1; i <= KL; ++i)
                        if (p[s] == i) {
                            const double t = w[0];
                            w[0] = w[i];
                            w[i] = t;
                        }
                    const double bj = w[0];
#pragma unroll
                    for (int i = 1; i <= KL; ++i)
                        if (j + i < N) w[i] = fma(-l[s][i - 1], bj, w[i]);
                    b[(size_t)j * stride] = bj;
#pragma unroll
                    for (int i = 0; i < KL; ++i) w[i] = w[i + 1];
                    w[KL] = bn[s];
                }
            }
#pragma unroll
            for (int s = 0; s < PRE; ++s) {
#pragma unroll
                for (int i = 0; i < KL; ++i) l[s][i] = ln[s][i];
                p[s] = pn[s];
                bn[s] = bnn[s];
            }
        }
    }
    double v[KV + 1];
#pragma unroll
    for (int i = 0; i <= KV; ++i) v[i] = N - 1 - i >= j0 ? b[(size_t)(N - 1 - i) * stride] : 0.0;
    double u[PRE][KV + 1], bn[PRE], un[PRE][KV + 1], bnn[PRE];
    auto get = [&](int jb, double (&uo)[PRE][KV + 1], double (&bo)[PRE]) {
#pragma unroll
        for (int s = 0; s < PRE; ++s) {
            const int j = jb - s;
#pragma unroll
            for (int i = 0; i <= KV; ++i) uo[s][i] = j - i >= 0 ? LU(KV - i, j) : 0.0;
            bo[s] = j - KV - 1 >= j0 ? b[(size_t)(j - KV - 1) * stride] : 0.0;
        }
    };
    get(N - 1, u, bn);
    for (int jb = N - 1; jb >= 0; jb -= PRE) {
        get(jb - PRE, un, bnn);
#pragma unroll
        for (int s = 0; s < PRE; ++s) {
            const int j = jb - s;
            if (j >= 0) {
                double x = v[0];
                if (x != 0.0) {
                    x = x / u[s][0];
#pragma unroll
                    for (int i = 1; i <= KV; ++i) v[i] = fma(-x, u[s][i], v[i]);
                }
                b[(size_t)j * stride] = x;
#pragma unroll
                for (int i = 0; i < KV; ++i) v[i] = v[i + 1];
                v[KV] = bn[s];
            }
        }
#pragma unroll
        for (int s = 0; s < PRE; ++s) {
#pragma unroll
            for (int i = 0; i <= KV; ++i) u[s][i] = un[s][i];
            bn[s] = bnn[s];
        }
    }
}

// thread = (mode, re/im); timestep.f90:109-121
__global__ void k_lu_solve(const double *__restrict__ lu, const unsigned char *__restrict__ piv,
                           double2 *b, int N, int H, int Hp, int BC) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int nh = t >> 1, part = t & 1;
    if (nh >= H) return;
    double *bp = reinterpret_cast<double *>(b) + 2 * (size_t)nh + part;
    const size_t stride = 2 * (size_t)Hp;
    if (BC == 1 && nh == 0) {
        for (int n = 0; n < N; ++n) bp[n * stride] = 0.0;
        return;
    }
    lu_solve_one(lu, piv, N, Hp, nh, bp, stride, 0);
}

int pf_launch_lu_solve(pf_ctx *ctx, int BC, const pf_lumesh *A, double2 *b) {
    const Geo &g = ctx->g;
    {
        ProfScope ps_(ctx, PF_K_LUSOLVE);
        k_lu_solve<<<grid1(2LL * g.H, 128), 128, 0, ctx->stream>>>(A->lu, A->piv, b, g.N, g.H, g.Hp, BC);
    }
    PF_LAUNCHED(ctx);
    return PF_OK;
}

// ------------------------------------------------- influence matrices
// Boundary residuals of (u+, u-, uz) at r=1 (velocity.f90:262-298).
__device__ __forceinline__ void eval_bc(const double2 *__restrict__ up, const double2 *__restrict__ um,
                                        const double2 *__restrict__ uz, const DevMesh &dm, const Geo &g,
                                        int nh, int k, int m, double BRe[4], double BIm[4]) {
    const int N = g.N;
    const size_t at = (size_t)(N - 1) * g.Hp + nh;
    const double2 p = up[at], q = um[at], z = uz[at];
    const double urRe = 0.5 * (p.x + q.x), urIm = 0.5 * (p.y + q.y);
    const double utRe = 0.5 * (p.y - q.y), utIm = -0.5 * (p.x - q.x);
    double drRe = 0.0, drIm = 0.0;
    for (int j = 0; j <= KL; ++j) {
        const size_t a = (size_t)(N - 1 - KL + j) * g.Hp + nh;
        const double w = dm.dr1[1 * (KL + 1) + j];
        drRe += w * (up[a].x + um[a].x);
        drIm += w * (up[a].y + um[a].y);
    }
    drRe = 0.5 * drRe;
    drIm = 0.5 * drIm;
    const double d = dm.rp[2 * N + (N - 1)];
    const double m_ = (double)(m * g.Mp), a_ = g.alpha * k;
    BRe[0] = p.x; BIm[0] = p.y;
    BRe[1] = q.x; BIm[1] = q.y;
    BRe[2] = -z.y; BIm[2] = z.x;
    BRe[3] = urRe * d + drRe - d * m_ * utIm - a_ * z.y;
    BIm[3] = urIm * d + drIm + d * m_ * utRe + a_ * z.x;
}

// Unit wall-value solutions and the mean-flux response (velocity.f90:160-168,
// 194-221), one thread per solve:
//   blockIdx.y 0..2  U1..U3: LD(p, m, z) x = e_{N-1} for the mode of the thread
//   blockIdx.y 3     Ui = LDz(0)^-1 [0,1,..,1,0] and d1 = 2 int Ui r dr
//   blockIdx.y 4     c4 = -LNp^-1 e_{N-1}, the pressure of a unit wall value
// Bound by the chain of a column (a division and an update): N = 40 in 24 us
// for all, where each of four solves in turn read its factors inside the chain
// (65 us each).
__global__ void __launch_bounds__(32) k_unit_solves(const LUJob job, double *__restrict__ U, double *__restrict__ Ui,
                                                    double2 *__restrict__ c4, DevMesh dm, Geo g, DevScalars *sc) {
    const int nh = blockIdx.x * blockDim.x + threadIdx.x;
    const int N = g.N, Hp = g.Hp;
    if (blockIdx.y == 3) {
        if (nh != 0 || !Ui) return;
        const LUJob::Set &A = job.s[2];
        for (int n = 0; n < N; ++n) Ui[n] = (n == 0 || n == N - 1) ? 0.0 : 1.0;
        lu_solve_one(A.lu, A.piv, N, Hp, 0, Ui, 1, 0);
        double d1 = 0.0;
        for (int n = 0; n < N; ++n) d1 += Ui[n] * dm.intrdr[n];
        sc->flux_d1 = 2.0 * d1;
        return;
    }
    if (nh >= g.H) return;
    const bool p = blockIdx.y == 4;
    const LUJob::Set &A = job.s[p ? 3 : blockIdx.y];
    double *b = p ? reinterpret_cast<double *>(c4 + nh) : U + (size_t)blockIdx.y * N * Hp + nh;
    const size_t stride = p ? 2 * (size_t)Hp : Hp;
    if (p && nh == 0) return;  // k = m = 0 has no pressure: c4 is zeros
    for (int n = N - 1 - KL; n < N; ++n) b[(size_t)n * stride] = n < N - 1 ? 0.0 : p ? -1.0 : 1.0;
    lu_solve_one(A.lu, A.piv, N, Hp, nh, b, stride, N - 1 - KL);
}

// U4..U6: the velocity of the unit pressure, grad c4 in the u+-, u- variables
__global__ void k_unit_pressure(const double2 *__restrict__ ur, const double2 *__restrict__ ut,
                                const double2 *__restrict__ uz, double *__restrict__ U, int N, Geo g) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long NH = (long long)N * g.Hp;
    if (t >= NH || t % g.Hp >= g.H) return;
    const double2 r = ur[t], v = ut[t];
    U[3 * NH + t] = r.x - v.y;
    U[4 * NH + t] = r.x + v.y;
    U[5 * NH + t] = uz[t].y;
}

// Each mode's 4x4 influence matrix, its columns the boundary residuals (up, um,
// i uz, div u at r = 1; velocity.f90:262-298) of U1, U2, U3 and U4..6, replaced
// by its inverse (mes_mat_invert, meshs.f90:231-243): Gauss-Jordan with partial
// pivoting; k=m=0 skipped (velocity.f90:222-225).
__global__ void __launch_bounds__(64) k_influence(const double *__restrict__ U, double *__restrict__ Ainv, DevMesh dm,
                                                  Geo g, LUStat *st) {
    const int nh = blockIdx.x * blockDim.x + threadIdx.x;
    if (nh >= g.H || nh == 0) return;
    const int N = g.N, Hp = g.Hp;
    int k, m;
    mode_km(nh, g.K, k, m);
    const double d = dm.rp[2 * N + (N - 1)], m_ = (double)(m * g.Mp), a_ = g.alpha * k;
    double a[4][4], b[4][4];
    auto column = [&](int j, const double *up, const double *um, const double *uz) {
        double dr = 0.0;
#pragma unroll
        for (int i = 0; i <= KL; ++i) {
            const size_t at = (size_t)(N - 1 - KL + i) * Hp + nh;
            dr += dm.dr1[1 * (KL + 1) + i] * ((up ? up[at] : 0.0) + (um ? um[at] : 0.0));
        }
        const size_t wall = (size_t)(N - 1) * Hp + nh;
        const double p = up ? up[wall] : 0.0, q = um ? um[wall] : 0.0, z = uz ? uz[wall] : 0.0;
        a[0][j] = p;
        a[1][j] = q;
        a[2][j] = -z;
        a[3][j] = 0.5 * (p + q) * d + 0.5 * dr - d * m_ * (-0.5 * (p - q)) - a_ * z;
    };
    const size_t NH = (size_t)N * Hp;
    column(0, U, nullptr, nullptr);
    column(1, nullptr, U + NH, nullptr);
    column(2, nullptr, nullptr, U + 2 * NH);
    column(3, U + 3 * NH, U + 4 * NH, U + 5 * NH);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) b[i][j] = (i == j) ? 1.0 : 0.0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        int p = c;
        double x = a[c][c];
#pragma unroll
        for (int r = c + 1; r < 4; ++r)
            if (fabs(a[r][c]) > fabs(x)) {
                p = r;
                x = a[r][c];
            }
        if (x == 0.0) {
            atomicCAS(&st->inv, 0, -(nh + 1));
            return;
        }
#pragma unroll
        for (int r = c + 1; r < 4; ++r)
            if (p == r)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    double t = a[r][q]; a[r][q] = a[c][q]; a[c][q] = t;
                    t = b[r][q]; b[r][q] = b[c][q]; b[c][q] = t;
                }
        const double inv = 1.0 / x;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            a[c][q] *= inv;
            b[c][q] *= inv;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            if (r == c) continue;
            const double f = a[r][c];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                a[r][q] -= f * a[c][q];
                b[r][q] -= f * b[c][q];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) Ainv[(size_t)(i * 4 + j) * Hp + nh] = b[i][j];
}

// vel_adjPPE(2): u += sum_j a_j U_j with a = -A^-1 B (velocity.f90:238-256).
__global__ void k_adjppe2(double2 *ur, double2 *ut, double2 *uz, const double *__restrict__ Ainv,
                          const double *__restrict__ U, DevMesh dm, Geo g) {
    const int nh = blockIdx.x * blockDim.x + threadIdx.x;
    if (nh >= g.H || nh == 0) return;
    int k, m;
    mode_km(nh, g.K, k, m);
    double BRe[4], BIm[4], aR[4], aI[4];
    eval_bc(ur, ut, uz, dm, g, nh, k, m, BRe, BIm);
    for (int i = 0; i < 4; ++i) {
        double sr = 0.0, si = 0.0;
        for (int j = 0; j < 4; ++j) {
            const double a = Ainv[(size_t)(i * 4 + j) * g.Hp + nh];
            sr += a * BRe[j];
            si += a * BIm[j];
        }
        aR[i] = -sr;
        aI[i] = -si;
    }
    const int N = g.N;
    for (int n = 0; n < N; ++n) {
        const size_t at = (size_t)n * g.Hp + nh;
        const double U1 = U[(size_t)(0 * N + n) * g.Hp + nh], U2 = U[(size_t)(1 * N + n) * g.Hp + nh];
        const double U3 = U[(size_t)(2 * N + n) * g.Hp + nh], U4 = U[(size_t)(3 * N + n) * g.Hp + nh];
        const double U5 = U[(size_t)(4 * N + n) * g.Hp + nh], U6 = U[(size_t)(5 * N + n) * g.Hp + nh];
        double2 r = ur[at], t = ut[at], z = uz[at];
        r.x = r.x + aR[0] * U1; r.y = r.y + aI[0] * U1;
        t.x = t.x + aR[1] * U2; t.y = t.y + aI[1] * U2;
        z.x = z.x - aI[2] * U3; z.y = z.y + aR[2] * U3;
        r.x = r.x + aR[3] * U4; r.y = r.y + aI[3] * U4;
        t.x = t.x + aR[3] * U5; t.y = t.y + aI[3] * U5;
        z.x = z.x - aI[3] * U6; z.y = z.y + aR[3] * U6;
        ur[at] = r; ut[at] = t; uz[at] = z;
    }
}

int pf_launch_adjppe2(pf_ctx *ctx) {
    const Geo &g = ctx->g;
    {
        ProfScope ps_(ctx, PF_K_INFL);
        k_adjppe2<<<grid1(g.H, 64), 64, 0, ctx->stream>>>(ctx->vel[0].d, ctx->vel[1].d, ctx->vel[2].d, ctx->Ainv,
                                                           ctx->U, ctx->dm, g);
    }
    PF_LAUNCHED(ctx);
    return PF_OK;
}

// ------------------------------------------------------- constant flux
// F=1: remove the mean-flux excess and update Pr0 (velocity.f90:170-175)
__global__ void k_flux1(double2 *uz, const double *__restrict__ Ui, DevMesh dm, Geo g, DevScalars *sc) {
    __shared__ double part[32];
    const int N = g.N;
    double s = 0.0;
    for (int n = threadIdx.x; n < N; n += blockDim.x) s += uz[(size_t)n * g.Hp].x * dm.intrdr[n];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x + 31) / 32; ++w) t += part[w];
        part[0] = t;
    }
    __syncthreads();
    const double d2 = 2.0 * part[0];
    const double d3 = -d2 / sc->flux_d1;
    for (int n = threadIdx.x; n < N; n += blockDim.x) {
        double2 v = uz[(size_t)n * g.Hp];
        v.x = v.x + d3 * Ui[n];
        uz[(size_t)n * g.Hp] = v;
    }
    if (threadIdx.x == 0) sc->Pr0 = sc->Pr0 + d3 * g.Re / 4.0;
}

int pf_launch_flux1(pf_ctx *ctx) {
    if (!ctx->cfg.const_flux) return PF_OK;
    {
        ProfScope ps_(ctx, PF_K_INFL);
        k_flux1<<<1, 256, 0, ctx->stream>>>(ctx->vel[2].d, ctx->Ui, ctx->dm, ctx->g, ctx->dsc);
    }
    PF_LAUNCHED(ctx);
    return PF_OK;
}

// ---------------------------------------------------------- vel_matrices
// The factor tiles of a set (pf_internal.cuh): thread per (tile matrix,
// column), 8 consecutive matrices of a tile on consecutive threads.  A matrix
// that is not factored (BC=1 at k=m=0) and padding are zeros, which solve to 0.
template <bool PIV, bool WIDE>
__device__ __forceinline__ void lu_tiles_body(const double *__restrict__ lu, const unsigned char *__restrict__ piv,
                                              double *__restrict__ tiles, const Geo &g, int BC) {
    constexpr int FR = ft_fwd_rows(PIV), BR = ft_back_rows(WIDE);
    const int N = g.N, Hp = g.Hp, nz = 16 * pf_mean_tiles(g), nt = nz + 8 * pf_paired_tiles(g);
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)nt * N) return;
    const int e = (int)(t % 8), j = (int)(t / 8 % N), c = (int)(t / 8 / N) * 8 + e;
    const int W = c < nz ? 16 : 8;
    const int m = c < nz ? 0 : 1 + (c - nz) / g.K, k = c < nz ? c : (c - nz) % g.K;
    const bool live = (c < nz ? k < g.K : m < g.M) && !(BC == 1 && c == 0);
    const int nh = m * (2 * g.K - 1) + k;
    double *o = tiles + (size_t)(c / W * W) * N * FT_ROWS + c % W;
    double *f = o + (size_t)j * FR * W, *b = o + ((size_t)N * FR + (size_t)(N - 1 - j) * BR) * W;
#pragma unroll
    for (int r = 1; r <= KL; ++r) f[(r - 1) * W] = live && j + r < N ? LU(KV + r, j) : 0.0;
    if (PIV) f[KL * W] = __hiloint2double(0, live && j < N - 1 ? piv[(size_t)j * Hp + nh] : 0);
    const double u = live ? LU(KV, j) : 0.0, hi = live ? 1.0 / u : 0.0;
    b[0] = hi;
    b[W] = fma(-u, hi, 1.0) * hi;
#pragma unroll
    for (int r = 1; r <= BR - 2; ++r) b[(r + 1) * W] = live && j - r >= 0 ? LU(KV - r, j) : 0.0;
}

// Set blockIdx.y in the form its factors need; the pressure set always in the
// full form.
__global__ void k_lu_tiles(const LUJob job, const Geo g) {
    const LUJob::Set &A = job.s[blockIdx.y];
    const int f = job.st->piv[blockIdx.y];
    if (!A.tiles) return;
    if (A.BC == 1 || f > 1) lu_tiles_body<true, true>(A.lu, A.piv, A.tiles, g, A.BC);
    else if (f) lu_tiles_body<true, false>(A.lu, A.piv, A.tiles, g, A.BC);
    else lu_tiles_body<false, false>(A.lu, A.piv, A.tiles, g, A.BC);
}

static void lu_job_add(LUJob &job, pf_lumesh *A, int PM, int BC, double c1, double c2) {
    A->PM = PM;
    A->BC = BC;
    A->c1 = c1;
    A->c2 = c2;
    job.s[job.n++] = {A->lu, A->piv, A->tiles, PM, BC, c1, c2};
}

// Factor the sets of a job: one launch for all, one for their tiles.
static int lu_job_launch(pf_ctx *ctx, const LUJob &job) {
    const Geo &g = ctx->g;
    PF_CUDA(cudaMemsetAsync(job.st, 0, sizeof(LUStat), ctx->stream));
    {
        ProfScope ps_(ctx, PF_K_FACTOR);
        k_lu_factor<<<dim3(grid1((long long)g.M * g.K, 32), job.n), 32, 0, ctx->stream>>>(job, ctx->dm, g);
    }
    PF_LAUNCHED(ctx);
    if (!job.s[0].tiles) return PF_OK;
    {
        ProfScope ps_(ctx, PF_K_FACTOR);
        const unsigned grid = grid1((long long)pf_tile_modes(g) * g.N, 128);
        k_lu_tiles<<<dim3(grid, job.n), 128, 0, ctx->stream>>>(job, g);
    }
    PF_LAUNCHED(ctx);
    return PF_OK;
}

static int lu_status(int info) {
    if (info == 0) return PF_OK;
    pf_set_error("tim_lumesh_init: zero pivot in column %d", info);
    return PF_ERR_SINGULAR;
}

// velocity.f90:120-146 including vel_adjustFlux(0) and vel_adjPPE(0): every
// set in one factorisation, every solve in one launch, one wait at the end
// (N = 48, 1481 modes: 1295 -> 125 us).  The pressure set and its solution
// depend on the mesh and alpha only and are kept over changes of dt.
int pf_vel_matrices_impl(pf_ctx *ctx) {
    const Geo &g = ctx->g;
    pf_graphs_reset(ctx);  // the graphs bake in 1/dt and the factor sets
    const pf_config &cfg = ctx->cfg;
    const int N = g.N, Hp = g.Hp;
    LUJob job = {};
    job.st = (LUStat *)ctx->lustat;
    const bool fresh = !ctx->LNp_set;
    double d1 = 1.0 / ctx->tim.dt;
    double d2 = -cfg.implicit * ctx->vel_nu / cfg.Re;
    lu_job_add(job, &ctx->LDp, 1, 0, d1, d2);
    lu_job_add(job, &ctx->LDm, -1, 0, d1, d2);
    lu_job_add(job, &ctx->LDz, 0, 0, d1, d2);
    if (fresh) lu_job_add(job, &ctx->LNp, 0, 1, 0.0, 1.0);
    PF_TRY(lu_job_launch(ctx, job));
    d2 = (1.0 - cfg.implicit) * ctx->vel_nu / cfg.Re;
    ctx->Ltp = {ctx, 1, d1, d2};
    ctx->Ltm = {ctx, -1, d1, d2};
    ctx->Ltz = {ctx, 0, d1, d2};
    double2 *c1 = ctx->s[0].d, *c2 = ctx->s[1].d, *c3 = ctx->s[2].d, *c4 = ctx->s[3].d;
    if (fresh) PF_CUDA(cudaMemsetAsync(c4, 0, (size_t)N * Hp * sizeof(double2), ctx->stream));
    {
        ProfScope ps_(ctx, PF_K_FACTOR);
        k_unit_solves<<<dim3(grid1(g.H, 32), fresh ? 5 : cfg.const_flux ? 4 : 3), 32, 0, ctx->stream>>>(
            job, ctx->U, cfg.const_flux ? ctx->Ui : nullptr, c4, ctx->dm, g, ctx->dsc);
    }
    PF_LAUNCHED(ctx);
    if (fresh) {
        PF_TRY(pf_launch_grad(ctx, c4, c1, c2, c3));
        {
            ProfScope ps_(ctx, PF_K_FACTOR);
            k_unit_pressure<<<grid1((long long)N * Hp, 128), 128, 0, ctx->stream>>>(c1, c2, c3, ctx->U, N, g);
        }
        PF_LAUNCHED(ctx);
    }
    {
        ProfScope ps_(ctx, PF_K_FACTOR);
        k_influence<<<grid1(g.H, 64), 64, 0, ctx->stream>>>(ctx->U, ctx->Ainv, ctx->dm, g, job.st);
    }
    PF_LAUNCHED(ctx);
    LUStat st;
    PF_CUDA(cudaMemcpyAsync(ctx->hsc, ctx->dsc, sizeof(DevScalars), cudaMemcpyDeviceToHost, ctx->stream));
    PF_CUDA(cudaMemcpyAsync(&st, job.st, sizeof(st), cudaMemcpyDeviceToHost, ctx->stream));
    PF_CUDA(cudaStreamSynchronize(ctx->stream));
    if (fresh) {
        PF_TRY(lu_status(st.info[3]));
        ctx->LNp.pivoted = st.piv[3];
        ctx->LNp_set = true;
    }
    pf_lumesh *LD[3] = {&ctx->LDp, &ctx->LDm, &ctx->LDz};
    for (int i = 0; i < 3; ++i) {
        PF_TRY(lu_status(st.info[i]));
        LD[i]->pivoted = st.piv[i];
    }
    if (cfg.const_flux && ctx->hsc->flux_d1 == 0.0) {
        pf_set_error("vel_adjustFlux: err 2");
        return PF_ERR_SINGULAR;
    }
    if (st.inv != 0) {
        pf_set_error("matrix inversion error 1 (influence matrix of mode %d)", -st.inv - 1);
        return PF_ERR_SINGULAR;
    }
    ctx->matrices_ready = true;
    ctx->matrices_gen++;
    return PF_OK;
}

// ------------------------------------------------------------------ C ABI
extern "C" int pf_tim_mesh_init(pf_ctx *ctx, int PM, double c1, double c2, pf_mesh **out) {
    PF_ARG(ctx && out && PM >= -1 && PM <= 1, "pf_tim_mesh_init: bad argument");
    *out = new pf_mesh{ctx, PM, c1, c2};
    return PF_OK;
}

extern "C" int pf_mesh_destroy(pf_mesh *A) {
    delete A;
    return PF_OK;
}

// host layout M[(nh*N + j)*(2KL+1) + row] == A(nh)%M(row+1, j+1)
extern "C" int pf_mesh_download(const pf_mesh *A, double *M) {
    PF_ARG(A && M, "null argument");
    const pf_ctx *ctx = A->ctx;
    const Geo &g = ctx->g;
    const int N = g.N;
    const HostMesh &hm = ctx->hm;
    for (int nh = 0; nh < g.H; ++nh) {
        int k, m;
        mode_km(nh, g.K, k, m);
        for (int j = 0; j < N; ++j)
            for (int row = 0; row < NBAND; ++row) {
                double v = A->c2 * hm.radLap[row * N + j];
                if (row == KL) {
                    const double r2 = hm.rp[1 * N + j];
                    double d = -(r2 * g.Mp * m * g.Mp * m) - g.alpha * k * g.alpha * k;
                    if (A->PM != 0) d = d - r2 - 2.0 * A->PM * g.Mp * m * r2;
                    v = v + A->c2 * d + A->c1;
                }
                M[((size_t)nh * N + j) * NBAND + row] = v;
            }
    }
    return PF_OK;
}

extern "C" int pf_tim_lumesh_init(pf_ctx *ctx, int PM, int BC, double c1, double c2, pf_lumesh **out) {
    PF_ARG(ctx && out && PM >= -1 && PM <= 1 && (BC == 0 || BC == 1), "pf_tim_lumesh_init: bad argument");
    *out = nullptr;
    pf_lumesh *A = new pf_lumesh();
    A->ctx = ctx;
    const Geo &g = ctx->g;
    int s = pf_alloc(ctx, (void **)&A->lu, (size_t)NLU * g.N * g.Hp * sizeof(double));
    if (s == PF_OK) s = pf_alloc(ctx, (void **)&A->piv, (size_t)g.N * g.Hp);
    if (s == PF_OK) {
        LUJob job = {};
        job.st = (LUStat *)ctx->lustat;
        lu_job_add(job, A, PM, BC, c1, c2);
        s = lu_job_launch(ctx, job);
    }
    if (s == PF_OK) {
        LUStat st;
        PF_CUDA(cudaMemcpyAsync(&st, ctx->lustat, sizeof(st), cudaMemcpyDeviceToHost, ctx->stream));
        PF_CUDA(cudaStreamSynchronize(ctx->stream));
        A->pivoted = st.piv[0];
        s = lu_status(st.info[0]);
    }
    if (s != PF_OK) {
        pf_lumesh_destroy(A);
        return s;
    }
    *out = A;
    return PF_OK;
}

extern "C" int pf_lumesh_destroy(pf_lumesh *A) {
    if (!A) return PF_OK;
    pf_ctx *ctx = A->ctx;
    cudaStreamSynchronize(ctx->stream);
    for (void *p : {(void *)A->lu, (void *)A->piv}) {
        for (size_t i = 0; i < ctx->allocs.size(); ++i)
            if (ctx->allocs[i] == p) {
                cudaFree(p);
                ctx->allocs.erase(ctx->allocs.begin() + i);
                break;
            }
    }
    ctx->bytes -= (size_t)NLU * ctx->g.N * ctx->g.Hp * sizeof(double) + (size_t)ctx->g.N * ctx->g.Hp;
    delete A;
    return PF_OK;
}

// host layout M[(nh*N + j)*(3KL+1) + row] == A(nh)%M(row+1, j+1), ipiv 1-based
extern "C" int pf_lumesh_download(const pf_lumesh *A, double *M, int *ipiv) {
    PF_ARG(A && M && ipiv, "null argument");
    pf_ctx *ctx = A->ctx;
    const Geo &g = ctx->g;
    std::vector<double> lu((size_t)NLU * g.N * g.Hp);
    std::vector<unsigned char> pv((size_t)g.N * g.Hp);
    PF_CUDA(cudaMemcpyAsync(lu.data(), A->lu, lu.size() * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    PF_CUDA(cudaMemcpyAsync(pv.data(), A->piv, pv.size(), cudaMemcpyDeviceToHost, ctx->stream));
    PF_CUDA(cudaStreamSynchronize(ctx->stream));
    for (int nh = 0; nh < g.H; ++nh)
        for (int j = 0; j < g.N; ++j) {
            for (int row = 0; row < NLU; ++row)
                M[((size_t)nh * g.N + j) * NLU + row] = lu[((size_t)row * g.N + j) * g.Hp + nh];
            ipiv[(size_t)nh * g.N + j] = j + 1 + pv[(size_t)j * g.Hp + nh];
        }
    return PF_OK;
}

extern "C" int pf_tim_lumesh_invert(int BC, const pf_lumesh *A, pf_coll *b) {
    PF_ARG(A && b && A->ctx == b->ctx && (BC == 0 || BC == 1), "pf_tim_lumesh_invert: bad argument");
    return pf_launch_lu_solve(b->ctx, BC, A, b->d);
}

extern "C" int pf_vel_influence_download(const pf_ctx *ctx, double *U, double *A) {
    PF_ARG(ctx, "null ctx");
    PF_ARG(ctx->matrices_ready, "pf_vel_influence_download: call pf_vel_matrices first");
    const Geo &g = ctx->g;
    const int N = g.N;
    std::vector<double> u((size_t)6 * N * g.Hp), a((size_t)16 * g.Hp);
    PF_CUDA(cudaMemcpyAsync(u.data(), ctx->U, u.size() * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    PF_CUDA(cudaMemcpyAsync(a.data(), ctx->Ainv, a.size() * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    PF_CUDA(cudaStreamSynchronize(ctx->stream));
    if (U)
        for (int c = 0; c < 6; ++c)
            for (int nh = 0; nh < g.H; ++nh)
                for (int n = 0; n < N; ++n)
                    U[((size_t)c * g.H + nh) * N + n] = u[((size_t)c * N + n) * g.Hp + nh];
    if (A)
        for (int nh = 0; nh < g.H; ++nh)
            for (int i = 0; i < 4; ++i)
                for (int j = 0; j < 4; ++j) A[(size_t)nh * 16 + j * 4 + i] = a[(size_t)(i * 4 + j) * g.Hp + nh];
    return PF_OK;
}
