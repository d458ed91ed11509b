// Particle-physics precompute on the device (FP64).
//
// Replaces the precompute launched by ClaritasForwardModel._prepare_gpu_particle_physics
// (CLARITAS/CLARITAS.py:6036-6965). The per-bin and per-angle arithmetic is the
// reference's (kernels :3488-3592, :3845-3921, :3925-4038), so the tables the
// photon kernel reads are identical to the reference's on the same GPU; only
// the parallel decomposition changes:
//  * Mie coefficients: one block per size bin, the three recurrences in a warp each
//    in shared memory instead of a global scratch array;
//  * phase pdf: the angular functions pi_n/tau_n, which depend only on the angle and
//    the order, come from a table made once, instead of a recurrence in every
//    (bin, angle) thread; where that table would be too large, threads run it, for
//    four bins at a time where there are many;
//  * Schiller-Naumann radial slip: one thread per (bin, radius) instead of one
//    thread for everything; the serial prefix sums and quadrature stay serial
//    per bin so their rounding is unchanged.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>
#include <cooperative_groups.h>
#include "kernels.h"

namespace clr {

#define PD_PI 3.141592653589793238462643383279502884

struct cdx { double re, im; };
__device__ __forceinline__ cdx CD(double re, double im) { cdx z; z.re = re; z.im = im; return z; }
__device__ __forceinline__ cdx cd_add(cdx a, cdx b) { return CD(a.re + b.re, a.im + b.im); }
__device__ __forceinline__ cdx cd_sub(cdx a, cdx b) { return CD(a.re - b.re, a.im - b.im); }
__device__ __forceinline__ cdx cd_mul(cdx a, cdx b) { return CD(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re); }
__device__ __forceinline__ cdx cd_scale(cdx a, double s) { return CD(a.re * s, a.im * s); }
// q / d for d > 0. A zero numerator (every imaginary part when the particles do not absorb) is its own quotient,
// sign included; the division would take its slow path for it.
// (Both tests on the bits: an FP64 comparison costs what an FP64 addition does.)
__device__ __forceinline__ double pos_div(double q, double d) {
    return (__double_as_longlong(q) << 1) == 0 ? q : q / d;
}
__device__ __forceinline__ double not_tiny(double d) {
    return __double_as_longlong(d) < __double_as_longlong(1e-300) ? 1e-300 : d;
}
__device__ __forceinline__ cdx cd_div(cdx a, cdx b) {
    const double d = not_tiny(b.re * b.re + b.im * b.im);
    return CD(pos_div(a.re * b.re + a.im * b.im, d), pos_div(a.im * b.re - a.re * b.im, d));
}
__device__ __forceinline__ double cd_abs2(cdx a) { return a.re * a.re + a.im * a.im; }
__device__ __forceinline__ double cd_rmc(cdx a, cdx b) { return a.re * b.re + a.im * b.im; }

// The serial FP64 sum 0 + v[0] + v[1] + ... (each addition rounded, in that order) by one warp; all lanes call and
// all get it. With `prefix` (which may be v itself) the partial sum after each value is stored there.
// One FP64 addition occupies its warp for 64 cycles whatever the lanes do, so a serial sum of non-negative terms
// runs in integers instead: while the sum s stays in one binade it is a multiple S of its ulp u, and s + x rounds to
// (S + x/u rounded to nearest) u. The lanes round 32 terms at once and add them by a scan. A term exactly half way
// between two multiples goes to the even sum, whose parity the lanes below it give; the term at which the sum leaves
// its binade (and one larger than the sum) is added in FP64. About 350 cycles per 32 terms against 2048.
// Terms that are negative, infinite or NaN are added one by one.
__device__ __forceinline__ double warp_serial_sum(const double* v, int n, double* prefix) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    constexpr long long kHidden = 1ll << 52, kMant = kHidden - 1;
    double s = 0.0, next = lane < n ? v[lane] : 0.0;
    for (int j = 0; j < n; j += 32) {
        const double x = next;
        next = j + 32 + lane < n ? v[j + 32 + lane] : 0.0;
        const long long xb = __double_as_longlong(x);
        double mine = 0.0;
        if (__all_sync(FULL, (unsigned long long)xb < 0x7ff0000000000000ull)) {
            const int xe = max((int)(xb >> 52), 1);
            const long long xm = (xb & kMant) | (xb >= kHidden ? kHidden : 0);
            for (int start = 0; start < 32;) {
                const long long sb = __double_as_longlong(s);
                const int se = (int)(sb >> 52), shift = se - xe;  // se 0: the sum is still 0 (or subnormal)
                const long long S = (sb & kMant) | kHidden;
                const bool in = lane >= start && xb != 0;
                const unsigned larger = __ballot_sync(FULL, in && (se == 0 || shift < 0));
                const int limit = larger ? __ffs(larger) - 1 : 32;
                long long xi = 0;
                bool tie = false;
                if (in && lane < limit && shift <= 53) {
                    xi = xm >> shift;
                    const long long rest = xm & ((1ll << shift) - 1), half = shift ? 1ll << (shift - 1) : 1;
                    if (rest > half) ++xi;
                    tie = rest == half;
                }
                unsigned odd = __ballot_sync(FULL, (xi & 1) != 0);
                for (unsigned t = __ballot_sync(FULL, tie); t; t &= t - 1u) {
                    const int l = __ffs(t) - 1;
                    const unsigned upto = 0xffffffffu >> (31 - l);  // lanes 0..l
                    if (((unsigned)S + __popc(odd & upto)) & 1u) {
                        if (lane == l) ++xi;
                        odd ^= 1u << l;
                    }
                }
                long long inc = xi;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const long long up = __shfl_up_sync(FULL, inc, o);
                    if (lane >= o) inc += up;
                }
                const unsigned leaves = __ballot_sync(FULL, S + inc >= 2 * kHidden && lane < limit);
                const int c = leaves ? __ffs(leaves) - 1 : limit;  // lanes start..c-1 are summed
                const double here = se == 0 ? s : __longlong_as_double(((long long)se << 52) | ((S + inc) & kMant));
                if (lane >= start && lane < c) mine = here;
                if (c > start) s = __shfl_sync(FULL, here, c - 1);
                start = c + 1;
                if (c < 32) {
                    s += __shfl_sync(FULL, x, c);
                    if (lane == c) mine = s;
                }
            }
        } else {
            for (int l = 0; l < 32; ++l) {
                s += __shfl_sync(FULL, x, l);
                if (l == lane) mine = s;
            }
        }
        if (prefix && j + lane < n) prefix[j + lane] = mine;
    }
    return s;
}

// One block of four warps per bin (:3495-3559). What bounds it is the serial chains, so the three recurrences run
// at the same time in a warp each: the downward log-derivative D_{n-1} = n/z - 1/(D_n + n/z) (for a real index in
// real arithmetic, where every imaginary part is exactly zero), and the upward Riccati-Bessel psi and chi. What is
// independent across orders is spread over all threads: the n/z and (2n+1)/x quotients before them, the a_n, b_n
// quotients and the terms of the efficiency sums after them. The six sums then run in six lanes of one warp.
// Every value has the one-thread expression, and every sum its order. The 63 bins of the full scene (up to 1500
// orders): 4.46 ms with the recurrences and sums one after the other in one lane.
// Shared memory: D[0..nmx], n/z[0..nmx] (complex) and psi[0..nstop+1], chi[0..nstop+1] (real), laid out
// for `order_cap` orders (at most CLR_MIE_MAX_ORDER; a launch over small particles asks for less, so more
// blocks share an SM). The a_n, b_n rows of `ab` are `order_cap` orders apart.
__host__ __device__ constexpr size_t mie_smem_bytes(int order_cap) {
    return (size_t)2 * (order_cap + 1) * sizeof(cdx) + (size_t)2 * (order_cap + 2) * sizeof(double);
}
constexpr size_t kMieSmem = mie_smem_bytes(CLR_MIE_MAX_ORDER);
constexpr int kMieThreads = 128;

__global__ void __launch_bounds__(kMieThreads) mie_coefficients_kernel(
    const double* __restrict__ diameter, const double* __restrict__ n_real, const double* __restrict__ k_imag,
    double n_medium, double wavelength, int n_particles, int order_cap, double* __restrict__ ab,
    int* __restrict__ nstop_out, double* size_parameter, double* qext, double* qsca, double* qabs, double* qback,
    double* asym_g, double* albedo, int* error_flag) {
    extern __shared__ cdx Dsh[];
    cdx* NZ = Dsh + (order_cap + 1);
    double* PSI = reinterpret_cast<double*>(NZ + (order_cap + 1));
    double* CHI = PSI + (order_cap + 2);
    const int p = n_particles - 1 - (int)blockIdx.x;  // the large sizes, usually last, first
    const int tid = threadIdx.x;
    double x = PD_PI * n_medium * diameter[p] / wavelength;
    if (!(x > 0.0) || !(n_real[p] > 0.0) || !(n_medium > 0.0) || !(wavelength > 0.0)) {
        if (tid == 0) {
            size_parameter[p] = x;
            nstop_out[p] = 0; qext[p] = qsca[p] = qabs[p] = qback[p] = asym_g[p] = 0.0; albedo[p] = 1.0;
            atomicCAS(error_flag, 0, 2);
        }
        return;
    }
    double mr = n_real[p] / n_medium, mi = k_imag[p] / n_medium;
    int nstop = (int)(x + 4.0 * cbrt(x) + 2.0);
    if (nstop < 1) nstop = 1;
    double mz = hypot(mr * x, mi * x);
    int nmx = (int)fmax((double)nstop, mz) + 128;
    if (nmx < nstop + 1) nmx = nstop + 1;
    if (nmx >= CLR_MIE_MAX_ORDER || nstop >= CLR_MIE_MAX_ORDER) {
        if (tid == 0) { size_parameter[p] = x; nstop_out[p] = 0; atomicCAS(error_flag, 0, 1); }
        return;
    }
    if (nmx > order_cap) {  // the host's bound on the orders of this launch was too small (never expected)
        if (tid == 0) { size_parameter[p] = x; nstop_out[p] = 0; atomicCAS(error_flag, 0, CLR_ERR_CODE_ORDER_CAP); }
        return;
    }
    const cdx z = CD(mr * x, mi * x);
    for (int n = 1 + tid; n <= nmx; n += kMieThreads) NZ[n] = cd_div(CD((double)n, 0.0), z);
    // (2n+1)/x of order n waits where psi_{n+1} and chi_{n+1} go: each recurrence reads it before it writes there
    for (int n = 1 + tid; n <= nstop; n += kMieThreads) PSI[n + 1] = CHI[n + 1] = (2.0 * n + 1.0) / x;
    __syncthreads();
    if (tid == 0) {
        size_parameter[p] = x;
        nstop_out[p] = nstop;
        cdx dn = CD(0.0, 0.0);
        Dsh[nmx] = dn;
        cdx nz = NZ[nmx];
        if (mi == 0.0) {
            for (int n = nmx; n >= 1; --n) {
                const cdx cur = nz;
                if (n > 1) nz = NZ[n - 1];
                const double b = dn.re + cur.re;
                dn.re = cur.re - pos_div(b, not_tiny(b * b));
                Dsh[n - 1] = dn;
            }
        } else {
            for (int n = nmx; n >= 1; --n) {
                const cdx cur = nz;
                if (n > 1) nz = NZ[n - 1];
                dn = cd_sub(cur, cd_div(CD(1.0, 0.0), cd_add(dn, cur)));
                Dsh[n - 1] = dn;
            }
        }
    } else if (tid == 32) {
        double psi_nm1 = sin(x), psi_n = sin(x) / x - cos(x);
        PSI[0] = psi_nm1; PSI[1] = psi_n;
        for (int n = 1; n <= nstop; ++n) {
            double psi_np1 = PSI[n + 1] * psi_n - psi_nm1;
            psi_nm1 = psi_n; psi_n = psi_np1;
            PSI[n + 1] = psi_n;
        }
    } else if (tid == 64) {
        double chi_nm1 = cos(x), chi_n = cos(x) / x + sin(x);
        CHI[0] = chi_nm1; CHI[1] = chi_n;
        for (int n = 1; n <= nstop; ++n) {
            double chi_np1 = CHI[n + 1] * chi_n - chi_nm1;
            chi_nm1 = chi_n; chi_n = chi_np1;
            CHI[n + 1] = chi_n;
        }
    }
    __syncthreads();
    const cdx m = CD(mr, mi);
    double4* abp = reinterpret_cast<double4*>(ab) + (size_t)p * order_cap;
    for (int j = tid; j < nstop; j += kMieThreads) {
        int n = j + 1;
        const double psi_nm1 = PSI[n - 1], psi_n = PSI[n], chi_nm1 = CHI[n - 1], chi_n = CHI[n];
        cdx xi_nm1 = CD(psi_nm1, -chi_nm1), xi_n = CD(psi_n, -chi_n);
        cdx dn = Dsh[n];
        cdx ca = cd_add(cd_div(dn, m), CD((double)n / x, 0.0));
        cdx cb = cd_add(cd_mul(m, dn), CD((double)n / x, 0.0));
        cdx aa = cd_div(cd_sub(cd_scale(ca, psi_n), CD(psi_nm1, 0.0)), cd_sub(cd_mul(ca, xi_n), xi_nm1));
        cdx bb = cd_div(cd_sub(cd_scale(cb, psi_n), CD(psi_nm1, 0.0)), cd_sub(cd_mul(cb, xi_n), xi_nm1));
        abp[j] = make_double4(aa.re, aa.im, bb.re, bb.im);
    }
    __syncthreads();
    // terms of the efficiency sums, in the same shared memory (at least 48 bytes per order)
    double* const T = reinterpret_cast<double*>(Dsh);
    const int row = nstop | 1;
    for (int j = tid; j < nstop; j += kMieThreads) {
        const int n = j + 1;
        const double cn = 2.0 * n + 1.0;
        const double4 q = abp[j];
        const cdx aa = CD(q.x, q.y), bb = CD(q.z, q.w);
        const double sign = (n & 1) ? -1.0 : 1.0;
        T[j] = cn * (aa.re + bb.re);
        T[row + j] = cn * (cd_abs2(aa) + cd_abs2(bb));
        T[2 * row + j] = cn * sign * (aa.re - bb.re);
        T[3 * row + j] = cn * sign * (aa.im - bb.im);
        T[4 * row + j] = cn / ((double)n * (n + 1.0)) * cd_rmc(aa, bb);
        double t1 = 0.0;
        if (j + 1 < nstop) {
            const double4 q2 = abp[j + 1];
            const cdx an = CD(q2.x, q2.y), bn = CD(q2.z, q2.w);
            t1 = (double)n * (n + 2.0) / (n + 1.0) * (cd_rmc(aa, an) + cd_rmc(bb, bn));
        }
        T[5 * row + j] = t1;
    }
    __syncthreads();
    if (tid >= 32) return;
    double sum = 0.0;
    if (tid < 6) {
        const double* t = T + tid * row;
        double next = t[0];
        for (int j = 0; j < nstop; ++j) {
            const double v = next;
            if (j + 1 < nstop) next = t[j + 1];
            sum += v;
        }
    }
    const double se = sum, ss = __shfl_sync(0xffffffffu, sum, 1), sbr = __shfl_sync(0xffffffffu, sum, 2),
                 sbi = __shfl_sync(0xffffffffu, sum, 3), t2 = __shfl_sync(0xffffffffu, sum, 4),
                 t1 = __shfl_sync(0xffffffffu, sum, 5);
    if (tid != 0) return;
    double x2 = x * x;
    double qe = 2.0 * se / x2, qs = 2.0 * ss / x2, qb = (sbr * sbr + sbi * sbi) / x2;
    if (qe < 0.0 && qe > -1e-12) qe = 0.0;
    if (qs < 0.0 && qs > -1e-12) qs = 0.0;
    double qa = qe - qs;
    if (qa < 0.0 && qa > -1e-10) qa = 0.0;
    double gg = qs > 0.0 ? 4.0 * (t1 + t2) / (x2 * qs) : 0.0;
    if (gg > 1.0) gg = 1.0;
    if (gg < -1.0) gg = -1.0;
    qext[p] = qe; qsca[p] = qs; qabs[p] = qa; qback[p] = qb; asym_g[p] = gg; albedo[p] = qe > 0.0 ? qs / qe : 1.0;
}

// theta_j = pi/2 (1 - cos(pi j/(nt-1))) (:3488-3493), plus the float copy the sampler reads
__global__ void theta_grid_kernel(double* theta, float* theta_f, int nt) {
    int j = blockDim.x * blockIdx.x + threadIdx.x;
    if (j >= nt) return;
    double v;
    if (j == 0) v = 0.0;
    else if (j == nt - 1) v = PD_PI;
    else { double u = (double)j / (double)(nt - 1); v = 0.5 * PD_PI * (1.0 - cos(PD_PI * u)); }
    theta[j] = v;
    theta_f[j] = (float)v;
}

// pi_n, tau_n of every angle and order (:3561-3581), the same for every bin: table[n - 1][angle], `pitch` angles apart
// (a multiple of 32). One warp per 32 angles: the recurrence is a chain of 8 (kFast: 6, with fused multiply-adds) FP64
// operations per order, which every warp of the pdf kernels would repeat for its own bins (8 of 28 operations with a
// bin per warp, 8 of 88 with four); from the table (L2-resident) they only load. The quotients of an order are
// identical to evaluating them inline. A build of 63 bins x 1801 angles 4.80 -> 4.25 ms, the tables of 128 scenarios
// x 64 bins 173.8 -> 135.8 ms (fast arithmetic 61.2 -> 35.3 ms); the table itself 0.46 ms beside the Mie kernel's 0.93.
constexpr int kLegStage = 64;
template <bool kFast>
__global__ void __launch_bounds__(32) legendre_table_kernel(const double* __restrict__ theta, int angles, int rows,
                                                            int pitch, double2* __restrict__ table) {
    __shared__ double QN[4][kLegStage];  // n, n+1, (2n+1)/n, (n+1)/n
    const int lane = threadIdx.x, j = blockIdx.x * 32 + lane;
    const double mu = j < angles ? cos(theta[j]) : 0.0;
    double pi_nm1 = 0.0, pi_n = 1.0;
    for (int k0 = 0; k0 < rows; k0 += kLegStage) {
        __syncwarp();
#pragma unroll
        for (int kk = lane; kk < kLegStage; kk += 32) {
            const double nf = (double)(k0 + kk + 1);
            QN[0][kk] = nf; QN[1][kk] = nf + 1.0;
            QN[2][kk] = (2.0 * nf + 1.0) / nf;
            QN[3][kk] = (nf + 1.0) / nf;
        }
        __syncwarp();
        const int kend = min(kLegStage, rows - k0);
        for (int kk = 0; kk < kend; ++kk) {
            double tau, pi_np1;
            if constexpr (kFast) {
                tau = fma(QN[0][kk] * mu, pi_n, -QN[1][kk] * pi_nm1);
                pi_np1 = fma(QN[2][kk] * mu, pi_n, -QN[3][kk] * pi_nm1);
            } else {
                tau = QN[0][kk] * mu * pi_n - QN[1][kk] * pi_nm1;
                pi_np1 = QN[2][kk] * mu * pi_n - QN[3][kk] * pi_nm1;
            }
            table[(size_t)(k0 + kk) * pitch + j] = make_double2(pi_n, tau);
            pi_nm1 = pi_n; pi_n = pi_np1;
        }
    }
}

// S1/S2 -> 0.5(|S1|^2+|S2|^2) sin(theta) for kPdfGroup bins at one angle per lane (:3561-3581). Bound by the FP64
// pipe (20 operations per bin and order; without the table of pi_n, tau_n 8 more per order; no contraction).
// A warp issues one FP64 instruction per 64 cycles, so few bins make the largest sizes' warps the longest: with four
// bins to a warp in blocks of 128 angles, the last blocks of 63 bins ran 4.4 ms where the pipe's work is 1.2 ms.
// One warp per block, the last bins (usually the largest, with the most orders) first, and one bin to a warp: with the
// table, four bins would only share its loads, which the FP64 pipe hides, and are slower at every size (ms in the
// reference's order / fast: 640 bins of the sweep workload 11.2 / 3.4 against 14.9 / 4.2 with four, 4096 bins 64.3 /
// 15.4 against 66.8 / 17.7; 640 bins of 257 angles 3.2 / 1.8 against 4.6 / 2.6).
// Coefficients and the quotients of an order (identical to evaluating them inline) are staged kPdfStage orders at
// a time.
// Without the table (thousands of angles and orders, so warps enough) four bins to a warp share the recurrence: 22
// operations per bin and order instead of 28 (fast arithmetic 17.5 instead of 22). The line is where that outweighs
// the longer warps of the largest sizes in both arithmetics (one bin / four bins, ms; 12289 angles in the reference's
// order, 24001 fast): 141 bins 28.7 / 30.0 and 14.5 / 12.6, 188 bins 38.0 / 36.9 and 19.0 / 15.9, 611 bins 120.5 /
// 101.1 and 58.5 / 47.5.
constexpr int kPdfManyBins = 160;
// Unused shared memory per block of one bin: about a dozen blocks per SM, the rest wait, so that a partition whose warps
// end early takes the next (282 bins of 1801 angles 5.9 ms, 7.2 with all resident; the fast kernel, whose own 4 KB are
// nearly the same, 1.8 ms against 2.0 for 141 bins of 2401 angles and within 3 % at most other sizes).
constexpr int kPdfPad = 14 * 1024;
constexpr int kPdfStage = 64;
template <int kPdfGroup, bool kTable>
__global__ void __launch_bounds__(32) phase_pdf_kernel(const double* __restrict__ theta, int nt, int n_particles,
                                                       int order_cap, const int* __restrict__ nstop,
                                                       const double* __restrict__ ab, const double2* __restrict__ table,
                                                       int pitch, double* __restrict__ pdf) {
    __shared__ double4 AB[kPdfGroup][kPdfStage];
    __shared__ double QN[5][kPdfStage];  // n, n+1, (2n+1)/(n(n+1)), (2n+1)/n, (n+1)/n
    const int lane = threadIdx.x, j = blockIdx.x * 32 + lane;
    const int g0 = (int)(gridDim.y - 1 - blockIdx.y) * kPdfGroup;
    const double th = j < nt ? theta[j] : 0.0, mu = kTable ? 0.0 : cos(th);
    double s1r[kPdfGroup], s1i[kPdfGroup], s2r[kPdfGroup], s2i[kPdfGroup];
    int ns[kPdfGroup];
    int kmax = 0;
#pragma unroll
    for (int g = 0; g < kPdfGroup; ++g) {
        s1r[g] = s1i[g] = s2r[g] = s2i[g] = 0.0;
        ns[g] = (g0 + g < n_particles) ? nstop[g0 + g] : 0;
        kmax = ns[g] > kmax ? ns[g] : kmax;
    }
    const double4* abp = reinterpret_cast<const double4*>(ab);
    double pi_nm1 = 0.0, pi_n = 1.0;
    double2 pt = make_double2(0.0, 0.0);
    if (kTable && kmax > 0) pt = table[j];
    for (int k0 = 0; k0 < kmax; k0 += kPdfStage) {
        __syncwarp();
#pragma unroll
        for (int h = 0; h < kPdfStage; h += 32) {
            const int kk = h + lane, k = k0 + kk;
            const double nf = (double)(k + 1);
            QN[2][kk] = (2.0 * nf + 1.0) / (nf * (nf + 1.0));
            if constexpr (!kTable) {
                QN[0][kk] = nf; QN[1][kk] = nf + 1.0;
                QN[3][kk] = (2.0 * nf + 1.0) / nf;
                QN[4][kk] = (nf + 1.0) / nf;
            }
#pragma unroll
            for (int g = 0; g < kPdfGroup; ++g)
                if (k < ns[g]) AB[g][kk] = abp[(size_t)(g0 + g) * order_cap + k];
        }
        __syncwarp();
        const int kend = min(kPdfStage, kmax - k0);
        for (int kk = 0; kk < kend; ++kk) {
            double tau;
            if constexpr (kTable) {
                pi_n = pt.x; tau = pt.y;
                if (k0 + kk + 1 < kmax) pt = table[(size_t)(k0 + kk + 1) * pitch + j];
            } else {
                tau = QN[0][kk] * mu * pi_n - QN[1][kk] * pi_nm1;
            }
            const double c = QN[2][kk];
#pragma unroll
            for (int g = 0; g < kPdfGroup; ++g) {
                if (k0 + kk < ns[g]) {
                    const double4 q = AB[g][kk];
                    const double ar = q.x, ai = q.y, br = q.z, bi = q.w;
                    s1r[g] += c * (ar * pi_n + br * tau);
                    s1i[g] += c * (ai * pi_n + bi * tau);
                    s2r[g] += c * (ar * tau + br * pi_n);
                    s2i[g] += c * (ai * tau + bi * pi_n);
                }
            }
            if constexpr (!kTable) {
                const double pi_np1 = QN[3][kk] * mu * pi_n - QN[4][kk] * pi_nm1;
                pi_nm1 = pi_n; pi_n = pi_np1;
            }
        }
    }
    if (j >= nt) return;
#pragma unroll
    for (int g = 0; g < kPdfGroup; ++g) {
        if (g0 + g < n_particles) {
            double intensity = 0.5 * (s1r[g] * s1r[g] + s1i[g] * s1i[g] + s2r[g] * s2r[g] + s2i[g] * s2i[g]);
            pdf[(size_t)(g0 + g) * nt + j] = intensity * sin(th);
        }
    }
}

// Production variant of the phase pdf (CLR_TABLES_FAST; no reference counterpart). The same S1/S2 sums,
// evaluated with fused multiply-adds on coefficients premultiplied by (2n+1)/(n(n+1)) (staged per block in
// shared memory), and for two angles at once: theta_j and theta_{nt-1-j}, which is pi - theta_j on the
// reference's grid to rounding. With pi_n(-mu) = (-1)^(n-1) pi_n(mu) and tau_n(-mu) = (-1)^n tau_n(mu), the
// sums over odd and over even orders of a pi_n, b tau_n, a tau_n and b pi_n give S1 and S2 at mu and at
// -mu: 8 FMAs per (bin, order) for both angles, against about 44 FP64 operations of the reference's order
// of operations for the two. Tables differ from the reference-order ones by rounding only (tested).
// pi_n and tau_n come from the table, for one bin in a one-warp block, the last bins first; many bins without a table
// share the recurrence, four to a block (both by the rule of phase_pdf_kernel).
constexpr int kPdfFastChunk = 128;  // orders staged per block
template <int kPdfFastGroup, int kThreads, bool kTable>
__global__ void __launch_bounds__(kThreads) phase_pdf_fast_kernel(const double* __restrict__ theta, int nt,
                                                             int n_particles, int order_cap,
                                                             const int* __restrict__ nstop,
                                                             const double* __restrict__ ab,
                                                             const double2* __restrict__ table, int pitch,
                                                             double* __restrict__ pdf) {
    __shared__ double4 AB[kPdfFastGroup][kPdfFastChunk];
    __shared__ double2 RC[kTable ? 1 : kPdfFastChunk];  // without the table: (2n+1)/n, (n+1)/n of the staged orders
    __shared__ double2 NF[kTable ? 1 : kPdfFastChunk];  // n, -(n+1)
    const int g0 = (int)(gridDim.y - 1 - blockIdx.y) * kPdfFastGroup;
    const int npair = (nt + 1) / 2;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = j < npair;
    int ns[kPdfFastGroup];
    int kmax = 0;
#pragma unroll
    for (int g = 0; g < kPdfFastGroup; ++g) {
        ns[g] = (g0 + g < n_particles) ? nstop[g0 + g] : 0;
        kmax = ns[g] > kmax ? ns[g] : kmax;
    }
    // per bin: odd-order sums P = a pi, Q = b tau, R = a tau, T = b pi (re, im), then the even-order ones
    double acc[kPdfFastGroup][16];
#pragma unroll
    for (int g = 0; g < kPdfFastGroup; ++g)
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[g][i] = 0.0;
    const double4* ab4 = reinterpret_cast<const double4*>(ab);
    // threads past the last pair of angles read the row's padding (or its last angle) and store nothing
    const double2* const col = kTable ? table + min(j, pitch - 1) : nullptr;
    double2 next[2] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
    if (kTable && kmax > 0) next[0] = col[0];
    if (kTable && kmax > 1) next[1] = col[pitch];
    const double mu = !kTable && active ? cos(theta[j]) : 0.0;
    double pi_nm1 = 0.0, pi_n = 1.0;
    for (int k0 = 0; k0 < kmax; k0 += kPdfFastChunk) {
        __syncthreads();
        for (int idx = threadIdx.x; idx < kPdfFastGroup * kPdfFastChunk; idx += blockDim.x) {
            const int g = idx / kPdfFastChunk, kk = idx % kPdfFastChunk, k = k0 + kk;
            double4 v = make_double4(0.0, 0.0, 0.0, 0.0);
            if (k < ns[g]) {
                const double4 q = ab4[(size_t)(g0 + g) * order_cap + k];
                const double nf = (double)(k + 1);
                const double c = (2.0 * nf + 1.0) / (nf * (nf + 1.0));
                v = make_double4(c * q.x, c * q.y, c * q.z, c * q.w);
            }
            AB[g][kk] = v;
        }
        if constexpr (!kTable)
            for (int kk = threadIdx.x; kk < kPdfFastChunk; kk += blockDim.x) {
                const double nf = (double)(k0 + kk + 1);
                RC[kk] = make_double2((2.0 * nf + 1.0) / nf, (nf + 1.0) / nf);
                NF[kk] = make_double2(nf, -(nf + 1.0));
            }
        __syncthreads();
        const int kend = min(kPdfFastChunk, kmax - k0);
        // k0 is even, so order n = k0 + kk + 1 is odd for even kk: odd-order sums go to acc[g][0..7], even-order
        // ones to acc[g][8..15]; the pair loop keeps every index a compile-time constant (registers, no stack).
        // Orders past kend carry zero coefficients, so the pair's second half may run past it.
        for (int kk = 0; kk < kend; kk += 2) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                double tau;
                if constexpr (kTable) {
                    pi_n = next[h].x; tau = next[h].y;
                    if (k0 + kk + h + 2 < kmax) next[h] = col[(size_t)(k0 + kk + h + 2) * pitch];
                } else {
                    tau = fma(NF[kk + h].x * mu, pi_n, NF[kk + h].y * pi_nm1);
                }
#pragma unroll
                for (int g = 0; g < kPdfFastGroup; ++g) {
                    const double4 q = AB[g][kk + h];
                    double* A = acc[g] + 8 * h;
                    A[0] = fma(q.x, pi_n, A[0]); A[1] = fma(q.y, pi_n, A[1]);  // P
                    A[2] = fma(q.z, tau, A[2]);  A[3] = fma(q.w, tau, A[3]);   // Q
                    A[4] = fma(q.x, tau, A[4]);  A[5] = fma(q.y, tau, A[5]);   // R
                    A[6] = fma(q.z, pi_n, A[6]); A[7] = fma(q.w, pi_n, A[7]);  // T
                }
                if constexpr (!kTable) {
                    const double pi_np1 = fma(RC[kk + h].x * mu, pi_n, -RC[kk + h].y * pi_nm1);
                    pi_nm1 = pi_n; pi_n = pi_np1;
                }
            }
        }
    }
    if (!active) return;
    const int jm = nt - 1 - j;
    const double sj = sin(theta[j]), sm = sin(theta[jm]);
#pragma unroll
    for (int g = 0; g < kPdfFastGroup; ++g) {
        if (g0 + g >= n_particles) continue;
        const double* o = acc[g];
        const double* e = acc[g] + 8;
        // S1(mu) = Po+Qo+Pe+Qe, S1(-mu) = Po-Qo-Pe+Qe, S2(mu) = Ro+To+Re+Te, S2(-mu) = -Ro+To+Re-Te
        const double s1r = o[0] + o[2] + e[0] + e[2], s1i = o[1] + o[3] + e[1] + e[3];
        const double s2r = o[4] + o[6] + e[4] + e[6], s2i = o[5] + o[7] + e[5] + e[7];
        pdf[(size_t)(g0 + g) * nt + j] = 0.5 * (s1r * s1r + s1i * s1i + s2r * s2r + s2i * s2i) * sj;
        if (jm != j) {
            const double m1r = o[0] - o[2] - e[0] + e[2], m1i = o[1] - o[3] - e[1] + e[3];
            const double m2r = -o[4] + o[6] + e[4] - e[6], m2i = -o[5] + o[7] + e[5] - e[7];
            pdf[(size_t)(g0 + g) * nt + jm] = 0.5 * (m1r * m1r + m1i * m1i + m2r * m2r + m2i * m2i) * sm;
        }
    }
}

// Trapezoid CDF per bin, normalised and forced monotone (:3583-3592); also the float copy. One block per bin: the
// trapezoid areas and the normalised values are independent per angle; the prefix sum runs in one warp in the
// serial order. A sum of non-negative areas divided by its total never decreases or passes 1, so the serial clamp
// runs only where a value says otherwise. The row is kept in shared memory where it fits. (63 bins, 1801 angles:
// 0.34 ms with one warp per bin and the sum in global memory.)
constexpr int kCdfThreads = 128;
constexpr int kCdfSmemAngles = 12288;
__global__ void __launch_bounds__(kCdfThreads) phase_cdf_kernel(const double* __restrict__ theta,
                                                                const double* __restrict__ pdf, int nt, int n_particles,
                                                                double* __restrict__ cdf, float* __restrict__ cdf_f,
                                                                int* error_flag) {
    extern __shared__ double cdf_row[];
    __shared__ double total;
    const int p = blockIdx.x, tid = threadIdx.x;
    const long long base = (long long)p * nt;
    double* const row = nt <= kCdfSmemAngles ? cdf_row : cdf + base;
    for (int j = 1 + tid; j < nt; j += kCdfThreads) {
        double area = 0.5 * (pdf[base + j] + pdf[base + j - 1]) * (theta[j] - theta[j - 1]);
        if (area < 0.0 && area > -1e-18) area = 0.0;
        row[j] = area;
    }
    if (tid == 0) row[0] = 0.0;
    __syncthreads();
    if (tid < 32) {
        const double s = warp_serial_sum(row, nt, row);
        if (tid == 0) total = s;
    }
    __syncthreads();
    const double s = total;
    if (!(s > 0.0) || !isfinite(s)) {
        if (tid == 0) atomicCAS(error_flag, 0, 3);
        for (int j = tid; j < nt; j += kCdfThreads) {
            const double v = (double)j / (double)(nt - 1);
            cdf[base + j] = v;
            cdf_f[base + j] = (float)v;
        }
        return;
    }
    for (int j = tid; j < nt; j += kCdfThreads) row[j] = row[j] / s;
    __syncthreads();
    bool clamp = false;
    for (int j = tid; j < nt; j += kCdfThreads) clamp |= !(row[j] >= (j ? row[j - 1] : 0.0) && row[j] <= 1.0);
    if (__syncthreads_or(clamp)) {
        if (tid == 0) {
            double prev = 0.0;
            for (int j = 0; j < nt; ++j) {
                double v = row[j];
                if (v < prev) v = prev;
                if (v > 1.0) v = 1.0;
                row[j] = v;
                prev = v;
            }
        }
        __syncthreads();
    }
    for (int j = tid; j < nt; j += kCdfThreads) {
        const double v = j == nt - 1 ? 1.0 : row[j];
        cdf[base + j] = v;
        cdf_f[base + j] = (float)v;
    }
}

// guide[p][k] = the first index j of bin p with cdf_f[j] >= k / kPhaseGuide (nt - 1 when none), found by the
// photon kernels' own search, so that a search restricted to [guide[k], guide[k+1]] returns its index
__global__ void phase_guide_kernel(const float* __restrict__ cdf_f, int nt, int n_particles, int* __restrict__ guide) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)n_particles * (kPhaseGuide + 1)) return;
    const int p = (int)(t / (kPhaseGuide + 1)), k = (int)(t % (kPhaseGuide + 1));
    const float u = (float)k / (float)kPhaseGuide;
    const float* c = cdf_f + (size_t)p * nt;
    int lo = 0, hi = nt - 1;
    while (lo < hi) { const int mid = (lo + hi) >> 1; if (u <= c[mid]) hi = mid; else lo = mid + 1; }
    guide[t] = lo;
}

__global__ void dummy_phase_kernel(double* theta, float* theta_f, double* cdf, float* cdf_f, int n_particles) {
    int p = blockDim.x * blockIdx.x + threadIdx.x;
    if (p == 0) { theta[0] = 0.0; theta[1] = PD_PI; theta_f[0] = 0.0f; theta_f[1] = (float)PD_PI; }
    if (p < n_particles) { cdf[2 * p] = 0.0; cdf[2 * p + 1] = 1.0; cdf_f[2 * p] = 0.0f; cdf_f[2 * p + 1] = 1.0f; }
}

// PSD normalisation (:3615-3635), rates and channel CDFs (:3845-3921), channel rate arrays
// (:6362-6375) and the float copies the photon kernel reads. One warp, n <= 64 bins: what is per bin runs in the
// lanes (two bins each), every sum serially over the bins in a lane of its own, from shared memory. Values and
// orders are those of the one-thread loop, which took 260 us for 63 bins: its dependent global accesses.
__device__ __forceinline__ double bin_sum(const double* v, int n, double* prefix = nullptr) {
    double s = 0.0;
    for (int i = 0; i < n; ++i) {
        s += v[i];
        if (prefix) prefix[i] = s;
    }
    return s;
}
__device__ __noinline__ void transport_body(int n, const double* __restrict__ d, const double* __restrict__ w_in,
                                            const double* __restrict__ qext, const double* __restrict__ qsca,
                                            const double* __restrict__ k_imag, const double* __restrict__ n_real,
                                            double concentration, double density, int weight_mode, int em,
                                            double wave_scale, double n_medium, double wavelength, double wave_rms,
                                            double* w, double* radius, double* nden, double* mug, double* mus,
                                            double* mue, double* muw, double* muev, double* gcdf, double* wcdf,
                                            double* pcdf, double* muscal, double* trace_geom, double* trace_wave,
                                            float* gcdf_f, float* wcdf_f, float* pn_f, float* pk_f, float* prad_f,
                                            int* error_flag) {
    __shared__ double B[5][CLR_MAX_BINS];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x;
    if (n < 1 || n > CLR_MAX_BINS) { if (lane == 0) atomicCAS(error_flag, 0, 20); return; }
    if (!(density > 0.0) || concentration < 0.0) { if (lane == 0) atomicCAS(error_flag, 0, 21); return; }
    for (int i = lane; i < n; i += 32) B[0][i] = w_in[i];
    __syncwarp();
    const double sw0 = bin_sum(B[0], n);
    if (!(sw0 > 0.0)) { if (lane == 0) atomicCAS(error_flag, 0, 22); return; }
    for (int i = lane; i < n; i += 32) {
        const double v = w_in[i] / sw0;
        w[i] = v;
        B[1][i] = v;
    }
    __syncwarp();
    const double sw = bin_sum(B[1], n);
    if (!(sw > 0.0)) { if (lane == 0) atomicCAS(error_flag, 0, 4); return; }
    for (int i = lane; i < n; i += 32) {
        const double r = 0.5 * d[i], m = density * (4.0 / 3.0) * PD_PI * r * r * r;
        radius[i] = r;
        B[2][i] = B[1][i] / sw;
        B[3][i] = m;
        B[0][i] = B[2][i] * m;
    }
    __syncwarp();
    const double avg_mass = bin_sum(B[0], n);
    double vg[2], vs[2], ve[2], vw[2];
    bool bad = false;
    for (int h = 0; h < 2; ++h) {
        const int i = h * 32 + lane;
        if (i >= n) continue;
        double nd = 0.0;
        if (weight_mode == 0) nd = concentration * B[2][i] / B[3][i];
        else nd = (avg_mass > 0.0 ? concentration / avg_mass : 0.0) * B[2][i];
        nden[i] = nd;
        const double r = 0.5 * d[i], qe = qext[i], qs = qsca[i], ki = k_imag[i];
        double sg = PD_PI * r * r, sa = fmax(qs, 0.0) * sg, se = fmax(qe, 0.0) * sg;
        double tol = 1e-10 * fmax(1.0, fmax(fabs(qe), fabs(qs)));
        bad |= !isfinite(ki) || ki < 0.0 || !isfinite(qe) || !isfinite(qs) || qe < -tol || qs < -tol ||
               qs > qe + tol || (ki == 0.0 && fabs(qe - qs) > tol);
        double swv = 0.0;
        if (em == 3) swv = wave_scale * fmax(qs - 1.0, 0.0) * sg;
        else if (em == 4 || em == 5) {
            double rate = (ki > 0.0) ? se : sa;
            swv = (ki > 0.0) ? ((sa > 0.0) ? rate * fmax(sa - sg, 0.0) / sa : 0.0) : fmax(sa - sg, 0.0);
        }
        vg[h] = nd * sg; vs[h] = nd * sa; ve[h] = nd * se; vw[h] = nd * swv;
    }
    if (__any_sync(FULL, bad)) { if (lane == 0) atomicCAS(error_flag, 0, 5); return; }
    __syncwarp();
    for (int h = 0; h < 2; ++h) {
        const int i = h * 32 + lane;
        if (i >= n) continue;
        mug[i] = vg[h]; mus[i] = vs[h]; mue[i] = ve[h]; muw[i] = vw[h];
        const double ki = k_imag[i];
        double mb;
        if (em == 0) mb = vg[h];
        else if (em == 1) mb = vs[h];
        else if (em == 2) mb = ve[h];
        else if (em == 3) mb = vg[h] + vw[h];
        else mb = (ki > 0.0) ? ve[h] : vs[h];
        muev[i] = mb;
        B[0][i] = vg[h]; B[1][i] = vs[h]; B[2][i] = ve[h]; B[3][i] = vw[h]; B[4][i] = mb;
    }
    __syncwarp();
    const double part = lane < 5 ? bin_sum(B[lane], n) : 0.0;
    const double mg = __shfl_sync(FULL, part, 0), ms = __shfl_sync(FULL, part, 1), me = __shfl_sync(FULL, part, 2),
                 mw = __shfl_sync(FULL, part, 3), mt = __shfl_sync(FULL, part, 4);
    const bool hyb = (em == 3) || (em == 4) || (em == 5);
    double mtrace_geom = ((em == 4) || (em == 5)) ? fmax(mt - mw, 0.0) : ((em == 3) ? mg : mt);
    double mtrace_wave = hyb ? mw : 0.0;
    for (int i = lane; i < n; i += 32) {
        const double ev = B[4][i], wv = B[3][i], ge = B[0][i];
        double mgi = ((em == 4) || (em == 5)) ? fmax(ev - wv, 0.0) : ge;
        double pg = hyb ? (mtrace_geom > 0.0 ? mgi / mtrace_geom : 0.0) : (mt > 0.0 ? ev / mt : 0.0);
        double pw = (hyb && mtrace_wave > 0.0 ? wv / mtrace_wave : 0.0), pt = (mt > 0.0 ? ev / mt : 0.0);
        if (em == 3) { trace_geom[i] = ge; trace_wave[i] = wv; }
        else if (em == 4 || em == 5) { trace_geom[i] = fmax(ev - wv, 0.0); trace_wave[i] = wv; }
        else { trace_geom[i] = ev; trace_wave[i] = 0.0; }
        B[0][i] = pg; B[1][i] = pw; B[2][i] = pt;
    }
    __syncwarp();
    if (lane < 3 && bin_sum(B[lane], n, B[lane]) > 0.0) B[lane][n - 1] = 1.0;
    __syncwarp();
    for (int i = lane; i < n; i += 32) {
        gcdf[i] = B[0][i]; wcdf[i] = B[1][i]; pcdf[i] = B[2][i];
        gcdf_f[i] = (float)B[0][i];
        wcdf_f[i] = (float)B[1][i];
        pn_f[i] = (float)n_real[i];
        pk_f[i] = (float)k_imag[i];
        prad_f[i] = (float)(0.5 * d[i]);
    }
    if (lane == 0) {
        muscal[0] = mtrace_geom; muscal[1] = mtrace_wave; muscal[2] = mg; muscal[3] = ms;
        muscal[4] = me; muscal[5] = mtrace_wave; muscal[6] = mt;
        double cwave = 1.0;
        if (hyb && wave_rms > 0.0 && wavelength > 0.0 && n_medium > 0.0) {
            double a = 4.0 * PD_PI * n_medium * wave_rms / wavelength;
            cwave = exp(-a * a);
            if (cwave < 0.0) cwave = 0.0;
            if (cwave > 1.0) cwave = 1.0;
        }
        muscal[7] = cwave;
    }
}

// The rates of one scenario and of many scenarios in one launch (a warp per scenario).
struct TransportJob {
    int n, weight_mode, em;
    const double *d, *w_in, *qext, *qsca, *k_imag, *n_real;
    double concentration, density, wave_scale, n_medium, wavelength, wave_rms;
    double *w, *radius, *nden, *mug, *mus, *mue, *muw, *muev, *gcdf, *wcdf, *pcdf, *muscal, *trace_geom, *trace_wave;
    float *gcdf_f, *wcdf_f, *pn_f, *pk_f, *prad_f;
    int* error_flag;
};
__device__ __forceinline__ void transport_job(const TransportJob& j) {
    transport_body(j.n, j.d, j.w_in, j.qext, j.qsca, j.k_imag, j.n_real, j.concentration, j.density, j.weight_mode,
                   j.em, j.wave_scale, j.n_medium, j.wavelength, j.wave_rms, j.w, j.radius, j.nden, j.mug, j.mus,
                   j.mue, j.muw, j.muev, j.gcdf, j.wcdf, j.pcdf, j.muscal, j.trace_geom, j.trace_wave, j.gcdf_f,
                   j.wcdf_f, j.pn_f, j.pk_f, j.prad_f, j.error_flag);
}
__global__ void __launch_bounds__(32) transport_kernel(TransportJob j) { transport_job(j); }
__global__ void __launch_bounds__(32) transport_batch_kernel(const TransportJob* __restrict__ jobs) {
    transport_job(jobs[blockIdx.x]);
}

// Schiller-Naumann terminal velocity by damped Newton (:3925-3937)
__device__ double sn_velocity(double v0, double d, double rho_w, double mu, double* out_Re, double* out_drag) {
    if (!(v0 > 0.0)) { *out_Re = 0.0; *out_drag = 1.0; return 0.0; }
    double v = v0, K = rho_w * d / mu;
    for (int it = 0; it < 24; ++it) {
        double Re = fmax(K * v, 0.0);
        double corr = 0.15 * pow(Re, 0.687);
        double f = v * (1.0 + corr) - v0;
        double df = 1.0 + 1.687 * corr;
        double vn = fmax(v - f / df, 0.0);
        if (fabs(vn - v) <= 2e-14 * fmax(1.0, fabs(v))) { v = vn; break; }
        v = vn;
    }
    double Re = fmax(K * v, 0.0), drag = 1.0 + 0.15 * pow(Re, 0.687);
    *out_Re = Re; *out_drag = drag;
    return v;
}

struct SedArgs {
    int n, TM, FSM, NQ, NRAD;
    double rho_p, rho_w, mu, grav, Dt, R, ZMIN, ZMEAN, DH, CORE;
};

__device__ __forceinline__ void sed_geometry(const SedArgs& a, double* R2, double* a2, double* Hinf, double* hbar,
                                             double* omega2, double* fR) {
    *R2 = a.R * a.R; *a2 = a.CORE * a.CORE; *Hinf = 0.0; *hbar = 0.0; *omega2 = 0.0;
    if (a.DH > 0.0 && a.FSM == 1) { *Hinf = a.DH; *hbar = 0.5 * a.DH; *omega2 = 2.0 * a.grav * a.DH / *R2; }
    else if (a.DH > 0.0 && a.FSM == 2) {
        *Hinf = a.DH * (*a2 + *R2) / *R2;
        *hbar = *Hinf * (1.0 - (*a2 / *R2) * log1p(*R2 / *a2));
        *omega2 = 2.0 * a.grav * *Hinf / *a2;
    }
    *fR = (a.FSM == 2) ? *R2 / (*a2 + *R2) : *R2;
}

// Per-bin radial slip table: one thread per (bin, radius) for the finite-Re models (:3975-3986).
__global__ void sediment_slip_kernel(SedArgs a, const double* __restrict__ diameter, double* __restrict__ wr_out) {
    const int i = blockIdx.y;
    const int j = blockDim.x * blockIdx.x + threadIdx.x;
    if (i >= a.n || j >= a.NRAD || a.TM == 0 || a.TM == 1) return;
    double R2, a2, Hinf, hbar, omega2, fR;
    sed_geometry(a, &R2, &a2, &Hinf, &hbar, &omega2, &fR);
    double d = diameter[i];
    double tau = a.rho_p * d * d / (18.0 * a.mu);
    double drad = a.R / (double)(a.NRAD - 1);
    double r = (double)j * drad, acc = 0.0;
    if (r > 0.0) acc = (a.FSM == 1) ? omega2 * r : ((a.FSM == 2) ? omega2 * r / pow(1.0 + r * r / a2, 2.0) : 0.0);
    double w0 = tau * acc, re = 0.0, drag = 1.0;
    wr_out[(size_t)i * a.NRAD + j] = sn_velocity(w0, d, a.rho_w, a.mu, &re, &drag);
}

// Per-bin coefficients, radial potential and normalisation (:3958-4035); one block per bin. The prefix sums of
// the radial potential and the quadrature sum run in the serial order in one warp (the potential's total is the
// last of its prefix sums: the reference adds the same terms twice); everything per radius, and the quadrature
// terms, each an independent exp/expm1 evaluation, in all threads. (63 bins, 2049 radii, 4096 points: 1.84 ms with
// the sums in one lane.)
constexpr int kSedThreads = 128;
__global__ void __launch_bounds__(kSedThreads) sediment_bin_kernel(SedArgs a, const double* __restrict__ diameter,
                                                                   const double* __restrict__ wr, double* sedA,
                                                                   double* sedB, double* sed_norm, double* sed_max,
                                                                   double* radial_log, double* terms, double* ws_out,
                                                                   int* error_flag) {
    __shared__ double shared_ws;
    const int i = blockIdx.x;
    const int tid = threadIdx.x;
    if (a.TM == 0) {
        if (tid == 0) { sedA[i] = 0.0; sedB[i] = 0.0; sed_norm[i] = 1.0; sed_max[i] = 1.0; ws_out[i] = 0.0; }
        return;
    }
    double R2, a2, Hinf, hbar, omega2, fR;
    sed_geometry(a, &R2, &a2, &Hinf, &hbar, &omega2, &fR);
    const double R = a.R, ZMIN = a.ZMIN, ZMEAN = a.ZMEAN, DH = a.DH;
    const int NRAD = a.NRAD, NQ = a.NQ, FSM = a.FSM, TM = a.TM;
    double Hmean = ZMEAN - ZMIN, dr = R / (double)NQ, drad = R / (double)(NRAD - 1);
    double d = diameter[i];
    double tau = a.rho_p * d * d / (18.0 * a.mu);
    double* RL = radial_log + (size_t)i * NRAD;
    const double Ac = tau * omega2 * ((FSM == 2) ? a2 : 1.0) / (2.0 * a.Dt);
    if (tid == 0) {
        double ws0 = (a.rho_p - a.rho_w) * a.grav * d * d / (18.0 * a.mu);
        double sre = 0.0, sdrag = 1.0;
        shared_ws = (TM == 2 || TM == 3) ? sn_velocity(ws0, d, a.rho_w, a.mu, &sre, &sdrag) : ws0;
    }
    if (TM == 1) {
        for (int j = tid; j < NRAD; j += kSedThreads) {
            double r = (double)j * drad, rr2 = r * r, f = (FSM == 2) ? rr2 / (a2 + rr2) : rr2;
            RL[j] = Ac * (f - fR);
        }
    } else {
        const double* W = wr + (size_t)i * NRAD;
        for (int j = tid; j < NRAD; j += kSedThreads) RL[j] = j > 0 ? 0.5 * (W[j - 1] + W[j]) * drad : 0.0;
        __syncthreads();
        if (tid < 32) (void)warp_serial_sum(RL, NRAD, RL);
        __syncthreads();
        const double total = RL[NRAD - 1];
        __syncthreads();
        for (int j = tid; j < NRAD; j += kSedThreads) {
            double psi = (RL[j] - total) / a.Dt;
            if (psi > 0.0) psi = 0.0;
            RL[j] = j == NRAD - 1 ? 0.0 : psi;
        }
    }
    __syncthreads();
    const double ws = shared_ws, Bc = ws / a.Dt;
    const double A_i = (TM == 1) ? Ac : ((fR > 0.0) ? -RL[0] / fR : 0.0);
    if (tid == 0) { sedA[i] = A_i; sedB[i] = Bc; ws_out[i] = ws; }
    double* T = terms + (size_t)i * NQ;
    for (int j = tid; j < NQ; j += kSedThreads) {
        double r = ((double)j + 0.5) * dr, rr2 = r * r;
        double zsurf = ZMEAN;
        if (FSM == 1 && DH > 0.0) zsurf = ZMEAN + DH * (rr2 / R2 - 0.5);
        else if (FSM == 2 && DH > 0.0) zsurf = ZMEAN - hbar + Hinf * rr2 / (a2 + rr2);
        double Hh = fmax(zsurf - ZMIN, 0.0);
        double rl;
        if (TM == 1) {
            double f = (FSM == 2) ? rr2 / (a2 + rr2) : rr2;
            rl = A_i * (f - fR);
        } else {
            double u = r / R * (double)(NRAD - 1);
            int k = (int)floor(u);
            if (k < 0) k = 0;
            if (k > NRAD - 2) k = NRAD - 2;
            double t = u - (double)k;
            rl = (1.0 - t) * RL[k] + t * RL[k + 1];
            if (rl > 0.0) rl = 0.0;
        }
        double radial = exp(rl);
        double iz = (fabs(Bc) < 1e-14) ? radial * Hh : radial * (-expm1(-Bc * Hh)) / Bc;
        T[j] = r * iz;
    }
    __syncthreads();
    if (tid >= 32) return;
    const double integ = warp_serial_sum(T, NQ, nullptr);
    if (tid != 0) return;
    double norm = (2.0 / (R2 * Hmean)) * integ * dr;
    if (!(norm > 0.0) || !isfinite(norm)) { atomicCAS(error_flag, 0, 34); return; }
    sed_norm[i] = norm;
    sed_max[i] = 1.0 / norm;
}

// Per-bin maximum of the (r, z) grid (the max of non-negative terms starting at 0, as the reference's
// serial scan, so the order of the reduction does not change the value). One block per bin.
__global__ void sediment_grid_max_kernel(const double* __restrict__ grid, long long plane, double* grid_max) {
    const int p = blockIdx.x;
    double mx = 0.0;
    for (long long c = threadIdx.x; c < plane; c += blockDim.x) {
        const double q = grid[p * plane + c];
        if (q > mx) mx = q;
    }
    __shared__ double red[256];
    red[threadIdx.x] = mx;
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h && red[threadIdx.x + h] > red[threadIdx.x]) red[threadIdx.x] = red[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) grid_max[p] = red[0];
}

// One warp, n <= 64 bins: the products in the lanes, the two sums serially in a lane each.
__device__ __noinline__ void majorant_body(const SedArgs& a, const double* trace_geom, const double* trace_wave,
                                           double* sed_A, double* sed_norm, double* sed_max, const double* grid_max,
                                           double* major, int* error_flag) {
    __shared__ double B[2][CLR_MAX_BINS];
    const int n = a.n, lane = threadIdx.x;
    const bool grid = a.TM == 3 && grid_max;
    double maxAeq = 0.0;
    for (int round = 0; round < (grid ? 2 : 1); ++round) {
        for (int i = lane; i < n; i += 32) {
            const double tg = trace_geom[i], tw = trace_wave[i];
            if (a.TM == 0) { B[0][i] = tg; B[1][i] = tw; continue; }
            double mx = sed_max[i];
            if (round == 1) {
                mx = grid_max[i];
                if (!(mx > 0.0)) mx = 1.0;
                sed_norm[i] = 1.0;
                sed_max[i] = mx;
            } else if (sed_A[i] > maxAeq) {
                maxAeq = sed_A[i];
            }
            B[0][i] = tg * mx;
            B[1][i] = tw * mx;
        }
        for (int o = 16; o > 0; o >>= 1) maxAeq = fmax(maxAeq, __shfl_xor_sync(0xffffffffu, maxAeq, o));
        __syncwarp();
        const double part = lane < 2 ? bin_sum(B[lane], n) : 0.0;
        const double mg = __shfl_sync(0xffffffffu, part, 0), mw = __shfl_sync(0xffffffffu, part, 1);
        if (lane == 0) {
            major[0] = mg; major[1] = mw; major[2] = mg + mw; major[3] = a.TM == 0 ? 0.0 : maxAeq;
            if (a.TM != 0 && round == 0 && (!(mg + mw >= 0.0) || !isfinite(mg + mw))) atomicCAS(error_flag, 0, 35);
        }
        __syncwarp();
    }
}

struct MajorantJob {
    SedArgs a;
    const double *trace_geom, *trace_wave, *grid_max;
    double *sed_A, *sed_norm, *sed_max, *major;
    int* error_flag;
};
__device__ __forceinline__ void majorant_job(const MajorantJob& j) {
    majorant_body(j.a, j.trace_geom, j.trace_wave, j.sed_A, j.sed_norm, j.sed_max, j.grid_max, j.major, j.error_flag);
}
__global__ void __launch_bounds__(32) sediment_majorant_kernel(MajorantJob j) { majorant_job(j); }
__global__ void __launch_bounds__(32) sediment_majorant_batch_kernel(const MajorantJob* __restrict__ jobs) {
    majorant_job(jobs[blockIdx.x]);
}

// Node tables of the (r, z) field for the counter-based stream: for channel ch (0 geometric, 1 wave) and
// node c, G = sum_i mu_ch[i] grid[i][c] (FP64, bin order) and a Walker/Vose alias table over the bins with
// probabilities mu_ch[i] grid[i][c] / G. One thread per (channel, node); reads of grid[i][c] coalesce over c.
// The host enables these tables only for grids with no negative value, where the reference's clamp of the
// interpolated value at zero never acts, so the interpolated sum equals the interpolation of the sums.
__global__ void sediment_node_kernel(const double* __restrict__ grid, const double* __restrict__ trace_geom,
                                     const double* __restrict__ trace_wave, int n, int plane, float2* node_mu,
                                     int2* node_alias, unsigned int* node_major_bits) {
    const int t = blockDim.x * blockIdx.x + threadIdx.x;
    if (t >= 2 * plane) return;
    const int ch = t / plane, c = t - ch * plane;
    const double* mu = ch ? trace_wave : trace_geom;
    double p[CLR_MAX_BINS];
    double G = 0.0;
    for (int i = 0; i < n; ++i) {
        p[i] = mu[i] * grid[(size_t)i * plane + c];
        G += p[i];
    }
    float* dst = reinterpret_cast<float*>(&node_mu[c]) + ch;
    *dst = (float)G;
    int2* A = node_alias + ((size_t)ch * plane + c) * n;
    if (!(G > 0.0)) {
        for (int i = 0; i < n; ++i) A[i] = make_int2(__float_as_int(1.0f), i);
    } else {
        unsigned char small[CLR_MAX_BINS], large[CLR_MAX_BINS];
        int ns = 0, nl = 0;
        for (int i = 0; i < n; ++i) {
            p[i] = p[i] * (double)n / G;
            if (p[i] < 1.0) small[ns++] = (unsigned char)i; else large[nl++] = (unsigned char)i;
        }
        while (ns > 0 && nl > 0) {
            const int sm = small[--ns], lg = large[--nl];
            A[sm] = make_int2(__float_as_int((float)p[sm]), lg);
            p[lg] = (p[lg] + p[sm]) - 1.0;
            if (p[lg] < 1.0) small[ns++] = (unsigned char)lg; else large[nl++] = (unsigned char)lg;
        }
        while (nl > 0) { const int i = large[--nl]; A[i] = make_int2(__float_as_int(1.0f), i); }
        while (ns > 0) { const int i = small[--ns]; A[i] = make_int2(__float_as_int(1.0f), i); }
    }
    if (ch == 0) {
        // majorant of the summed field: max over nodes of G_geom + G_wave (non-negative, so the
        // float bit patterns order like the values)
        double Gw = 0.0;
        for (int i = 0; i < n; ++i) Gw += trace_wave[i] * grid[(size_t)i * plane + c];
        const float tot = (float)(G + Gw) * (1.0f + 4.0f * 1.1920928955078125e-7f);
        atomicMax(node_major_bits, __float_as_uint(tot));
    }
}

// ---------------- meridional advection-diffusion field (sediment model 3 without a supplied grid) ----------------
// The reference solves, per size bin, the stationary axisymmetric advection-diffusion of the sediment in
// the secondary (meridional) circulation of the stirred cell on a cell-centred (r, z) grid: upwind finite
// volumes with no-flux walls, red-black SOR, per-bin mass renormalisation every 20 iterations and at every
// convergence check, stopping at the first check (after at least min(1000, max) iterations) where the
// largest relative residual over all bins is within tolerance (CLARITAS/CLARITAS.py:4040-4215, driven by
// :6451-6725, one launch per half-sweep). Here one cooperative launch does all of it: a cluster of CTAs
// per bin keeps its bin's plane in shared memory; the bins meet only at the checks (a bounded grid barrier) to agree on
// the largest residual. Every cell value, sum order and stopping iteration is the reference's.

// free-surface height and slope at radius r (:4046-4057)
__device__ void merid_surface(int FSM, double r, double ZMEAN, double R, double DH, double CORE, double* zs, double* hp) {
    double rr = fmin(fmax(r, 0.0), R), rr2 = rr * rr, R2 = R * R;
    *zs = ZMEAN; *hp = 0.0;
    if (!(DH > 0.0) || FSM == 0) return;
    if (FSM == 1) { *zs = ZMEAN + DH * (rr2 / R2 - 0.5); *hp = 2.0 * DH * rr / R2; return; }
    double a2 = CORE * CORE, Hinf = DH * (a2 + R2) / R2;
    double hbar = Hinf * (1.0 - (a2 / R2) * log1p(R2 / a2));
    *zs = ZMEAN - hbar + Hinf * rr2 / (a2 + rr2);
    *hp = 2.0 * Hinf * a2 * rr / ((a2 + rr2) * (a2 + rr2));
}
// secondary-circulation velocity from the streamfunction psi = -2U r^2 (1-r^2/R^2)^2 eta(1-eta) (:4059-4073);
// zs, hp: merid_surface at r
__device__ void merid_velocity(double r, double z, double zs, double hp, double ZMIN, double R, int FSM, double DH,
                               double CORE, double UPEAK, double* ur, double* uz) {
    *ur = 0.0; *uz = 0.0;
    if (!(UPEAK > 0.0) || !(R > 0.0) || !(DH > 0.0) || (FSM == 2 && !(CORE > 0.0))) return;
    double rr = fmin(fmax(r, 0.0), R), R2 = R * R, rr2 = rr * rr;
    double H = zs - ZMIN;
    if (!(H > 0.0)) return;
    double eta = (z - ZMIN) / H;
    if (eta < 0.0) eta = 0.0;
    if (eta > 1.0) eta = 1.0;
    double sq = rr2 / R2, f = eta * (1.0 - eta), fp = 1.0 - 2.0 * eta;
    double Apsi = 2.0 * UPEAK, om = 1.0 - sq;
    *ur = Apsi * rr * om * om * fp / H;
    *uz = -Apsi * (2.0 * om * (1.0 - 3.0 * sq) * f - rr * om * om * fp * eta * hp / H);
}
// radial slip interpolated from the per-bin table (:4075-4082)
__device__ double merid_slip(int p, double r, double R, const double* WR, int NRAD) {
    if (NRAD < 2 || !(R > 0.0)) return 0.0;
    double q = fmin(fmax(r / R, 0.0), 1.0) * (double)(NRAD - 1);
    int j = (int)floor(q);
    double t = q - (double)j;
    if (j >= NRAD - 1) { j = NRAD - 2; t = 1.0; }
    long long b = (long long)p * (long long)NRAD;
    return (1.0 - t) * WR[b + j] + t * WR[b + j + 1];
}
// a point inside the liquid (:4084-4089); zs: merid_surface at its radius
__device__ __forceinline__ int merid_fluid(double z, double zs, double ZMIN) { return z >= ZMIN && z < zs; }
// the finite-Re drift-diffusion field at a cell centre (sediment_local_scale with model 2, :1560-1593),
// which starts the iteration (:4100-4112)
__device__ double merid_initial(int FSM, int p, const double* SA, const double* SB, const double* SN, const double* RL,
                                int NRAD, float x, float z, float R, float ZMIN) {
    (void)FSM; (void)SA;
    double rr2 = (double)x * (double)x + 0.0 * 0.0;
    double R2 = (double)R * (double)R;
    if (rr2 > R2) rr2 = R2;
    double rr = sqrt(fmax(rr2, 0.0));
    double u = (R > 0.0) ? rr / (double)R * (double)(NRAD - 1) : 0.0;
    int j = (int)floor(u);
    if (j < 0) j = 0;
    if (j > NRAD - 2) j = NRAD - 2;
    double t = u - (double)j;
    long long base = (long long)p * (long long)NRAD;
    double radial_log = (1.0 - t) * RL[base + j] + t * RL[base + j + 1];
    if (radial_log > 0.0) radial_log = 0.0;
    double h = fmax((double)z - (double)ZMIN, 0.0);
    double logrel = radial_log - SB[p] * h;
    double ns = SN[p];
    if (!(ns > 0.0)) return 0.0;
    return exp(logrel) / ns;
}

__device__ __forceinline__ unsigned long long merid_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Barrier over the co-resident CTAs of a cooperative launch; gives up (error 91) after two seconds.
__device__ bool merid_grid_barrier(unsigned* count, unsigned* gen, unsigned nblocks, int* err) {
    __shared__ int ok_s;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok_s = 1;
        volatile unsigned* vgen = gen;
        const unsigned g = *vgen;
        __threadfence();
        if (atomicAdd(count, 1u) + 1u == nblocks) {
            *count = 0u;
            __threadfence();
            atomicAdd(gen, 1u);
        } else {
            const unsigned long long t0 = merid_ns();
            while (*vgen == g) {
                if (merid_ns() - t0 > 2000000000ull) { ok_s = 0; atomicCAS(err, 0, 91); break; }
            }
        }
        __threadfence();
    }
    __syncthreads();
    return ok_s != 0;
}

// A bin's rows are shared out over the CTAs of one thread-block cluster.
__device__ __forceinline__ void cluster_sync() { cooperative_groups::this_cluster().sync(); }
// the same shared-memory variable in the cluster's CTA `rank`
__device__ __forceinline__ double* in_cluster(double* local, unsigned rank) {
    return cooperative_groups::this_cluster().map_shared_rank(local, rank);
}

struct MeridArgs {
    int n, NR, NZ, NRAD, FSM, max_it, check_every, cluster, mass_in_smem, coef_in_smem;
    double R, ZMIN, ZMEAN, ZGRIDMAX, DH, CORE, UPEAK, Dt, OMEGA, TOL;
    const double *sedA, *sedB, *sed_norm, *radial_log, *wr, *ws;
    double* grid;       // [n][NR][NZ]
    double* coef;       // [n][kMeridPlanes][NR*NZ]: work planes, see below
    double* grid_max;   // [n] largest value over the liquid cells
    double* residual;   // [2][n] residual of every bin at the last two checks
    unsigned* bar;      // [2] barrier count and generation (zero before the launch)
    int* err;           // first error code
    int* iterations;    // [1] iterations done (the reference's solver_iterations)
    double* max_residual;  // [1]
};

constexpr int kMeridThreads = 512;
constexpr int kMeridMaxCluster = 8;
// work planes per bin: AE, AW, AN, AS, AP and 1/AP of the relaxed cells in list order, the lists (cells of one
// colour after the other, then the liquid cells in the reference's order; 2 x 32 bit per cell), the mass terms
constexpr int kMeridPlanes = 8;

// num / ap, correctly rounded, with rap = 1 / ap correctly rounded: one residual step on num * rap (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990). Three
// FP64 operations on the relaxation's bounding pipe against the eight or more of a division. No operand here is
// near the ends of the exponent range; an infinite or NaN num stays one.
__device__ __forceinline__ double merid_div(double num, double ap, double rap) {
    const double q = num * rap;
    return fma(fma(-ap, q, num), rap, q);
}

// The solver is bound by the FP64 pipe (one warp instruction per 16 cycles per SM), so: only liquid cells of one
// colour are listed, in full warps (a pass over the plane keeps half the lanes of every FP64 instruction idle);
// the division costs three operations; and a bin's rows are spread over a cluster of CTAs so that n bins use
// cluster x n SMs, neighbours' boundary rows written through distributed shared memory. 64 bins of 48x96 cells,
// 1250 iterations: 78 ms with one CTA per bin over the whole plane. Values, order of every sum and stopping
// iteration are unchanged.
__global__ void __launch_bounds__(kMeridThreads) meridional_solve_kernel(MeridArgs a) {
    extern __shared__ __align__(16) unsigned char msm[];
    const int NR = a.NR, NZ = a.NZ, plane = NR * NZ, tid = threadIdx.x, lane = tid & 31;
    const unsigned CS = (unsigned)a.cluster, rank = cooperative_groups::this_cluster().block_rank();
    const int p = blockIdx.x / a.cluster;
    const int i0 = (int)((long long)NR * rank / CS), i1 = (int)((long long)NR * (rank + 1) / CS);  // this CTA's rows
    // shared memory: the plane (every CTA holds all of it; its own rows and their two neighbours are current)
    // with a zero row and cell on either side, the free surface at cell centres and faces, the liquid mask and,
    // where it fits, the mass terms
    double* const G0 = reinterpret_cast<double*>(msm);
    const int pad = NZ + 1;
    double* const G = G0 + pad;
    double* const zsC = G0 + plane + 2 * pad;
    double* const hpC = zsC + NR;
    double* const zsF = hpC + NR;
    double* const hpF = zsF + NR + 1;
    double* const mass_sm = hpF + NR + 1;
    unsigned char* const act = reinterpret_cast<unsigned char*>(mass_sm + (a.mass_in_smem ? plane : 0));
    __shared__ double red[kMeridThreads / 32];
    __shared__ double from_rank[kMeridMaxCluster];  // rank 0: a value of every CTA
    __shared__ double scale_s, go_s;                // written by rank 0 into every CTA
    __shared__ int scan_s[3][kMeridThreads / 32];
    const double dr = a.R / (double)NR, dz = (a.ZGRIDMAX - a.ZMIN) / (double)NZ;
    double* const work = a.coef + (size_t)p * kMeridPlanes * plane;
    const int b0 = i0 * NZ, b1 = i1 * NZ;
    // the relaxed cells' coefficients and list: in shared memory where they fit (every cluster barrier would have
    // the next sweep fetch them from L2 again), else in this CTA's part of the work planes
    const size_t cells = (size_t)(b1 - b0), stride = a.coef_in_smem ? cells : (size_t)plane;
    double* const AE = a.coef_in_smem ? reinterpret_cast<double*>(act + ((plane + 15) & ~15)) : work + b0;
    double *const AW = AE + stride, *const AN = AW + stride, *const AS = AN + stride, *const AP = AS + stride,
           *const RAP = AP + stride;
    int* const lists = reinterpret_cast<int*>(work + 6 * (size_t)plane);
    int* const relax_list = a.coef_in_smem ? reinterpret_cast<int*>(RAP + stride) : lists + b0;
    int* const liquid_list = lists + plane + b0;
    double* const mass_terms = a.mass_in_smem ? mass_sm : work + 7 * (size_t)plane;
    // the free surface depends on the radius only
    for (int i = tid; i <= NR; i += kMeridThreads) {
        if (i < NR) merid_surface(a.FSM, ((double)i + 0.5) * dr, a.ZMEAN, a.R, a.DH, a.CORE, &zsC[i], &hpC[i]);
        merid_surface(a.FSM, (double)i * dr, a.ZMEAN, a.R, a.DH, a.CORE, &zsF[i], &hpF[i]);
    }
    for (int c = tid; c < pad; c += kMeridThreads) { G0[c] = 0.0; G[plane + c] = 0.0; }
    __syncthreads();
    // liquid cells (:4091-4098) and the starting field (:4100-4112)
    for (int c = tid; c < plane; c += kMeridThreads) {
        const int i = c / NZ, k = c - i * NZ;
        const double zc = a.ZMIN + ((double)k + 0.5) * dz;
        const int liquid = merid_fluid(zc, zsC[i], a.ZMIN);
        act[c] = (unsigned char)liquid;
        double g = 0.0;
        if (liquid && i >= i0 - 1 && i <= i1) {
            const float x = (float)(((double)i + 0.5) * dr), z = (float)zc;
            g = merid_initial(a.FSM, p, a.sedA, a.sedB, a.sed_norm, a.radial_log, a.NRAD, x, z, (float)a.R, (float)a.ZMIN);
        }
        G[c] = g;
    }
    __syncthreads();
    // upwind finite-volume coefficients of this CTA's rows (:4114-4159), compacted: the cells the sweeps relax
    // (liquid, with a positive diagonal), colour 0 then colour 1, and the liquid cells in plane order
    int n_relax[2] = {0, 0}, n_liquid = 0, liquid_before = 0;
    for (int c = tid; c < b0; c += kMeridThreads) liquid_before += act[c];
    for (int o = 16; o > 0; o >>= 1) liquid_before += __shfl_xor_sync(0xffffffffu, liquid_before, o);
    if (lane == 0) scan_s[0][tid >> 5] = liquid_before;
    __syncthreads();
    liquid_before = 0;
    for (int w = 0; w < kMeridThreads / 32; ++w) liquid_before += scan_s[0][w];
    for (int colour = 0; colour < 2; ++colour) {
        for (int base = b0; base < b1; base += kMeridThreads) {
            const int c = base + tid;
            bool relax = false, liquid = false;
            double ae = 0.0, aw = 0.0, an = 0.0, as = 0.0, ap = 0.0;
            if (c < b1) {
                const int i = c / NZ, k = c - i * NZ;
                liquid = act[c] != 0;
                if (liquid && ((i + k) & 1) == colour) {
                    double rc = ((double)i + 0.5) * dr, zc = a.ZMIN + ((double)k + 0.5) * dz;
                    double rw = (double)i * dr, re = (double)(i + 1) * dr;
                    double Az = 0.5 * (re * re - rw * rw), ur = 0.0, uz = 0.0, V = 0.0, F = 0.0, diff = 0.0;
                    if (i + 1 < NR && act[(i + 1) * NZ + k] && merid_fluid(zc, zsF[i + 1], a.ZMIN)) {
                        merid_velocity(re, zc, zsF[i + 1], hpF[i + 1], a.ZMIN, a.R, a.FSM, a.DH, a.CORE, a.UPEAK, &ur, &uz);
                        V = ur + merid_slip(p, re, a.R, a.wr, a.NRAD); F = V * re * dz; diff = a.Dt * re * dz / dr;
                        ae = diff + fmax(-F, 0.0); ap += diff + fmax(F, 0.0);
                    }
                    if (i > 0 && act[(i - 1) * NZ + k] && merid_fluid(zc, zsF[i], a.ZMIN)) {
                        merid_velocity(rw, zc, zsF[i], hpF[i], a.ZMIN, a.R, a.FSM, a.DH, a.CORE, a.UPEAK, &ur, &uz);
                        V = ur + merid_slip(p, rw, a.R, a.wr, a.NRAD); F = -V * rw * dz; diff = a.Dt * rw * dz / dr;
                        aw = diff + fmax(-F, 0.0); ap += diff + fmax(F, 0.0);
                    }
                    double zf = zc + 0.5 * dz;
                    if (k + 1 < NZ && act[i * NZ + k + 1] && merid_fluid(zf, zsC[i], a.ZMIN)) {
                        merid_velocity(rc, zf, zsC[i], hpC[i], a.ZMIN, a.R, a.FSM, a.DH, a.CORE, a.UPEAK, &ur, &uz);
                        V = uz - a.ws[p]; F = V * Az; diff = a.Dt * Az / dz;
                        an = diff + fmax(-F, 0.0); ap += diff + fmax(F, 0.0);
                    }
                    zf = zc - 0.5 * dz;
                    if (k > 0 && act[i * NZ + k - 1] && merid_fluid(zf, zsC[i], a.ZMIN)) {
                        merid_velocity(rc, zf, zsC[i], hpC[i], a.ZMIN, a.R, a.FSM, a.DH, a.CORE, a.UPEAK, &ur, &uz);
                        V = uz - a.ws[p]; F = -V * Az; diff = a.Dt * Az / dz;
                        as = diff + fmax(-F, 0.0); ap += diff + fmax(F, 0.0);
                    }
                    relax = ap > 0.0;
                }
            }
            const unsigned below = (1u << lane) - 1u;
            const unsigned mr = __ballot_sync(0xffffffffu, relax), ml = __ballot_sync(0xffffffffu, liquid);
            __syncthreads();
            if (lane == 0) { scan_s[1][tid >> 5] = __popc(mr); scan_s[2][tid >> 5] = __popc(ml); }
            __syncthreads();
            int at_r = __popc(mr & below), at_l = __popc(ml & below), tot_r = 0, tot_l = 0;
            for (int w = 0; w < kMeridThreads / 32; ++w) {
                if (w < (tid >> 5)) { at_r += scan_s[1][w]; at_l += scan_s[2][w]; }
                tot_r += scan_s[1][w]; tot_l += scan_s[2][w];
            }
            if (relax) {
                const int q = (colour ? n_relax[0] : 0) + n_relax[colour] + at_r;
                relax_list[q] = c;
                AE[q] = ae; AW[q] = aw; AN[q] = an; AS[q] = as; AP[q] = ap; RAP[q] = 1.0 / ap;
            }
            n_relax[colour] += tot_r;
            if (colour == 0) {
                if (liquid) liquid_list[n_liquid + at_l] = c;
                n_liquid += tot_l;
            }
        }
    }
    // this CTA's mass terms go to rank 0 (its shared memory, or the bin's global plane)
    double* const mass_out = a.mass_in_smem ? in_cluster(mass_sm, 0u) : mass_terms;
    cluster_sync();
    int mass_count = 0;
    for (int c = tid; c < plane; c += kMeridThreads) mass_count += act[c];
    for (int o = 16; o > 0; o >>= 1) mass_count += __shfl_xor_sync(0xffffffffu, mass_count, o);
    if (lane == 0) scan_s[0][tid >> 5] = mass_count;
    __syncthreads();
    mass_count = 0;
    for (int w = 0; w < kMeridThreads / 32; ++w) mass_count += scan_s[0][w];
    // per-bin mass renormalisation (:4176-4187): the terms in parallel, their sum in the reference's order
    auto normalize = [&]() {
        for (int j = tid; j < n_liquid; j += kMeridThreads) {
            const int c = liquid_list[j], i = c / NZ;
            double rw = (double)i * dr, re = (double)(i + 1) * dr, vol = 0.5 * (re * re - rw * rw) * dz;
            mass_out[liquid_before + j] = G[c] * vol;
        }
        cluster_sync();
        if (rank == 0 && tid < 32) {
            const double mass = warp_serial_sum(mass_terms, mass_count, nullptr);
            double target = 0.5 * a.R * a.R * (a.ZMEAN - a.ZMIN);
            const bool bad = !(mass > 0.0) || !(target > 0.0) || !isfinite(mass);
            if (bad && lane == 0) atomicCAS(a.err, 0, 41);
            if (lane < (int)CS) *in_cluster(&scale_s, (unsigned)lane) = bad ? 1.0 : target / mass;
        }
        cluster_sync();
        // own rows and the neighbours' boundary rows (solid cells are zero)
        const double sc = scale_s;
        const int lo = max(0, i0 - 1) * NZ, hi = min(NR, i1 + 1) * NZ;
        for (int c = lo + tid; c < hi; c += kMeridThreads) G[c] *= sc;
        cluster_sync();
    };
    double* const G_down = rank > 0 ? in_cluster(G, rank - 1) : nullptr;  // G in the CTAs of the rows below and above
    double* const G_up = rank + 1 < CS ? in_cluster(G, rank + 1) : nullptr;
    const double keep = 1.0 - a.OMEGA;
    // one colour of the red-black SOR sweep (:4161-4174)
    auto relax = [&](int colour) {
        const int q0 = colour ? n_relax[0] : 0, q1 = q0 + n_relax[colour];
        for (int q = q0 + tid; q < q1; q += kMeridThreads) {
            const int c = relax_list[q];
            double num = AE[q] * G[c + NZ];
            num += AW[q] * G[c - NZ];
            num += AN[q] * G[c + 1];
            num += AS[q] * G[c - 1];
            double nv = keep * G[c] + a.OMEGA * merid_div(num, AP[q], RAP[q]);
            // nv not finite, or nv < 1e-14: on the bits, which the FP64 pipe need not see
            const long long bits = __double_as_longlong(nv);
            if ((bits & 0x7ff0000000000000LL) == 0x7ff0000000000000LL || bits < __double_as_longlong(1e-14)) nv = 1e-14;
            G[c] = nv;
            if (c < b0 + NZ && G_down) G_down[c] = nv;
            if (c >= b1 - NZ && G_up) G_up[c] = nv;
        }
        cluster_sync();
    };
    // the largest of one value per CTA over the cluster, in every thread of rank 0
    auto cluster_max = [&](double m) -> double {
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0) red[tid >> 5] = m;
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < kMeridThreads / 32; ++w) m = fmax(m, red[w]);
            *in_cluster(&from_rank[rank], 0u) = m;
        }
        cluster_sync();
        double all = 0.0;
        if (rank == 0)
            for (unsigned q = 0; q < CS; ++q) all = fmax(all, from_rank[q]);
        return all;
    };
    // the decision of rank 0's first thread in every CTA of the cluster
    auto agree = [&](double v) -> double {
        if (rank == 0 && tid == 0)
            for (unsigned q = 0; q < CS; ++q) *in_cluster(&go_s, q) = v;
        cluster_sync();
        const double r = go_s;
        cluster_sync();
        return r;
    };
    // largest relative residual of the bin (:4189-4197)
    auto residual = [&]() -> double {
        double mr = 0.0;
        for (int q = tid; q < n_relax[0] + n_relax[1]; q += kMeridThreads) {
            const int c = relax_list[q];
            double num = AE[q] * G[c + NZ];
            num += AW[q] * G[c - NZ];
            num += AN[q] * G[c + 1];
            num += AS[q] * G[c - 1];
            const double ap = AP[q];
            double den = fmax(fabs(ap * G[c]), 1e-30), r = fabs(ap * G[c] - num) / den;
            if (r > mr) mr = r;
        }
        return cluster_max(mr);
    };
    normalize();
    const int min_it = a.max_it < 1000 ? a.max_it : 1000;
    int done = 0, last_checked = 0, checks = 0;
    double worst = 0.0;
    // the bins meet through rank 0 of each cluster; every CTA of a cluster follows its decision
    // (0 go on, 1 stop before the first sweep, 2 converged, 3 give up)
    double verdict = 0.0;
    if (rank == 0) {
        // the initial normalisation is checked before the first sweep (:6561-6575)
        if (!merid_grid_barrier(a.bar, a.bar + 1, (unsigned)a.n, a.err) || *(volatile int*)a.err) verdict = 1.0;
    }
    verdict = agree(verdict);
    for (int it = 1; it <= a.max_it && verdict == 0.0; ++it) {
        relax(0);
        relax(1);
        if (it % 20 == 0) normalize();
        if (it % a.check_every == 0 || it == a.max_it) {
            normalize();
            const double r = residual();
            if (rank == 0) {
                double* slot = a.residual + (size_t)(checks & 1) * a.n;
                if (tid == 0) slot[p] = r;
                if (!merid_grid_barrier(a.bar, a.bar + 1, (unsigned)a.n, a.err)) {
                    verdict = 3.0;
                } else {
                    worst = 0.0;
                    for (int q = 0; q < a.n; ++q) worst = fmax(worst, ((volatile double*)slot)[q]);
                    last_checked = it;
                    ++checks;
                    if (*(volatile int*)a.err) verdict = 3.0;
                    else if (it >= min_it && worst <= a.TOL) { done = it; verdict = 2.0; }
                }
            }
            verdict = agree(verdict);
        }
    }
    if (done == 0) done = last_checked ? last_checked : a.max_it;
    if (p == 0 && rank == 0 && tid == 0) { *a.iterations = done; *a.max_residual = worst; }
    double mx = 0.0;
    for (int c = b0 + tid; c < b1; c += kMeridThreads)
        if (act[c] && G[c] > mx) mx = G[c];
    __syncthreads();
    // extend each column above the free surface with its highest liquid value (:4199-4205)
    for (int i = i0 + tid; i < i1; i += kMeridThreads) {
        int top = -1;
        for (int k = NZ - 1; k >= 0; --k)
            if (act[i * NZ + k]) { top = k; break; }
        if (top < 0) { for (int k = 0; k < NZ; ++k) G[i * NZ + k] = 1.0; continue; }
        const double q = G[i * NZ + top];
        for (int k = top + 1; k < NZ; ++k) G[i * NZ + k] = q;
    }
    __syncthreads();
    for (int c = b0 + tid; c < b1; c += kMeridThreads) a.grid[(size_t)p * plane + c] = G[c];
    mx = cluster_max(mx);
    if (rank == 0 && tid == 0) a.grid_max[p] = mx;  // the majorant kernel takes 1 where this is not positive (:4207-4209)
    cluster_sync();  // no CTA leaves while another may still write to it
}

size_t meridional_coef_doubles(int n, int nr, int nz) { return (size_t)n * kMeridPlanes * nr * nz; }

cudaError_t enqueue_meridional_solve(ParticleBuffers& pb, const clr_scene_params& sp, const clr_sediment_spec& ss,
                                     cudaStream_t st) {
    MeridArgs a;
    a.n = pb.n; a.NR = pb.grid_nr; a.NZ = pb.grid_nz; a.NRAD = pb.n_radial; a.FSM = sp.free_surface_model;
    a.max_it = ss.solver_max_iterations; a.check_every = ss.solver_check_interval;
    a.R = ss.rin; a.ZMIN = ss.zmin; a.ZMEAN = ss.zmean; a.ZGRIDMAX = ss.grid_zmax; a.DH = ss.vortex_delta_h;
    a.CORE = ss.vortex_core_radius; a.UPEAK = ss.meridional_peak_speed; a.Dt = ss.eddy_diffusivity;
    a.OMEGA = ss.solver_sor; a.TOL = ss.solver_tolerance;
    a.sedA = pb.sedA; a.sedB = pb.sedB; a.sed_norm = pb.sed_norm; a.radial_log = pb.sed_radial_log; a.wr = pb.sed_wr;
    a.ws = pb.sed_ws; a.grid = pb.sed_grid; a.coef = pb.merid_coef; a.grid_max = pb.grid_max;
    a.residual = pb.merid_residual; a.bar = pb.merid_bar; a.err = pb.err; a.iterations = pb.merid_stats;
    a.max_residual = reinterpret_cast<double*>(pb.merid_residual + 2 * (size_t)pb.n);
    const size_t plane = (size_t)a.NR * a.NZ, limit = 226 * 1024;
    const size_t base = (plane + 2 * ((size_t)a.NZ + 1) + 4 * (size_t)a.NR + 2) * sizeof(double) + ((plane + 15) & ~(size_t)15);
    cudaError_t e = cudaFuncSetAttribute(meridional_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
    if (e != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(pb.merid_bar, 0, 2 * sizeof(unsigned), st)) != cudaSuccess) return e;
    // the largest cluster with every bin's cluster resident at once (the bins wait for one another at the checks)
    // and at least four rows per CTA
    for (a.cluster = kMeridMaxCluster;; a.cluster /= 2) {
        // beside the planes, as they fit: a CTA's coefficients (52 bytes per cell of its rows), rank 0's mass terms
        const size_t rows = ((size_t)a.NR + a.cluster - 1) / a.cluster, coef = rows * a.NZ * (6 * sizeof(double) + sizeof(int));
        size_t smem = base;
        a.coef_in_smem = smem + coef <= limit ? 1 : 0;
        if (a.coef_in_smem) smem += coef;
        a.mass_in_smem = smem + plane * sizeof(double) <= limit ? 1 : 0;
        if (a.mass_in_smem) smem += plane * sizeof(double);
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[2];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)a.cluster; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        at[1].id = cudaLaunchAttributeCooperative;
        at[1].val.cooperative = 1;
        cfg.gridDim = dim3((unsigned)(a.n * a.cluster)); cfg.blockDim = dim3(kMeridThreads);
        cfg.dynamicSmemBytes = smem; cfg.stream = st; cfg.attrs = at; cfg.numAttrs = 1;
        if (a.cluster > 1) {
            if (a.NR < 4 * a.cluster) continue;
            int fit = 0;
            if (cudaOccupancyMaxActiveClusters(&fit, meridional_solve_kernel, &cfg) != cudaSuccess || fit < a.n) {
                (void)cudaGetLastError();
                continue;
            }
        }
        cfg.numAttrs = 2;
        return cudaLaunchKernelEx(&cfg, meridional_solve_kernel, a);
    }
}

// Upper bound of the orders the Mie kernel needs for n bins: the largest nmx = max(nstop, |m x|) + 128 of
// the bins (:3506-3512), recomputed on the host from the same inputs with a few orders of slack for
// libm differences in cbrt and hypot, and never above CLR_MIE_MAX_ORDER (bins past that limit fail in
// the kernel with the reference's error code 1 before using shared memory).
int mie_order_bound(const double* d, const double* nr, const double* k, int n, double n_medium, double wavelength) {
    int cap = 1;
    for (int i = 0; i < n; ++i) {
        const double x = PD_PI * n_medium * d[i] / wavelength;
        if (!(x > 0.0) || !(n_medium > 0.0)) continue;
        const double mz = std::hypot(nr[i] / n_medium * x, k[i] / n_medium * x);
        const double nstop = x + 4.0 * std::cbrt(x) + 2.0;
        const double nmx = std::fmax(nstop, mz) + 128.0 + 8.0;
        cap = nmx >= (double)CLR_MIE_MAX_ORDER ? CLR_MIE_MAX_ORDER : std::max(cap, (int)nmx + 1);
    }
    return std::min(cap, (int)CLR_MIE_MAX_ORDER);
}

int particle_order_cap(const clr_particle_spec& ps) {
    return mie_order_bound(ps.diameter_m, ps.n_real, ps.k_imag, ps.n_bins, ps.n_medium, ps.wavelength_m);
}

static cudaError_t set_table_attributes() {
    cudaError_t e = cudaFuncSetAttribute(mie_coefficients_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kMieSmem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(phase_cdf_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(kCdfSmemAngles * sizeof(double)));
}

// Angles per row of a Legendre table (the fast tables mirror angles: half of them), and its orders for bins of a
// launch with this order bound (the bound holds the 128 extra orders of the downward recurrence).
static int legendre_pitch(int nt, bool fast) { return ((fast ? (nt + 1) / 2 : nt) + 31) & ~31; }
static int legendre_rows(int order_cap) {
    return order_cap >= CLR_MIE_MAX_ORDER ? CLR_MIE_MAX_ORDER : std::max(order_cap - 128, 1);
}
// No table above kLegendreMaxBytes (1801 angles and 1500 orders take 43 MB, which L2 holds; the table grows with the
// angles times the orders, which no other array does).
constexpr size_t kLegendreMaxBytes = (size_t)256 << 20;
size_t legendre_table_bytes(int nt, int order_cap, bool fast) {
    const size_t bytes = (size_t)legendre_rows(order_cap) * legendre_pitch(nt, fast) * sizeof(double2);
    return bytes <= kLegendreMaxBytes ? bytes : 0;
}
cudaError_t enqueue_legendre_table(double* theta, float* theta_f, int nt, int order_cap, bool fast, double2* table,
                                   cudaStream_t st) {
    const int pitch = legendre_pitch(nt, fast), rows = legendre_rows(order_cap);
    theta_grid_kernel<<<(nt + 127) / 128, 128, 0, st>>>(theta, theta_f, nt);
    if (fast) legendre_table_kernel<true><<<pitch / 32, 32, 0, st>>>(theta, (nt + 1) / 2, rows, pitch, table);
    else legendre_table_kernel<false><<<pitch / 32, 32, 0, st>>>(theta, nt, rows, pitch, table);
    return cudaGetLastError();
}

// Mie coefficients and efficiencies of n bins, then (hybrid event models) the theta grid and the phase
// pdf and CDF, else the two-point placeholder tables. `b.ab` holds n * order_cap a_n/b_n pairs and
// `b.pdf` n * nt values. The error word is not reset here.
cudaError_t enqueue_mie_tables(const double* d, const double* nr, const double* k, int n, double n_medium,
                               double wavelength, int nt, bool hybrid, int order_cap, const MiePhaseBuffers& b,
                               cudaStream_t st, bool fast_pdf) {
    cudaError_t e = set_table_attributes();
    if (e != cudaSuccess) return e;
    mie_coefficients_kernel<<<n, kMieThreads, mie_smem_bytes(order_cap), st>>>(
        d, nr, k, n_medium, wavelength, n, order_cap, b.ab, b.nstop, b.x, b.qext, b.qsca, b.qabs, b.qback, b.g,
        b.albedo, b.err);
    if (hybrid) {
        if (!b.table) theta_grid_kernel<<<(nt + 127) / 128, 128, 0, st>>>(b.theta, b.theta_f, nt);
        else if (b.table_ready && (e = cudaStreamWaitEvent(st, b.table_ready, 0)) != cudaSuccess) return e;
        const int pairs = (nt + 1) / 2, pitch = legendre_pitch(nt, fast_pdf);
        const bool many = !b.table && n >= kPdfManyBins;
        auto ordered = [&](auto kernel, int group, size_t pad) {
            kernel<<<dim3((nt + 31) / 32, (n + group - 1) / group), 32, pad, st>>>(b.theta, nt, n, order_cap, b.nstop, b.ab,
                                                                                   b.table, pitch, b.pdf);
        };
        auto fast = [&](auto kernel, int group, int threads, size_t pad) {
            kernel<<<dim3((pairs + threads - 1) / threads, (n + group - 1) / group), threads, pad, st>>>(
                b.theta, nt, n, order_cap, b.nstop, b.ab, b.table, pitch, b.pdf);
        };
        if (fast_pdf) {
            if (b.table) fast(phase_pdf_fast_kernel<1, 32, true>, 1, 32, kPdfPad);
            else if (many) fast(phase_pdf_fast_kernel<4, 128, false>, 4, 128, 0);
            else fast(phase_pdf_fast_kernel<1, 32, false>, 1, 32, kPdfPad);
        } else {
            if (b.table) ordered(phase_pdf_kernel<1, true>, 1, kPdfPad);
            else if (many) ordered(phase_pdf_kernel<4, false>, 4, 0);
            else ordered(phase_pdf_kernel<1, false>, 1, kPdfPad);
        }
        const size_t row = nt <= kCdfSmemAngles ? (size_t)nt * sizeof(double) : 0;
        phase_cdf_kernel<<<n, kCdfThreads, row, st>>>(b.theta, b.pdf, nt, n, b.cdf, b.cdf_f, b.err);
    } else {
        dummy_phase_kernel<<<(n + 127) / 128, 128, 0, st>>>(b.theta, b.theta_f, b.cdf, b.cdf_f, n);
    }
    if (b.guide) {
        const long long cells = (long long)n * (kPhaseGuide + 1);
        phase_guide_kernel<<<(unsigned)((cells + 255) / 256), 256, 0, st>>>(b.cdf_f, hybrid ? nt : 2, n, b.guide);
    }
    return cudaGetLastError();
}

// Mie efficiencies, asymmetry, theta grid and phase CDF of n bins into buffers the caller supplies
// (the first steps of enqueue_particle_precompute, with no buffer of its own). Used by the
// allocation-free entry point.
cudaError_t enqueue_mie_phase(const double* d, const double* nr, const double* k, int n, double n_medium,
                              double wavelength, int nt, const MiePhaseBuffers& b, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(b.err, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    return enqueue_mie_tables(d, nr, k, n, n_medium, wavelength, nt, true, CLR_MIE_MAX_ORDER, b, st);
}

static TransportJob transport_job_of(ParticleBuffers& pb, const clr_scene_params& sp, const clr_particle_spec& ps) {
    TransportJob j;
    j.n = pb.n; j.weight_mode = ps.weight_mode; j.em = sp.event_model;
    j.d = pb.d; j.w_in = pb.w; j.qext = pb.qext; j.qsca = pb.qsca; j.k_imag = pb.kidx; j.n_real = pb.nidx;
    j.concentration = ps.concentration_kg_m3; j.density = ps.density_kg_m3; j.wave_scale = ps.hybrid_wave_scale;
    j.n_medium = ps.n_medium; j.wavelength = ps.wavelength_m; j.wave_rms = ps.wave_rms_height_m;
    j.w = pb.w; j.radius = pb.radius; j.nden = pb.nden; j.mug = pb.mug; j.mus = pb.mus; j.mue = pb.mue;
    j.muw = pb.muw; j.muev = pb.muev; j.gcdf = pb.gcdf; j.wcdf = pb.wcdf; j.pcdf = pb.pcdf; j.muscal = pb.muscal;
    j.trace_geom = pb.trace_geom; j.trace_wave = pb.trace_wave; j.gcdf_f = pb.gcdf_f; j.wcdf_f = pb.wcdf_f;
    j.pn_f = pb.pn_f; j.pk_f = pb.pk_f; j.prad_f = pb.prad_f; j.error_flag = pb.err;
    return j;
}

static SedArgs sed_args_of(const ParticleBuffers& pb, const clr_scene_params& sp, const clr_sediment_spec& ss) {
    SedArgs a;
    a.n = pb.n; a.TM = sp.sediment_model; a.FSM = sp.free_surface_model; a.NQ = ss.n_quad; a.NRAD = ss.n_radial;
    a.rho_p = ss.particle_density; a.rho_w = ss.water_density; a.mu = ss.water_viscosity; a.grav = ss.gravity;
    // FP64 geometry as the reference passes it to its sediment kernels (the host fills it from the scene's
    // FP32 values when the caller leaves it zero)
    a.Dt = ss.eddy_diffusivity; a.R = ss.rin; a.ZMIN = ss.zmin; a.ZMEAN = ss.zmean;
    a.DH = ss.vortex_delta_h; a.CORE = ss.vortex_core_radius;
    (void)sp;
    return a;
}

static MajorantJob majorant_job_of(ParticleBuffers& pb, const SedArgs& a) {
    MajorantJob j;
    j.a = a; j.trace_geom = pb.trace_geom; j.trace_wave = pb.trace_wave; j.grid_max = a.TM == 3 ? pb.grid_max : nullptr;
    j.sed_A = pb.sedA; j.sed_norm = pb.sed_norm; j.sed_max = pb.sed_max; j.major = pb.sed_major; j.error_flag = pb.err;
    return j;
}

// Sediment bin coefficients (and the finite-Re slip table, the grid maxima) of one scenario.
static void enqueue_sediment_bins(ParticleBuffers& pb, const SedArgs& a, cudaStream_t st) {
    if (a.TM == 2 || a.TM == 3) {
        dim3 g((a.NRAD + 127) / 128, a.n);
        sediment_slip_kernel<<<g, 128, 0, st>>>(a, pb.d, pb.sed_wr);
    }
    sediment_bin_kernel<<<a.n, kSedThreads, 0, st>>>(a, pb.d, pb.sed_wr, pb.sedA, pb.sedB, pb.sed_norm, pb.sed_max,
                                            pb.sed_radial_log, pb.sed_terms, pb.sed_ws, pb.err);
    if (a.TM == 3 && !pb.merid_coef)  // a supplied grid: its largest value per bin (the solver gives its own)
        sediment_grid_max_kernel<<<a.n, 256, 0, st>>>(pb.sed_grid, (long long)pb.grid_nr * pb.grid_nz, pb.grid_max);
}

static cudaError_t enqueue_node_tables(ParticleBuffers& pb, cudaStream_t st) {
    if (!pb.node_tables) return cudaSuccess;
    const int plane = pb.grid_nr * pb.grid_nz;
    cudaError_t e = cudaMemsetAsync(pb.node_major, 0, sizeof(float), st);
    if (e != cudaSuccess) return e;
    sediment_node_kernel<<<(2 * plane + 127) / 128, 128, 0, st>>>(pb.sed_grid, pb.trace_geom, pb.trace_wave, pb.n,
                                                                  plane, pb.node_mu, pb.node_alias,
                                                                  reinterpret_cast<unsigned int*>(pb.node_major));
    return cudaSuccess;
}

// The scene-dependent rest of the precompute of one scenario, after its Mie tables: PSD normalisation
// and rates, sediment coefficients, majorants and node tables.
cudaError_t enqueue_scene_rates(ParticleBuffers& pb, const clr_scene_params& sp, const clr_particle_spec& ps,
                                const clr_sediment_spec& ss, cudaStream_t st) {
    transport_kernel<<<1, 32, 0, st>>>(transport_job_of(pb, sp, ps));
    const SedArgs a = sed_args_of(pb, sp, ss);
    enqueue_sediment_bins(pb, a, st);
    if (pb.merid_coef) {
        cudaError_t e = enqueue_meridional_solve(pb, sp, ss, st);
        if (e != cudaSuccess) return e;
    }
    sediment_majorant_kernel<<<1, 32, 0, st>>>(majorant_job_of(pb, a));
    cudaError_t e = enqueue_node_tables(pb, st);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

size_t scene_rates_batch_scratch(int n) { return (size_t)n * (sizeof(TransportJob) + sizeof(MajorantJob)) + 256; }

// The same for n scenarios: the rate and majorant kernels of all scenarios run as one launch each (a warp
// per scenario); the sediment bins and node tables stay per scenario. `d_scratch` holds
// scene_rates_batch_scratch(n) bytes of device memory for the job descriptions.
cudaError_t enqueue_scene_rates_batch(ParticleBuffers* const* pbs, const clr_scene_params* sps,
                                      const clr_particle_spec* pss, const clr_sediment_spec* sss, int n,
                                      void* d_scratch, cudaStream_t st) {
    std::vector<TransportJob> tj(n);
    std::vector<MajorantJob> mj(n);
    std::vector<SedArgs> sa(n);
    for (int i = 0; i < n; ++i) {
        tj[i] = transport_job_of(*pbs[i], sps[i], pss[i]);
        sa[i] = sed_args_of(*pbs[i], sps[i], sss[i]);
        mj[i] = majorant_job_of(*pbs[i], sa[i]);
    }
    TransportJob* d_tj = static_cast<TransportJob*>(d_scratch);
    MajorantJob* d_mj = reinterpret_cast<MajorantJob*>(
        (reinterpret_cast<uintptr_t>(d_tj + n) + 255) & ~(uintptr_t)255);
    // pageable sources: the copies are staged before the calls return
    cudaError_t e = cudaMemcpyAsync(d_tj, tj.data(), n * sizeof(TransportJob), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    e = cudaMemcpyAsync(d_mj, mj.data(), n * sizeof(MajorantJob), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    transport_batch_kernel<<<n, 32, 0, st>>>(d_tj);
    for (int i = 0; i < n; ++i) enqueue_sediment_bins(*pbs[i], sa[i], st);
    for (int i = 0; i < n; ++i)
        if (pbs[i]->merid_coef && (e = enqueue_meridional_solve(*pbs[i], sps[i], sss[i], st)) != cudaSuccess) return e;
    sediment_majorant_batch_kernel<<<n, 32, 0, st>>>(d_mj);
    for (int i = 0; i < n; ++i)
        if ((e = enqueue_node_tables(*pbs[i], st)) != cudaSuccess) return e;
    return cudaGetLastError();
}

cudaError_t enqueue_particle_precompute(ParticleBuffers& pb, const clr_scene_params& sp, const clr_particle_spec& ps,
                                        const clr_sediment_spec& ss, const SideStream& side, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(pb.err, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    MiePhaseBuffers b;
    b.ab = pb.ab;
    b.nstop = pb.nstop; b.x = pb.x; b.qext = pb.qext; b.qsca = pb.qsca; b.qabs = pb.qabs; b.qback = pb.qback;
    b.g = pb.g; b.albedo = pb.albedo; b.theta = pb.theta; b.theta_f = pb.theta_f; b.pdf = pb.pdf;
    b.cdf = pb.phase_cdf; b.cdf_f = pb.phase_cdf_f; b.guide = pb.phase_guide; b.err = pb.err;
    const int em = sp.event_model;
    const bool hybrid = em == 3 || em == 4 || em == 5, fast = ps.table_arithmetic == CLR_TABLES_FAST;
    const int cap = particle_order_cap(ps);
    if (hybrid && pb.legendre) {  // the angular functions beside the Mie coefficients, which leave most SMs free
        b.table = pb.legendre;
        b.table_ready = side.done;
        if ((e = cudaEventRecord(side.start, st)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(side.stream, side.start, 0)) != cudaSuccess) return e;
        if ((e = enqueue_legendre_table(pb.theta, pb.theta_f, pb.nt, cap, fast, pb.legendre, side.stream)) != cudaSuccess)
            return e;
        if ((e = cudaEventRecord(side.done, side.stream)) != cudaSuccess) return e;
    }
    e = enqueue_mie_tables(pb.d, pb.nidx, pb.kidx, pb.n, ps.n_medium, ps.wavelength_m, pb.nt, hybrid, cap, b, st, fast);
    if (e != cudaSuccess) return e;
    return enqueue_scene_rates(pb, sp, ps, ss, st);
}

}  // namespace clr
