// Maxwell matrix of a small panel problem whose panels already sit in device
// memory, computed without allocating memory: every intermediate lives in one
// file-scope device array of fixed size, g_small_scratch below.
//
// The algorithm is the reference's dense path (cap/solver.rs:100-134):
// assemble the potential-coefficient matrix P (Wilton closed form at panel
// centroids, cap/solver.rs:81-97), LU-factor it with partial pivoting, solve
// one unit-potential right-hand side per conductor (cap/solver.rs:55-63) and
// accumulate C[i][j] = sum over conductor i's panels of sigma * area
// (cap/solver.rs:64-71).  Here the right-hand sides are carried as extra
// columns of the factorised matrix, so the blocked LU leaves L^-1 P_perm B in
// them and only a back substitution with U remains.
//
// Limits: at most kMaxPanels panels and kMaxCond conductors.  Scratch layout
// (doubles, row stride kLd = kMaxPanels + kMaxCond):
//   [0, kMaxPanels * kLd)        augmented system [P | B], factorised in place
//   cen  3 per panel, area 1 per panel
//   piv, act  kMaxPanels uint16 each: pivot rows in elimination order, and the
//        rows not yet pivoted
//   status int32 word: bit 0 zero pivot, bit 1 conductor index out of range
// Only the status word has to start at zero; the call clears it itself before
// its first launch.  Every other element the call reads it has written earlier
// in the same call.
#include <cstdint>
#include <mutex>
#include <string>

#include "dmma.cuh"
#include "gpx_common.h"
#include "wilton.cuh"

namespace gpx {

namespace {

constexpr int kMaxPanels = 512;
constexpr int kMaxCond = 64;
constexpr int kLd = kMaxPanels + kMaxCond;
constexpr int kNb = 32;  // LU column-block width
constexpr int kMaxDevices = 64;
constexpr size_t kOffCen = (size_t)kMaxPanels * kLd;
constexpr size_t kOffArea = kOffCen + 3 * kMaxPanels;
constexpr size_t kOffPiv = kOffArea + kMaxPanels;
constexpr size_t kOffStatus = kOffPiv + kMaxPanels / 2;
constexpr size_t kScratchDoubles = kOffStatus + 32;  // 297,248 doubles = 2,377,984 bytes
constexpr int kStatusSingular = 1, kStatusBadConductor = 2;

static __device__ __align__(256) double g_small_scratch[kScratchDoubles];

__device__ __forceinline__ int* status_of(double* S) { return reinterpret_cast<int*>(S + kOffStatus); }

// Centroid and area (area-weighted triangle fan, integrals/panel.rs:29-67) of
// each panel, and row i of the right-hand sides: B[i][j] = 1 if panel i lies
// on conductor j.
__global__ void k_small_setup(double* __restrict__ S, const double* __restrict__ verts,
                              const int32_t* __restrict__ cond, int n, int ncond) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double q[4][3];
    for (int k = 0; k < 4; ++k)
        for (int d = 0; d < 3; ++d) q[k][d] = verts[12 * (int64_t)i + 3 * k + d];
    const int nv = (q[3][0] == q[2][0] && q[3][1] == q[2][1] && q[3][2] == q[2][2]) ? 3 : 4;
    double asum = 0.0, acc[3] = {0.0, 0.0, 0.0};
    for (int k = 1; k < nv - 1; ++k) {
        const double a[3] = {q[k][0] - q[0][0], q[k][1] - q[0][1], q[k][2] - q[0][2]};
        const double b[3] = {q[k + 1][0] - q[0][0], q[k + 1][1] - q[0][1], q[k + 1][2] - q[0][2]};
        const double c[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]};
        const double t = sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]) * 0.5;
        for (int d = 0; d < 3; ++d) acc[d] += (q[0][d] + q[k][d] + q[k + 1][d]) * (1.0 / 3.0) * t;
        asum += t;
    }
    for (int d = 0; d < 3; ++d) S[kOffCen + 3 * i + d] = asum == 0.0 ? q[0][d] : acc[d] * (1.0 / asum);
    S[kOffArea + i] = asum;
    const int ci = cond[i];
    if (ci < 0 || ci >= ncond) atomicOr(status_of(S), kStatusBadConductor);
    double* row = S + (size_t)i * kLd + kMaxPanels;
    for (int j = 0; j < ncond; ++j) row[j] = j == ci ? 1.0 : 0.0;
}

// P[t][s] = coef * Wilton integral of source panel s at the centroid of t.
// Thread per source panel, kAsmTargets targets per CTA row: 32 left 330 panels
// on 33 CTAs, each thread with 32 integrals in a row.
constexpr int kAsmTargets = 4;
__global__ void __launch_bounds__(128) k_small_assemble(double* __restrict__ S, const double* __restrict__ verts,
                                                        int n, double coef) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const int t0 = blockIdx.y * kAsmTargets;
    if (s >= n) return;
    SrcPanel sp;
    prep_source(verts + 12 * (int64_t)s, sp);
    const double* cen = S + kOffCen;
    const int t1 = min(n, t0 + kAsmTargets);
    for (int t = t0; t < t1; ++t) S[(size_t)t * kLd + s] = coef * wilton(sp, cen[3 * t], cen[3 * t + 1], cen[3 * t + 2]);
}

// Rows are never moved: the factorisation keeps the physical row of every
// pivot (piv, in elimination order) and the list of rows not yet pivoted (act).
__device__ __forceinline__ uint16_t* piv_of(double* S) { return reinterpret_cast<uint16_t*>(S + kOffPiv); }
__device__ __forceinline__ uint16_t* act_of(double* S) { return piv_of(S) + kMaxPanels; }

// Column q of the columns right of the panel: P columns [c0, c0 + nq1), then
// the right-hand-side columns.
__device__ __forceinline__ int right_col(int q, int c0, int nq1) {
    return q < nq1 ? c0 + q : kMaxPanels + (q - nq1);
}

// LU with partial pivoting of the column panel [k0, k0 + w) over the m rows
// not yet pivoted, one thread per row with the row's 32 values in registers,
// then U12 = L11^-1 A12 for the columns right of it, one thread per column.
// Bound: the serial chain of the columns.  A column takes one barrier: each
// warp finds its largest magnitude (warp max of the two halves of the double)
// and its row's owner puts the row and its reciprocal pivot in shared memory,
// then every thread picks the largest of the 16 (ties: the lowest thread, the
// earliest row) and eliminates its own row in registers, moving it one place
// down: the current column is always place 0, so the loop body is the same code
// for every column (unrolled over the columns it outgrew the instruction
// cache).  Rows stay in place, nothing is swapped.  61 us at 470 rows, 18 at 22;
// two rows a thread, a division in every thread ahead of the search, and U12 in
// a kernel of its own all measured slower.
constexpr int kPanelWarps = kMaxPanels / 32;
__global__ void __launch_bounds__(kMaxPanels) k_small_panel(double* __restrict__ S, int n, int ncond, int k0, int w) {
    __shared__ __align__(16) double cand[2][kPanelWarps][kNb + 2];  // the warps' best rows; [kNb]: 1 / pivot
    __shared__ uint2 best[2][kPanelWarps];                          // their magnitudes (high, low word)
    __shared__ int win_lane[2][kPanelWarps];
    __shared__ __align__(16) double Lt[kNb][kNb + 2];               // Lt[r][j] = L11[r + j][r], pivot order
    __shared__ int wcount[kPanelWarps];
    __shared__ uint16_t prow[kNb];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m = n - k0;
    uint16_t *piv = piv_of(S), *act = act_of(S);
    const int row = tid < m ? (k0 == 0 ? tid : (int)act[tid]) : 0;
    bool active = tid < m;
    double x[kNb];
    double* src = S + (size_t)row * kLd + k0;  // k0 a multiple of 32: 16-byte aligned
#pragma unroll
    for (int j = 0; j < kNb; j += 2) {
        double2 v = make_double2(0.0, 0.0);
        if (active && j < w) v = *reinterpret_cast<const double2*>(src + j);  // kLd columns: j + 1 is readable
        x[j] = v.x;
        x[j + 1] = j + 1 < w ? v.y : 0.0;
    }
    for (int c = 0; c < w; ++c) {
        const int buf = c & 1;
        // a NaN never wins over a number; inactive rows own nothing
        const double a = x[0] == x[0] ? fabs(x[0]) : 0.0;
        const unsigned hi = active ? (unsigned)__double2hiint(a) : 0u;
        const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
        const unsigned lo = active && hi == mh ? (unsigned)__double2loint(a) : 0u;
        const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
        const unsigned who = __ballot_sync(0xffffffffu, active && hi == mh && lo == ml);
        const int owner = who ? __ffs(who) - 1 : -1;
        if (lane == owner) {
#pragma unroll
            for (int j = 0; j < kNb; j += 2)
                *reinterpret_cast<double2*>(&cand[buf][warp][j]) = make_double2(x[j], x[j + 1]);
            cand[buf][warp][kNb] = x[0] != 0.0 ? 1.0 / x[0] : 0.0;
        }
        if (lane == 0) {
            best[buf][warp] = make_uint2(mh, ml);
            win_lane[buf][warp] = owner;
        }
        __syncthreads();
        const int wl = lane < kPanelWarps ? win_lane[buf][lane] : -1;
        const uint2 bk = lane < kPanelWarps ? best[buf][lane] : make_uint2(0u, 0u);
        const unsigned h2 = wl >= 0 ? bk.x : 0u;
        const unsigned gh = __reduce_max_sync(0xffffffffu, h2);
        const unsigned l2 = wl >= 0 && h2 == gh ? bk.y : 0u;
        const unsigned gl = __reduce_max_sync(0xffffffffu, l2);
        const unsigned wwho = __ballot_sync(0xffffffffu, wl >= 0 && h2 == gh && l2 == gl);
        const int pw = __ffs(wwho) - 1;  // a row is left (c < w <= m)
        const int pl = __shfl_sync(0xffffffffu, wl, pw);
        const double* pr = cand[buf][pw];
        if (warp == pw && lane == pl) {
            active = false;
            prow[c] = (uint16_t)row;
            piv[k0 + c] = (uint16_t)row;
            if (!(a > 0.0)) atomicOr(status_of(S), kStatusSingular);
#pragma unroll
            for (int j = 0; j < kNb; ++j)
                if (c + j < w) src[c + j] = x[j];  // U's row
        }
        if (active) {
            const double l = x[0] * pr[kNb];
            src[c] = l;
            x[0] = x[1] - l * pr[1];
#pragma unroll
            for (int j = 2; j < kNb; j += 2) {
                const double2 p = *reinterpret_cast<const double2*>(pr + j);
                x[j - 1] = x[j] - l * p.x;
                x[j] = x[j + 1 < kNb ? j + 1 : j] - l * p.y;
            }
            x[kNb - 1] = 0.0;
        }
    }
    // the rows left, in the same order
    const unsigned left = __ballot_sync(0xffffffffu, active);
    if (lane == 0) wcount[warp] = __popc(left);
    __syncthreads();  // also: the panel's columns in S are written
    int base = 0;
    for (int k = 0; k < warp; ++k) base += wcount[k];
    if (active) act[base + __popc(left & ((1u << lane) - 1u))] = (uint16_t)row;
    for (int e = tid; e < kNb * kNb; e += kMaxPanels) {
        const int r = e / kNb, j = e % kNb;
        Lt[r][j] = j > 0 && r + j < w ? S[(size_t)prow[r + j] * kLd + k0 + r] : 0.0;
    }
    __syncthreads();
    // U12, in the pivots' own rows; the current row is always x[0]
    const int nq1 = n - k0 - w;
    for (int q = tid; q < nq1 + ncond; q += kMaxPanels) {
        double* col = S + right_col(q, k0 + w, nq1);
#pragma unroll
        for (int r = 0; r < kNb; ++r) x[r] = r < w ? col[(size_t)prow[r] * kLd] : 0.0;
        for (int r = 0; r < w; ++r) {
            const double y = x[0];
            col[(size_t)prow[r] * kLd] = y;
            const double* lt = Lt[r];
            x[0] = x[1] - lt[1] * y;
#pragma unroll
            for (int j = 2; j < kNb; j += 2) {
                const double2 p = *reinterpret_cast<const double2*>(lt + j);
                x[j - 1] = x[j] - p.x * y;
                x[j] = x[j + 1 < kNb ? j + 1 : j] - p.y * y;
            }
            x[kNb - 1] = 0.0;
        }
    }
}

// Trailing update A22 -= L21 U12 on 32 x 32 tiles (64 x 64 would leave most
// SMs without one): rows act[0, nr), columns right_col(q, k0 + w, nr) for
// q < nr + ncond, contraction over the w <= kNb pivots of the panel.
__global__ void __launch_bounds__(256) k_small_update(double* __restrict__ S, int k0, int w, int nr, int ncond) {
    __shared__ double As[kNb][33];  // [c][i]
    __shared__ double Bs[kNb][33];  // [c][q]
    const uint16_t *piv = piv_of(S), *act = act_of(S);
    const int nq = nr + ncond;
    const int i0 = blockIdx.y * 32, q0 = blockIdx.x * 32;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
#pragma unroll
    for (int e = tid; e < kNb * 32; e += 256) {
        const int ii = e / kNb, c = e % kNb;
        As[c][ii] = (i0 + ii < nr && c < w) ? S[(size_t)act[i0 + ii] * kLd + k0 + c] : 0.0;
    }
#pragma unroll
    for (int e = tid; e < kNb * 32; e += 256) {
        const int c = e / 32, qq = e % 32;
        Bs[c][qq] = (q0 + qq < nq && c < w) ? S[(size_t)piv[k0 + c] * kLd + right_col(q0 + qq, k0 + w, nr)] : 0.0;
    }
    double old[2][2];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const int ii = i0 + ty + 16 * u, qq = q0 + tx + 16 * v;
            old[u][v] = ii < nr && qq < nq ? S[(size_t)act[ii] * kLd + right_col(qq, k0 + w, nr)] : 0.0;
        }
    __syncthreads();
    double acc[2][2] = {};
#pragma unroll
    for (int c = 0; c < kNb; ++c) {
        const double a0 = As[c][ty], a1 = As[c][ty + 16], b0 = Bs[c][tx], b1 = Bs[c][tx + 16];
        acc[0][0] += a0 * b0;
        acc[0][1] += a0 * b1;
        acc[1][0] += a1 * b0;
        acc[1][1] += a1 * b1;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const int ii = i0 + ty + 16 * u, qq = q0 + tx + 16 * v;
            if (ii < nr && qq < nq) S[(size_t)act[ii] * kLd + right_col(qq, k0 + w, nr)] = old[u][v] - acc[u][v];
        }
}

// Inverts the diagonal blocks of U in place (upper triangular; the pivots'
// own rows), one warp per block, one lane per column.  A zero pivot (the call
// then fails with its status) inverts to zero.
__global__ void __launch_bounds__(32) k_small_invert(double* __restrict__ S, int n) {
    __shared__ double Us[kNb][kNb + 1];
    const int k0 = blockIdx.x * kNb, w = min(kNb, n - k0), lane = threadIdx.x;
    const uint16_t* piv = piv_of(S) + k0;
#pragma unroll
    for (int r = 0; r < kNb; ++r)
        Us[r][lane] = r < w && lane < w && lane >= r ? S[(size_t)piv[r] * kLd + k0 + lane] : 0.0;
    __syncwarp();
    const double d = Us[lane][lane], inv = d != 0.0 ? 1.0 / d : 0.0;
    double z[kNb];
#pragma unroll
    for (int r = kNb - 1; r >= 0; --r) {
        double t0 = r == lane ? 1.0 : 0.0, t1 = 0.0;
#pragma unroll
        for (int c = r + 1; c < kNb; ++c) {
            if (c & 1)
                t1 -= Us[r][c] * z[c];
            else
                t0 -= Us[r][c] * z[c];
        }
        z[r] = (t0 + t1) * __shfl_sync(0xffffffffu, inv, r);
    }
#pragma unroll
    for (int r = 0; r < kNb; ++r)
        if (r < w && lane < w && lane >= r) S[(size_t)piv[r] * kLd + k0 + lane] = z[r];
}

// Back substitution with U (its diagonal blocks inverted) and the charge sums
// (cap/solver.rs:64-71), one CTA per 8 right-hand-side columns.  The unknowns
// are 64 tiles of 8 rows x 8 columns in the accumulators of 16 warps.  Per
// block of 32 unknowns, from the last: its tiles go to shared memory, four
// warps multiply them by the inverse, and every warp subtracts U x from its
// rows above, all with FP64 matrix instructions; the coefficients were read
// before the barriers.  With a triangle solve per block, one lane per unknown,
// 470 panels took 128 us here, now 50.
//   out[i][j] = sum over panels k of conductor i of x_j[k] area[k], panels in
//   ascending order.
constexpr int kBackCols = 8;
constexpr int kBackTiles = kMaxPanels / 8 / 16;  // row tiles per warp
__global__ void __launch_bounds__(512) k_small_back(double* __restrict__ S, const int32_t* __restrict__ cond, int n,
                                                    int ncond, double* __restrict__ out) {
    __shared__ double Xs[kMaxPanels][kBackCols];      // the solution
    __shared__ double Bs[kNb][kBackCols + 4];         // the block's right-hand side
    const uint16_t* piv = piv_of(S);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
    const int j0 = blockIdx.x * kBackCols, nc = min(kBackCols, ncond - j0);
    const double* rowp[kBackTiles];
    double acc[kBackTiles][2];
#pragma unroll
    for (int i = 0; i < kBackTiles; ++i) {
        const int k = 8 * (warp + 16 * i) + g;
        rowp[i] = S + (size_t)(k < n ? piv[k] : 0) * kLd;
#pragma unroll
        for (int h = 0; h < 2; ++h) acc[i][h] = k < n && 2 * q + h < nc ? rowp[i][kMaxPanels + j0 + 2 * q + h] : 0.0;
    }
    for (int k0 = (n - 1) / kNb * kNb; k0 >= 0; k0 -= kNb) {
        const int w = min(kNb, n - k0), t0 = k0 / 8;
        // this warp's rows of the block's columns: U above it, its inverse inside
        double u[kBackTiles][kNb / 4];
#pragma unroll
        for (int i = 0; i < kBackTiles; ++i) {
            const int t = warp + 16 * i, k = 8 * t + g;
            if (t < t0 + kNb / 8)
#pragma unroll
                for (int s = 0; s < kNb / 4; ++s) {
                    const int c = 4 * s + q;
                    u[i][s] = c < w && k < n && k0 + c >= k ? rowp[i][k0 + c] : 0.0;
                }
            if (t >= t0 && t < t0 + kNb / 8)
#pragma unroll
                for (int h = 0; h < 2; ++h) Bs[8 * (t - t0) + g][2 * q + h] = acc[i][h];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kBackTiles; ++i) {
            const int t = warp + 16 * i;
            if (t >= t0 && t < t0 + kNb / 8) {
                double x[2] = {0.0, 0.0};
#pragma unroll
                for (int s = 0; s < kNb / 4; ++s) dmma(x, u[i][s], Bs[4 * s + q][g]);
#pragma unroll
                for (int h = 0; h < 2; ++h) Xs[8 * t + g][2 * q + h] = x[h];
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kBackTiles; ++i)
            if (warp + 16 * i < t0)
#pragma unroll
                for (int s = 0; s < kNb / 4; ++s) dmma(acc[i], -u[i][s], Xs[k0 + 4 * s + q][g]);
    }
    __syncthreads();
    const double* area = S + kOffArea;
    for (int e = tid; e < ncond * nc; e += 512) {
        const int i = e / nc, j = e % nc;
        double sum = 0.0;
#pragma unroll 8
        for (int k = 0; k < n; ++k)
            if (cond[k] == i) sum += Xs[k][j] * area[k];
        out[(size_t)i * ncond + j0 + j] = sum;
    }
}

std::mutex g_small_mu[kMaxDevices];
double* g_small_ptr[kMaxDevices] = {};

// Device address of this device's scratch array.  The first call on a device
// (made with that device current and its lock held) looks the address up and
// loads every kernel this entry point launches.  With CUDA's lazy module
// loading a kernel is otherwise loaded, and its device memory taken, on its
// first launch: a later call that reaches a kernel the earlier calls did not
// (k_small_update runs only above 32 panels) would then allocate.  Querying each kernel's
// attributes here loads them all up front.
double* small_scratch(int dev) {
    if (!g_small_ptr[dev]) {
        void* p = nullptr;
        GPX_CUDA(cudaGetSymbolAddress(&p, g_small_scratch));
        const void* kernels[] = {(const void*)k_small_setup,  (const void*)k_small_assemble, (const void*)k_small_panel,
                                 (const void*)k_small_update, (const void*)k_small_invert,   (const void*)k_small_back};
        for (const void* k : kernels) {
            cudaFuncAttributes fa{};
            GPX_CUDA(cudaFuncGetAttributes(&fa, k));
        }
        g_small_ptr[dev] = static_cast<double*>(p);
    }
    return g_small_ptr[dev];
}

// Rejects a pointer that is not device or managed memory usable on `dev`, or
// that is misaligned for its element type.
void check_device_ptr(const void* p, size_t align, int dev, const char* what) {
    cudaPointerAttributes a{};
    const cudaError_t e = cudaPointerGetAttributes(&a, p);
    if (e != cudaSuccess) {
        cudaGetLastError();
        throw Error(GPX_ERR_INVALID_ARG, std::string(what) + " is not a CUDA pointer");
    }
    const bool ok = (a.type == cudaMemoryTypeDevice && a.device == dev) || a.type == cudaMemoryTypeManaged;
    if (!ok)
        throw Error(GPX_ERR_INVALID_ARG,
                    std::string(what) + " must be device (or managed) memory of the context's device");
    if (reinterpret_cast<uintptr_t>(p) % align != 0)
        throw Error(GPX_ERR_INVALID_ARG, std::string(what) + " is misaligned");
}

inline unsigned cdiv(int a, int b) { return (unsigned)((a + b - 1) / b); }

void small_solve(Ctx& c, int64_t n_panels, const double* verts, const int32_t* cond, int ncond, double* out) {
    if (n_panels < 1 || n_panels > kMaxPanels)
        throw Error(GPX_ERR_INVALID_ARG, "n_panels = " + std::to_string(n_panels) +
                                             " is outside [1, 512], the static-scratch limit; use gpx_cap_solve");
    const int n = (int)n_panels;
    if (ncond < 1 || ncond > kMaxCond)
        throw Error(GPX_ERR_INVALID_ARG, "n_conductors = " + std::to_string(ncond) +
                                             " is outside [1, 64], the static-scratch limit; use gpx_cap_solve");
    if (!verts || !cond || !out) throw Error(GPX_ERR_INVALID_ARG, "null pointer");
    const int dev = c.device;
    if (dev < 0 || dev >= kMaxDevices) throw Error(GPX_ERR_INVALID_ARG, "device index above 63");
    GPX_CUDA(cudaSetDevice(dev));
    check_device_ptr(verts, alignof(double), dev, "d_verts");
    check_device_ptr(cond, alignof(int32_t), dev, "d_conductor");
    check_device_ptr(out, alignof(double), dev, "d_maxwell_out");
    std::lock_guard<std::mutex> lock(g_small_mu[dev]);
    double* S = small_scratch(dev);
    cudaStream_t s = c.stream;
    int* status = reinterpret_cast<int*>(S + kOffStatus);
    GPX_CUDA(cudaMemsetAsync(status, 0, sizeof(int), s));
    int64_t launches = 0;
    k_small_setup<<<cdiv(n, 128), 128, 0, s>>>(S, verts, cond, n, ncond);
    GPX_LAUNCH_CHECK();
    k_small_assemble<<<dim3(cdiv(n, 128), cdiv(n, kAsmTargets)), 128, 0, s>>>(S, verts, n, kCoulomb);
    GPX_LAUNCH_CHECK();
    launches += 2;
    for (int k0 = 0; k0 < n; k0 += kNb) {
        const int w = std::min(kNb, n - k0), nr = n - k0 - w;
        k_small_panel<<<1, kMaxPanels, 0, s>>>(S, n, ncond, k0, w);
        GPX_LAUNCH_CHECK();
        launches += 1;
        if (nr > 0) {
            k_small_update<<<dim3(cdiv(nr + ncond, 32), cdiv(nr, 32)), 256, 0, s>>>(S, k0, w, nr, ncond);
            GPX_LAUNCH_CHECK();
            launches += 1;
        }
    }
    k_small_invert<<<cdiv(n, kNb), 32, 0, s>>>(S, n);
    GPX_LAUNCH_CHECK();
    k_small_back<<<cdiv(ncond, kBackCols), 512, 0, s>>>(S, cond, n, ncond, out);
    GPX_LAUNCH_CHECK();
    launches += 2;
    int hstatus = 0;
    GPX_CUDA(cudaMemcpyAsync(&hstatus, status, sizeof(int), cudaMemcpyDeviceToHost, s));
    GPX_CUDA(cudaStreamSynchronize(s));
    c.launches += launches;
    if (hstatus & kStatusBadConductor)
        throw Error(GPX_ERR_INVALID_ARG, "a conductor index is outside [0, n_conductors)");
    if (hstatus & kStatusSingular) throw Error(GPX_ERR_CAPACITANCE, "singular potential matrix (zero LU pivot)");
}

}  // namespace

}  // namespace gpx

extern "C" gpx_status gpx_cap_solve_small_static(gpx_ctx* ctx, int64_t n_panels, const double* d_verts,
                                                 const int32_t* d_conductor, int32_t n_conductors,
                                                 double* d_maxwell_out) {
    if (!ctx) return GPX_ERR_INVALID_ARG;
    ctx->impl.last_error.clear();
    try {
        gpx::small_solve(ctx->impl, n_panels, d_verts, d_conductor, n_conductors, d_maxwell_out);
        return GPX_OK;
    } catch (const gpx::Error& e) {
        ctx->impl.last_error = e.what();
        return e.status;
    } catch (const std::exception& e) {
        ctx->impl.last_error = e.what();
        return GPX_ERR_INTERNAL;
    } catch (...) {
        ctx->impl.last_error = "unknown error";
        return GPX_ERR_INTERNAL;
    }
}
