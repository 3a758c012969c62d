// FP64 kernels of the potential-coefficient operator.
//
//  * near-field assembly: closed-form Wilton integral of 1/|p - r'| over each
//    source panel (integrals/panel.rs:147-208), CTAs over <= 64 rows of a target
//    leaf and a share of its sources, whose prepared panels lie in shared memory;
//  * near-field apply: dense leaf blocks times R right-hand sides on FP64
//    matrix instructions (FP32 on the CUDA cores);
//  * far field: Chebyshev P2M, M2M, M2L, L2L, L2P (fmm/bbfmm.rs:209-448).
#include <algorithm>

#include "dmma.cuh"
#include "gpx_common.h"
#include "kernels.cuh"
#include "wilton.cuh"

namespace gpx {

namespace {

constexpr int kAsmThreads = 256;
constexpr int kAsmTile = 64;

// One CTA per work item (target leaf, <= 64 rows) and every gridDim.y-th tile
// of 64 sources: rows of the leaf's P block m_t x S_t, row-major; a thread has
// one source of the tile and every fourth row.  The tile's panels are prepared
// once, in shared memory, and read from there for each row: with a panel in a
// thread's registers (128) two CTAs shared an SM, now three do.
// Bound: the FP64 pipe (about 1,900 multiply-add slots per entry: 4 edges of 2
// square roots, log1p, 2 arc tangents and their divisions), at about half its
// rate, since each entry is one chain of them.  147.8 M entries 12.9 -> 9.8 ms.
// Three CTAs leave 80 registers a thread, two fewer than the kernel would take:
// 28 bytes of spill stores and 36 of loads.  143.2 M entries take 9.5 ms so, and
// 10.8 with two CTAs and no spills.
__global__ void __launch_bounds__(kAsmThreads, 3) k_near_assemble(DevPlan p, double* __restrict__ P, double coef) {
    const int it = p.item_order[blockIdx.x], t = p.item_leaf[it], r0 = p.item_row0[it];
    const int64_t tb = p.leaf_begin[t];
    const int m = min((int)(p.leaf_begin[t + 1] - tb), r0 + 64);
    const int S = p.near_S[t];
    const int Sp = (S + 3) & ~3;
    const int64_t off = p.nval_off[t];
    __shared__ int64_t s_beg[28];
    __shared__ int32_t s_pre[29];
    __shared__ SrcPanel s_panel[kAsmTile];  // 43 doubles each: lanes on consecutive panels hit distinct banks
    if (threadIdx.x < 32) near_ranges_warp(p, t, threadIdx.x, s_beg, s_pre);
    __syncthreads();
    const int j = threadIdx.x % kAsmTile, row0 = r0 + threadIdx.x / kAsmTile;
    for (int base = kAsmTile * blockIdx.y; base < S; base += kAsmTile * gridDim.y) {
        const int cnt = min(kAsmTile, S - base);
        if (threadIdx.x < cnt) {
            int s = base + threadIdx.x, e = 0;
            while (s_pre[e + 1] <= s) ++e;
            prep_source(p.verts + 12 * (s_beg[e] + (s - s_pre[e])), s_panel[threadIdx.x]);
        }
        __syncthreads();
        if (j < cnt)
            for (int row = row0; row < m; row += kAsmThreads / kAsmTile) {
                const double* c = p.cent + 3 * (tb + row);
                P[off + (int64_t)row * Sp + base + j] = coef * wilton(s_panel[j], c[0], c[1], c[2]);
                asm volatile("" ::: "memory");  // the panel is read again per row, not kept in 86 registers
            }
        __syncthreads();
    }
}

__global__ void k_diag_inv(DevPlan p, const double* __restrict__ P, double* __restrict__ inv) {
    const int t = blockIdx.x;
    const int64_t tb = p.leaf_begin[t];
    const int m = (int)(p.leaf_begin[t + 1] - tb);
    const int Sp = (p.near_S[t] + 3) & ~3;
    for (int r = threadIdx.x; r < m; r += blockDim.x) {
        double d = P[p.nval_off[t] + (int64_t)r * Sp + r];  // self leaf is the first source block
        inv[tb + r] = fabs(d) > 1e-30 ? 1.0 / d : 1.0;
    }
}

// FP64 near apply: per work item (target leaf, <= 64 rows) and chunk of 8 NT
// right-hand sides, Y[rows][.] = P_t[rows][0:S] X[src(0:S)][.] on FP64 matrix
// instructions.  KC source panels per stage go through a cp.async ring of three
// stages (two where four CTAs of 64 columns share an SM): the item's P rows
// (contiguous along the contraction) and the gathered X rows (contiguous along
// the right-hand sides).  Four warps: WN = NT / NTW of
// them side by side over the columns, WM over the 8-row tiles (tile i belongs
// to warp i % WM), so narrow chunks do not leave warps without work.  Row tiles
// past the item's rows are skipped: a 12-row leaf costs 16 rows.  One warp runs
// the whole contraction of an output, in ascending order, and the instruction
// itself is the ascending chain of fused multiply-adds, so every result has
// the bits of a scalar loop: the mixed path's inner solves, whose TF32 far
// field truncates, turn any other rounding of the residual into another
// iterate.  Pitches of 4 more than a multiple of 8 doubles keep fragment reads free of
// bank conflicts.  P rows are padded to a multiple of 4 entries and R is a
// multiple of 4, so every 16-byte copy is aligned.
// Bound: the FP64 rate from R = 32 up (2 R flop per 8-byte entry), below it
// the stream of P and the gathers of X from L2.  At R = 64 the rest is the
// copies' instructions (with a division, a range search and 64-bit products in
// each they outnumbered the matrix instructions eight to one), padding to
// whole 8-row tiles (11 %) and the last wave.  Per apply, against 64 x 64 FMA
// tiles of 64 threads: 147.8 M entries, R = 64 0.76 ms (1.56 before, 1.01 with
// the index arithmetic in every copy; 0.51 at the FP64 rate), R = 24 0.34 ms,
// R = 8 0.24 (0.18 for the stream of P); 7.5 M entries in 12-row leaves, R =
// 24 74 us (297); 470 panels all pairs, R = 4 18 us (70).  The items run largest first: that
// alone took the 12-row leaves from 106 to 74 us.
template <int NT>
struct NearMma {
    static constexpr int NTW = NT % 3 == 0 ? 3 : NT == 1 ? 1 : 2;  // column tiles per warp
    static constexpr int WN = NT / NTW, WM = 4 / WN;
    static constexpr int KC = NT == 1 ? 32 : 16, S = NT == 8 ? 2 : 3;
    static constexpr int PP = KC + 4, XP = 8 * NT + 4;
    static constexpr int kMinCtas = NT == 8 ? 4 : 2;
};
template <int NT>
__global__ void __launch_bounds__(128, NearMma<NT>::kMinCtas) k_near_apply_mma(DevPlan p, const double* __restrict__ P,
                                                        const double* __restrict__ X, double* __restrict__ Y, int R,
                                                        int tile_rows) {
    using C = NearMma<NT>;
    constexpr int NTW = C::NTW, WM = C::WM, MT = 8 / WM, KC = C::KC, S = C::S, PP = C::PP, XP = C::XP;
    const int it = p.item_order[blockIdx.x], t = p.item_leaf[it], r0 = p.item_row0[it];
    const int rc = blockIdx.y * (8 * NT);
    const int64_t tb = p.leaf_begin[t] + r0;
    const int m = min((int)(p.leaf_begin[t + 1] - p.leaf_begin[t]) - r0, 64);
    const int cols = min(8 * NT, R - rc);
    const int nsrc = p.near_S[t], Sp = (nsrc + 3) & ~3;
    const double* Pi = P + p.nval_off[t] + (int64_t)r0 * Sp;
    __shared__ int64_t s_beg[28];
    __shared__ int32_t s_pre[29];
    extern __shared__ __align__(16) double near_smem[];
    double* Ps = near_smem;                       // [S][tile_rows][PP]
    double* Xs = Ps + S * tile_rows * PP;         // [S][KC][XP]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
    if (warp == 0) near_ranges_warp(p, t, lane, s_beg, s_pre);
    __syncthreads();
    const int nst = (Sp + KC - 1) / KC, mt = (m + 7) >> 3;
    // Copies of one stage: P rows prow, prow + RS, .. from column pk on; X rows
    // by panel number (rows only grow, so the near leaf they lie in is kept
    // with its first row's address).
    constexpr int TP = KC / 2, RS = 128 / TP;
    const int prow = tid / TP, pk = 2 * (tid % TP);
    const double* pp = Pi + (int64_t)prow * Sp + pk;
    const int64_t pstep = (int64_t)RS * Sp;
    const double* xe = X;
    int e = -1, xend = 0, ist = 0, islot = 0;
    auto issue = [&] {
        if (ist < nst) {
            const int k0 = ist * KC;
            double* ps = Ps + islot * tile_rows * PP + prow * PP + pk;
            double* xs = Xs + islot * KC * XP;
            const bool pok = k0 + pk < Sp;
#pragma unroll
            for (int i = 0; i < 64 / RS; ++i)
                if (prow + RS * i < m) cp_async_16(ps + RS * i * PP, pok ? pp + i * pstep : P, pok);
            pp += KC;
#pragma unroll
            for (int i = 0; i < (KC * NT + 31) / 32; ++i) {
                const int id = tid + 128 * i;
                if (KC * NT % 32 != 0 && id >= KC * 4 * NT) break;
                const int kk = id / (4 * NT), c = 2 * (id % (4 * NT)), k = k0 + kk;
                if (k < nsrc)
                    while (k >= xend) {
                        ++e;
                        xend = s_pre[e + 1];
                        xe = X + (s_beg[e] - s_pre[e]) * R + rc;
                    }
                const bool ok = k < nsrc && c < cols;
                cp_async_16(xs + kk * XP + c, ok ? xe + (int64_t)k * R + c : X, ok);
            }
            ++ist;
            islot = islot + 1 == S ? 0 : islot + 1;
        }
        cp_async_fence();
    };
    const int wn = warp % C::WN, wm = warp / C::WN;
    double acc[MT][NTW][2];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NTW; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll
    for (int st = 0; st < S - 1; ++st) issue();
    for (int st = 0, slot = 0; st < nst; ++st, slot = slot + 1 == S ? 0 : slot + 1) {
        cp_async_wait_for<S - 2>();
        __syncthreads();
        issue();
        const double* ps = Ps + slot * tile_rows * PP + (8 * wm + g) * PP + q;
        const double* xs = Xs + slot * KC * XP + q * XP + 8 * NTW * wn + g;
#pragma unroll
        for (int h = 0; h < KC; h += 16) {
            double b[4][NTW];
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int j = 0; j < NTW; ++j) b[k][j] = xs[(h + 4 * k) * XP + 8 * j];
#pragma unroll
            for (int i = 0; i < MT; ++i)
                if (wm + WM * i < mt) {
                    // rows m .. 8 mt - 1 of the last tile hold leftovers of
                    // other stages or items: their outputs are never stored
                    double a[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) a[k] = ps[8 * WM * i * PP + h + 4 * k];
#pragma unroll
                    for (int k = 0; k < 4; ++k)
#pragma unroll
                        for (int j = 0; j < NTW; ++j) dmma(acc[i][j], a[k], b[k][j]);
                }
        }
    }
    cp_async_wait_for<0>();
#pragma unroll
    for (int i = 0; i < MT; ++i) {
        const int row = 8 * (wm + WM * i) + g;
        if (row >= m) continue;
#pragma unroll
        for (int j = 0; j < NTW; ++j) {
            const int c = 8 * (NTW * wn + j) + 2 * q;
            if (c < cols)
                *reinterpret_cast<double2*>(Y + (tb + row) * R + rc + c) = make_double2(acc[i][j][0], acc[i][j][1]);
        }
    }
}

// FP32 near apply on the CUDA cores (the mixed path's mixed_near 1) as a
// register-tiled GEMM per work item (target leaf, <= 64 rows) and 64-wide
// chunk of right-hand sides: 64 threads, 8 x 8 outputs per thread (rows
// ty+8i, columns tx+8j: every shared-memory read is a broadcast or
// conflict-free), the contraction staged 32 source panels at a time with
// cp.async into a double buffer so the next tile's loads overlap this tile's
// FMAs.  Rows of P are padded to a multiple of 4 entries and R is a multiple
// of 4, so every 16-byte copy is aligned.
__global__ void __launch_bounds__(64) k_near_apply32(DevPlan p, const float* __restrict__ P,
                                                     const float* __restrict__ X, double* __restrict__ Y, int R) {
    constexpr int V = 4;        // elements per 16-byte copy
    constexpr int KC = 32;      // contraction chunk
    constexpr int PP = KC + V;  // Ps row pitch (16-byte multiple, conflict-free)
    constexpr int XP = 64 + V;  // Xs row pitch
    const int it = p.item_order[blockIdx.x], t = p.item_leaf[it], r0 = p.item_row0[it];
    const int rc = blockIdx.y * 64;
    const int64_t tb = p.leaf_begin[t] + r0;
    const int m = min((int)(p.leaf_begin[t + 1] - p.leaf_begin[t]) - r0, 64);
    const int S = p.near_S[t];
    const int Sp = (S + 3) & ~3;
    const float* Pi = P + p.nval_off[t] + (int64_t)r0 * Sp;
    __shared__ int64_t s_beg[28];
    __shared__ int32_t s_pre[29];
    __shared__ int64_t s_gid[2][KC];
    __shared__ __align__(16) float Ps[2][64][PP];  // [row][k]
    __shared__ __align__(16) float Xs[2][KC][XP];  // [k][col]
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
    if (tid < 32) near_ranges_warp(p, t, tid, s_beg, s_pre);
    __syncthreads();
    const int nchunk = (Sp + KC - 1) / KC;
    auto gather_ids = [&](int c) {
        if (tid < KC) {
            const int sidx = c * KC + tid;
            int64_t g = 0;
            if (sidx < S) {
                int e = 0;
                while (s_pre[e + 1] <= sidx) ++e;
                g = s_beg[e] + (sidx - s_pre[e]);
            }
            s_gid[c & 1][tid] = g;
        }
    };
    auto issue = [&](int c) {
        const int k0 = c * KC, buf = c & 1;
#pragma unroll
        for (int q = 0; q < KC / V; ++q) {  // P tile: 64 rows x KC
            const int id = tid + 64 * q, row = id / (KC / V), kc = (id % (KC / V)) * V;
            const bool ok = row < m && k0 + kc < Sp;
            cp_async_16(&Ps[buf][row][kc], ok ? Pi + (int64_t)row * Sp + k0 + kc : P, ok);
        }
#pragma unroll
        for (int q = 0; q < KC / V; ++q) {  // X tile: KC x 64 columns
            const int id = tid + 64 * q, kk = id / (64 / V), cc = (id % (64 / V)) * V;
            const bool ok = k0 + kk < S && rc + cc < R;
            cp_async_16(&Xs[buf][kk][cc], ok ? X + s_gid[buf][kk] * R + rc + cc : X, ok);
        }
        cp_async_fence();
    };
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
    gather_ids(0);
    __syncthreads();
    issue(0);
    for (int c = 0; c < nchunk; ++c) {
        if (c + 1 < nchunk) gather_ids(c + 1);
        __syncthreads();
        if (c + 1 < nchunk) {
            issue(c + 1);
            cp_async_wait_for<1>();
        } else {
            cp_async_wait_for<0>();
        }
        __syncthreads();
        const int buf = c & 1;
#pragma unroll 4
        for (int kk = 0; kk < KC; ++kk) {
            float a[8], b[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = Ps[buf][ty + 8 * i][kk];
#pragma unroll
            for (int j = 0; j < 8; ++j) b[j] = Xs[buf][kk][tx + 8 * j];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] += a[i] * b[j];
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int row = ty + 8 * i;
        if (row >= m) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int col = rc + tx + 8 * j;
            if (col < R) Y[(tb + row) * R + col] = (double)acc[i][j];
        }
    }
}

// 1-D Chebyshev interpolation weights S_n(x, x_m) (fmm/chebyshev.rs:41-74).
__device__ __forceinline__ void cheb_w(double x, int n, const double* roots, double* out) {
    double tx[8];
    tx[0] = 1.0;
    if (n > 1) tx[1] = x;
    for (int k = 2; k < n; ++k) tx[k] = 2.0 * x * tx[k - 1] - tx[k - 2];
    const double inv_n = 1.0 / n;
    for (int m = 0; m < n; ++m) {
        const double xm = roots[m];
        double sum = 0.5, prev = 1.0, cur = xm;
        for (int k = 1; k < n; ++k) {
            double tk;
            if (k == 1) {
                tk = xm;
            } else {
                tk = 2.0 * xm * cur - prev;
                prev = cur;
                cur = tk;
            }
            sum += tk * tx[k];
        }
        out[m] = 2.0 * inv_n * sum;
    }
}

// One thread per panel: W[j][m] for all n^3 nodes (node stride, padding zero).
__global__ void k_src_weights(DevPlan p, int quad, double* __restrict__ W) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= p.N) return;
    const int n = p.n, ns = p.ns;
    const double* ctr = p.leaf_ctr + 3 * p.leaf_of[j];
    const double ih = 1.0 / p.leaf_half;
    double* out = W + j * ns;
    for (int m = 0; m < ns; ++m) out[m] = 0.0;
    double w[3][8];
    if (quad == 0) {
        for (int d = 0; d < 3; ++d) cheb_w((p.cent[3 * j + d] - ctr[d]) * ih, n, p.roots, w[d]);
        for (int a = 0; a < n; ++a)
            for (int b = 0; b < n; ++b)
                for (int c = 0; c < n; ++c) out[(a * n + b) * n + c] = (w[0][a] * w[1][b]) * w[2][c];
        return;
    }
    // 2x2 Gauss rule on the bilinear map of the quad (a triangle is the quad
    // with a collapsed edge); weights normalised to sum to one.
    const double* v = p.verts + 12 * j;
    const double g = 0.57735026918962576451;
    double jw[4], pts[4][3], jsum = 0.0;
    for (int q = 0; q < 4; ++q) {
        const double u = (q & 1) ? g : -g, t = (q & 2) ? g : -g;
        const double N[4] = {0.25 * (1 - u) * (1 - t), 0.25 * (1 + u) * (1 - t), 0.25 * (1 + u) * (1 + t),
                             0.25 * (1 - u) * (1 + t)};
        const double dNu[4] = {-0.25 * (1 - t), 0.25 * (1 - t), 0.25 * (1 + t), -0.25 * (1 + t)};
        const double dNt[4] = {-0.25 * (1 - u), -0.25 * (1 + u), 0.25 * (1 + u), 0.25 * (1 - u)};
        double xu[3] = {0, 0, 0}, xt[3] = {0, 0, 0};
        for (int d = 0; d < 3; ++d) {
            pts[q][d] = 0.0;
            for (int k = 0; k < 4; ++k) {
                pts[q][d] += N[k] * v[3 * k + d];
                xu[d] += dNu[k] * v[3 * k + d];
                xt[d] += dNt[k] * v[3 * k + d];
            }
        }
        const double cx = xu[1] * xt[2] - xu[2] * xt[1], cy = xu[2] * xt[0] - xu[0] * xt[2],
                     cz = xu[0] * xt[1] - xu[1] * xt[0];
        jw[q] = sqrt(cx * cx + cy * cy + cz * cz);
        jsum += jw[q];
    }
    for (int q = 0; q < 4; ++q) {
        const double wq = jsum > 0.0 ? jw[q] / jsum : 0.25;
        for (int d = 0; d < 3; ++d) cheb_w((pts[q][d] - ctr[d]) * ih, n, p.roots, w[d]);
        for (int a = 0; a < n; ++a)
            for (int b = 0; b < n; ++b) {
                const double wab = wq * w[0][a] * w[1][b];
                for (int c = 0; c < n; ++c) out[(a * n + b) * n + c] += wab * w[2][c];
            }
    }
}

__global__ void k_potential_matrix(const double* __restrict__ sv, int64_t ns, const double* __restrict__ pts,
                                   int64_t nt, double* __restrict__ out, double coef) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t t0 = (int64_t)blockIdx.y * 64;
    if (s >= ns) return;
    SrcPanel sp;
    prep_source(sv + 12 * s, sp);
    for (int64_t t = t0; t < min(nt, t0 + 64); ++t)
        out[t * ns + s] = coef * wilton(sp, pts[3 * t], pts[3 * t + 1], pts[3 * t + 2]);
}

}  // namespace

void launch_near_assemble(Ctx& c, const DevPlan& p, int64_t nnz, double* P, double coef) {
    if (p.nleaf == 0) return;
    KTimer t(c, K_NEAR_ASSEMBLE, 8.0 * nnz, (double)nnz);
    k_near_assemble<<<dim3(p.nitems, assembly_split(p.nitems)), kAsmThreads, 0, c.stream>>>(p, P, coef);
    GPX_LAUNCH_CHECK();
    c.launches += 1;
}

void launch_diag_inv(Ctx& c, const DevPlan& p, const double* P, double* inv) {
    if (p.nleaf == 0) return;
    KTimer t(c, K_SMALL, 16.0 * p.N, 0.0);
    k_diag_inv<<<p.nleaf, 128, 0, c.stream>>>(p, P, inv);
    GPX_LAUNCH_CHECK();
    c.launches += 1;
}

template <int NT>
static void near_mma(Ctx& c, const DevPlan& p, const double* P, const double* X, double* Y, int R) {
    using C = NearMma<NT>;
    const int tile_rows = std::min(64, (p.max_leaf + 7) & ~7);
    const int smem = (int)sizeof(double) * C::S * (tile_rows * C::PP + C::KC * C::XP);
    set_smem_once(k_near_apply_mma<NT>, smem);
    k_near_apply_mma<NT><<<dim3(p.nitems, (R + 8 * NT - 1) / (8 * NT)), 128, smem, c.stream>>>(p, P, X, Y, R, tile_rows);
    GPX_LAUNCH_CHECK();
}

void launch_near_apply(Ctx& c, const DevPlan& p, int64_t nnz, const double* P, const double* X, double* Y, int R) {
    if (p.nleaf == 0) return;
    KTimer t(c, K_NEAR_APPLY64, 8.0 * nnz + 16.0 * (double)p.N * R, 2.0 * (double)nnz * R);
    switch (rhs_chunk(R, 64) / 8) {  // tiles of 5 and 7 would leave warps without columns
        case 1: near_mma<1>(c, p, P, X, Y, R); break;
        case 2: near_mma<2>(c, p, P, X, Y, R); break;
        case 3: near_mma<3>(c, p, P, X, Y, R); break;
        case 4: near_mma<4>(c, p, P, X, Y, R); break;
        case 5:
        case 6: near_mma<6>(c, p, P, X, Y, R); break;
        default: near_mma<8>(c, p, P, X, Y, R); break;
    }
    c.launches += 1;
}

void launch_near_apply32(Ctx& c, const DevPlan& p, int64_t nnz, const float* P, const float* X, double* Y, int R) {
    if (p.nleaf == 0) return;
    KTimer t(c, K_NEAR_APPLY, 4.0 * nnz + 12.0 * (double)p.N * R, 2.0 * (double)nnz * R);
    k_near_apply32<<<dim3(p.nitems, (R + 63) / 64), 64, 0, c.stream>>>(p, P, X, Y, R);
    GPX_LAUNCH_CHECK();
    c.launches += 1;
}

__global__ void k_to_f32(const double* __restrict__ a, float* __restrict__ b, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        b[i] = (float)a[i];
}

void launch_to_f32(Ctx& c, const double* a, float* b, int64_t n) {
    if (n == 0) return;
    KTimer t(c, K_VEC, 12.0 * n, 0.0);
    k_to_f32<<<(unsigned)std::min<int64_t>((n + 255) / 256, 148 * 32), 256, 0, c.stream>>>(a, b, n);
    GPX_LAUNCH_CHECK();
    c.launches += 1;
}

void launch_src_weights(Ctx& c, const DevPlan& p, int quad, double* W) {
    if (p.N == 0) return;
    KTimer t(c, K_SMALL);
    k_src_weights<<<(unsigned)((p.N + 127) / 128), 128, 0, c.stream>>>(p, quad, W);
    GPX_LAUNCH_CHECK();
    c.launches += 1;
}

void launch_potential_matrix(Ctx& c, const double* sv, int64_t ns, const double* pts, int64_t nt, double* out,
                             double coef) {
    if (ns == 0 || nt == 0) return;
    KTimer t(c, K_NEAR_ASSEMBLE, 8.0 * ns * nt, (double)ns * nt);
    dim3 g((unsigned)((ns + 127) / 128), (unsigned)((nt + 63) / 64));
    k_potential_matrix<<<g, 128, 0, c.stream>>>(sv, ns, pts, nt, out, coef);
    GPX_LAUNCH_CHECK();
    c.launches += 1;
}

}  // namespace gpx
