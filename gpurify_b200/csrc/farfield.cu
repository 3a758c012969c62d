// Chebyshev far field (fmm/bbfmm.rs:209-448) for R right-hand sides, in FP64
// (plain path) or FP32 (mixed path), for expansion orders 2 to 6.
// Expansions are stored per box as E[box][r][node] with a node stride ns =
// n^3 rounded up to a multiple of 32 (node index fastest, padding nodes zero):
// one right-hand side's expansion is one contiguous, 128-byte-aligned row,
// which is also the K-major operand row of the tensor-core M2L (m2l_tc.cu).
//
//  P2M  E[leaf][r][m]  = sum_j W_j[m] a_j X[j][r]          (W: source weights)
//  M2M  E[par][r][.]   = sum_children (Mx (x) My (x) Mz) E[child][r][.]
//  M2L  L[t][r][m]    += (1/half) sum_s sum_l K_off[m][l] E[s][r][l]
//  L2L  L[child][r][.] += (Mx (x) My (x) Mz)^T L[par][r][.]
//  L2P  Y[j][r]       += coef sum_m S(c_j)[m] L[leaf][r][m]  (collocation point)
//
// P2M and L2P are register-tiled GEMMs per work item of at most 64 panels of
// one leaf (so large leaves spread over several CTAs).  M2M and L2L run one
// CTA per parent box over all eight octants at once: the 1-D operator of an axis
// depends only on the child's bit along that axis, so the eight children's
// contractions share partial sums along a binary tree (z, then y, then x for
// M2M; the reverse for L2L): 14 n^4 multiply-adds per parent and right-hand
// side instead of 24 n^4.
#include "dmma.cuh"
#include "farfield.cuh"
#include "krylov.cuh"

namespace gpx {

namespace {

// Panels per near-field work item (the plan's kRowsPerItem).
constexpr int kItemPanels = 64;

template <int N>
struct Ord {
    static constexpr int n3 = N * N * N;
    static constexpr int ns = (n3 + 31) & ~31;
};

// FP64 P2M and L2P on FP64 matrix instructions, one CTA per (work item = leaf
// and <= 64 of its panels, chunk of 8 NT right-hand sides).  Both are bound by
// latency and L2 at the leaves' sizes (12 to 64 panels): each stages what its
// warps share once and has no stage loop.
//
// P2M: E[leaf][r][m] = sum_j W[j][m] (a_j X[j][r]).  One warp per 32 nodes;
// the item's X rows are staged (zero past the item), the W rows, which each
// warp reads in its own columns only, go from L2 straight to registers, four
// panels ahead.  The weights have the node stride (padding zero).
template <int N, int NT>
__global__ void __launch_bounds__(Ord<N>::ns) k_p2m_mma(DevPlan p, const int32_t* __restrict__ slot,
                                                        const double* __restrict__ X, const double* __restrict__ W,
                                                        bool mul_area, double* __restrict__ E, int R) {
    constexpr int NS = Ord<N>::ns, XP = 8 * NT + 4;
    const int it = blockIdx.x, t = p.item_leaf[it], r0 = p.item_row0[it];
    const int rc = blockIdx.y * (8 * NT), cols = min(8 * NT, R - rc);
    const int64_t j0 = p.leaf_begin[t] + r0;
    const int cnt = (int)min((int64_t)kItemPanels, p.leaf_begin[t + 1] - j0), cnt4 = (cnt + 3) & ~3;
    extern __shared__ __align__(16) unsigned char far_smem[];
    double* Xs = reinterpret_cast<double*>(far_smem);  // [kItemPanels][XP]
    double* as = Xs + kItemPanels * XP;                // [kItemPanels]
    for (int e = threadIdx.x; e < cnt4 * 4 * NT; e += NS) {
        const int k = e / (4 * NT), c = 2 * (e % (4 * NT));
        const bool ok = k < cnt && c < cols;
        cp_async_16(Xs + k * XP + c, ok ? X + (j0 + k) * R + rc + c : X, ok);
    }
    cp_async_fence();
    for (int k = threadIdx.x; k < cnt4; k += NS) as[k] = mul_area && k < cnt ? p.area[j0 + k] : 1.0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
    const double* w = W + j0 * NS + 32 * warp + g;
    double acc[NT][4][2];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    double nx[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) nx[j] = __ldg(w + (int64_t)min(q, cnt - 1) * NS + 8 * j);
    cp_async_wait_for<0>();
    __syncthreads();
    for (int k = 0; k < cnt4; k += 4) {
        double b[4];
        const double* wn = w + (int64_t)min(k + 4 + q, cnt - 1) * NS;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            b[j] = nx[j];
            nx[j] = __ldg(wn + 8 * j);
        }
        const double ar = as[k + q];
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const double a = ar * Xs[(k + q) * XP + 8 * i + g];
#pragma unroll
            for (int j = 0; j < 4; ++j) dmma(acc[i][j], a, b[j]);
        }
    }
    const int64_t box = slot[it] < 0 ? (int64_t)p.leaf_box0 + t : (int64_t)p.nbox + slot[it];
    double* out = E + (box * R + rc + g) * NS + 32 * warp + 2 * q;
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        if (8 * i + g >= cols) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            *reinterpret_cast<double2*>(out + (int64_t)(8 * i) * NS + 8 * j) =
                make_double2(acc[i][j][0], acc[i][j][1]);
    }
}

// L2P: Y[j][r] += coef sum_m S_j[m] L[leaf][r][m].  The leaf's local rows are
// staged; four warps share the item as tasks of 16 panels x 8 NTW columns.
// The separable weights S_j[m] = (wx[a] wy[b]) wz[c] are formed in registers
// from the panel's n^2 products and n values in shared memory; explicit
// weights (WT) come from L2 with the node stride, times a_j if mul_area.
template <int N, int NT, bool WT>
__global__ void __launch_bounds__(128) k_l2p_mma(DevPlan p, const double* __restrict__ L,
                                                 const double* __restrict__ Wt, bool mul_area, double* __restrict__ Y,
                                                 int R, double coef) {
    constexpr int N3 = Ord<N>::n3, NS = Ord<N>::ns, LP = NS + 4, NN = N * N;
    constexpr int NTW = NT % 2 == 0 ? 2 : NT == 1 ? 1 : 3, NG = NT / NTW;
    const int it = blockIdx.x, t = p.item_leaf[it], r0 = p.item_row0[it];
    const int rc = blockIdx.y * (8 * NT), cols = min(8 * NT, R - rc);
    const int64_t j0 = p.leaf_begin[t] + r0;
    const int cnt = (int)min((int64_t)kItemPanels, p.leaf_begin[t + 1] - j0);
    extern __shared__ __align__(16) unsigned char far_smem[];
    double* Ls = reinterpret_cast<double*>(far_smem);      // [8 NT][LP]
    double* wz = Ls + 8 * NT * LP;                         // [kItemPanels][N]
    double* wxy = wz + kItemPanels * N;                    // [kItemPanels][NN]
    uint16_t* tab = reinterpret_cast<uint16_t*>(wxy + kItemPanels * NN);  // per node: xy pair << 4 | z
    const double* src = L + ((int64_t)(p.leaf_box0 + t) * R + rc) * NS;
    for (int e = threadIdx.x; e < 8 * NT * (NS / 2); e += 128) {
        const int r = e / (NS / 2), m = 2 * (e % (NS / 2));
        cp_async_16(Ls + r * LP + m, r < cols ? src + (int64_t)r * NS + m : L, r < cols);
    }
    cp_async_fence();
    if constexpr (!WT) {
        const double* w = p.w1d + j0 * 3 * N;
        for (int e = threadIdx.x; e < kItemPanels * NN; e += 128) {
            const int j = e / NN, ab = e % NN;
            wxy[e] = j < cnt ? w[j * 3 * N + ab / N] * w[j * 3 * N + N + ab % N] : 0.0;
        }
        for (int e = threadIdx.x; e < kItemPanels * N; e += 128) {
            const int j = e / N;
            wz[e] = j < cnt ? w[j * 3 * N + 2 * N + e % N] : 0.0;
        }
        // padding nodes: any weight does, their local expansion is zero
        for (int m = threadIdx.x; m < NS; m += 128) tab[m] = m < N3 ? (uint16_t)((m / N) << 4 | (m % N)) : 0;
    }
    cp_async_wait_for<0>();
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
    const int ntask = ((cnt + 15) >> 4) * NG;
    for (int task = warp; task < ntask; task += 4) {
        const int p0 = (task / NG) * 16, c0 = (task % NG) * 8 * NTW;
        double acc[2][NTW][2];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < NTW; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
        const double* lb = Ls + (c0 + g) * LP + q;
        const double* wrow[2];
        double ar[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int j = min(p0 + 8 * i + g, cnt - 1);
            wrow[i] = WT ? Wt + (j0 + j) * NS + q : nullptr;
            ar[i] = WT && mul_area ? p.area[j0 + j] : 1.0;
        }
#pragma unroll 4
        for (int s = 0; s < (N3 + 7) / 8; ++s) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {  // nodes 8 s + 4 h .. + 3, ascending
                double a[2];
                if constexpr (WT) {
#pragma unroll
                    for (int i = 0; i < 2; ++i) a[i] = __ldg(wrow[i] + 8 * s + 4 * h) * ar[i];
                } else {
                    const int tn = tab[8 * s + 4 * h + q];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int j = p0 + 8 * i + g;
                        a[i] = wxy[j * NN + (tn >> 4)] * wz[j * N + (tn & 15)];
                    }
                }
#pragma unroll
                for (int j = 0; j < NTW; ++j) {
                    const double b = lb[8 * j * LP + 8 * s + 4 * h];
#pragma unroll
                    for (int i = 0; i < 2; ++i) dmma(acc[i][j], a[i], b);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int j = p0 + 8 * i + g;
            if (j >= cnt) continue;
#pragma unroll
            for (int n = 0; n < NTW; ++n) {
                const int c = c0 + 8 * n + 2 * q;
                if (c >= cols) continue;
                double2* y = reinterpret_cast<double2*>(Y + (j0 + j) * R + rc + c);
                double2 v = *y;
                v.x += coef * acc[i][n][0];
                v.y += coef * acc[i][n][1];
                *y = v;
            }
        }
    }
}

template <int N, int NT>
void run_p2m64(Ctx& c, const DevPlan& p, const int32_t* slot, const double* X, const FarWeights<double>& w, double* E,
               int R) {
    const int smem = (int)sizeof(double) * (kItemPanels * (8 * NT + 4) + kItemPanels);
    set_smem_once(k_p2m_mma<N, NT>, smem);
    k_p2m_mma<N, NT><<<dim3(p.nitems, (R + 8 * NT - 1) / (8 * NT)), Ord<N>::ns, smem, c.stream>>>(
        p, slot, X, w.src, w.src_area, E, R);
    GPX_LAUNCH_CHECK();
    c.launches += 1;
}

template <int N, int NT>
void run_l2p64(Ctx& c, const DevPlan& p, const double* L, const FarWeights<double>& w, double* Y, int R, double coef) {
    const int smem = (int)sizeof(double) * (8 * NT * (Ord<N>::ns + 4) + kItemPanels * (N + N * N)) + 2 * Ord<N>::ns;
    const dim3 grid(p.nitems, (R + 8 * NT - 1) / (8 * NT));
    if (w.tgt) {
        set_smem_once(k_l2p_mma<N, NT, true>, smem);
        k_l2p_mma<N, NT, true><<<grid, 128, smem, c.stream>>>(p, L, w.tgt, w.tgt_area, Y, R, coef);
    } else {
        set_smem_once(k_l2p_mma<N, NT, false>, smem);
        k_l2p_mma<N, NT, false><<<grid, 128, smem, c.stream>>>(p, L, nullptr, false, Y, R, coef);
    }
    GPX_LAUNCH_CHECK();
    c.launches += 1;
}

// Column chunks as in the M2L (m2l_fac.cu), widths of 5 and 7 tiles rounded up.
template <int N, class F>
void by_chunk(int R, F&& run) {
    switch (rhs_chunk(R, Ord<N>::ns > 128 ? 32 : 64) / 8) {
        case 1: run(std::integral_constant<int, 1>()); break;
        case 2: run(std::integral_constant<int, 2>()); break;
        case 3: run(std::integral_constant<int, 3>()); break;
        case 4: run(std::integral_constant<int, 4>()); break;
        case 5:
        case 6:
            if constexpr (Ord<N>::ns <= 128) run(std::integral_constant<int, 6>());
            break;
        default:
            if constexpr (Ord<N>::ns <= 128) run(std::integral_constant<int, 8>());
    }
}

// CTAs per SM the FP32 P2M and L2P are compiled for at orders <= 5: four
// (64 registers, no spills) instead of the two that 90 registers allowed, so
// more warps hide the latency of each staged slice's global loads.
template <int N>
constexpr int kMinCtas() {
    return N <= 5 ? 4 : 1;
}

// FP32 P2M as a GEMM per (work item = leaf and <= 64 of its panels, chunk of
// RW = 16, 32 or 64 rows r): E[leaf][r][m] = sum_j W[j][m] * (a_j X[j][r]).
// The work items are the near-field items (64 panels each), so a leaf of a few
// hundred panels spreads over several CTAs instead of serialising one: the
// first item of a leaf writes E[leaf], each further item writes a partial
// expansion at box index nbox + slot, and k_p2m_fix adds the partials in item
// order (deterministic).
// 256 threads; thread (tm, tr) holds nodes MI tm .. MI tm + MI - 1 and rows
// RT tr .. RT tr + RT - 1, RT = RW / 8.  Panels are staged 32 at a time.  Every
// row r < Rb and node m < ns of the chunk is written (zeros outside r < R, m < n3).
template <int N, int RW>
__global__ void __launch_bounds__(256, kMinCtas<N>())
    k_p2m32(DevPlan p, const int32_t* __restrict__ slot, const float* __restrict__ X, const float* __restrict__ W,
            bool mul_area, float* __restrict__ E, int R, int Rb) {
    constexpr int N3 = Ord<N>::n3, NS = Ord<N>::ns, MI = NS / 32, RT = RW / 8;
    constexpr int KP = 32;       // panels per staged chunk
    constexpr int QW = RW + 4;   // Qs row stride: 16-byte aligned rows
    const int it = blockIdx.x;
    const int t = p.item_leaf[it], r0 = p.item_row0[it];
    const int rc = blockIdx.y * RW;
    const int64_t lb = p.leaf_begin[t];
    const int64_t j0 = lb + r0, j1 = min(lb + r0 + kItemPanels, p.leaf_begin[t + 1]);
    __shared__ float Ws[KP][NS + 1];
    __shared__ __align__(16) float Qs[KP][QW];
    const int tid = threadIdx.x, tm = tid >> 3, tr = tid & 7;
    float acc[MI][RT];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < RT; ++j) acc[i][j] = 0.f;
    for (int64_t jb = j0; jb < j1; jb += KP) {
        const int cnt = (int)min((int64_t)KP, j1 - jb);
        __syncthreads();
        for (int e = tid; e < KP * NS; e += 256) {
            const int k = e / NS, m = e % NS;
            Ws[k][m] = k < cnt ? W[(jb + k) * NS + m] : 0.f;
        }
        for (int e = tid; e < KP * RW; e += 256) {
            const int k = e / RW, r = e % RW;
            Qs[k][r] = (k < cnt && rc + r < R) ? (mul_area ? (float)p.area[jb + k] : 1.f) * X[(jb + k) * R + rc + r]
                                               : 0.f;
        }
        __syncthreads();
        for (int k = 0; k < cnt; ++k) {
            float a[MI], b[RT];
#pragma unroll
            for (int i = 0; i < MI; ++i) a[i] = Ws[k][MI * tm + i];
#pragma unroll
            for (int j = 0; j < RT; j += 2) {
                const float2 v = *reinterpret_cast<const float2*>(&Qs[k][RT * tr + j]);
                b[j] = v.x, b[j + 1] = v.y;
            }
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < RT; ++j) acc[i][j] += a[i] * b[j];
        }
    }
    const int64_t box = slot[it] < 0 ? (int64_t)p.leaf_box0 + t : (int64_t)p.nbox + slot[it];
    float* out = E + (box * Rb + rc) * NS;
#pragma unroll
    for (int j = 0; j < RT; ++j) {
        const int r = RT * tr + j;
        if (rc + r >= Rb) continue;
#pragma unroll
        for (int i = 0; i < MI; ++i) {
            const int m = MI * tm + i;
            out[(int64_t)r * NS + m] = (m < N3 && rc + r < R) ? acc[i][j] : 0.f;
        }
    }
}

// E[leaf] += the partial expansions of its further work items, in item order.
// One CTA per (leaf with several items, 1024-value chunk of its Rb x ns block).
template <class T>
__global__ void __launch_bounds__(256) k_p2m_fix(int nbox, int leaf_box0, const int32_t* __restrict__ fix_leaf,
                                                 const int32_t* __restrict__ fix_first,
                                                 const int32_t* __restrict__ fix_cnt, T* __restrict__ E,
                                                 int64_t block) {
    const int f = blockIdx.x;
    const int64_t e = ((int64_t)blockIdx.y * 256 + threadIdx.x) * 4;
    if (e >= block) return;
    T* dst = E + ((int64_t)leaf_box0 + fix_leaf[f]) * block + e;
    T v0 = dst[0], v1 = dst[1], v2 = dst[2], v3 = dst[3];
    const int s0 = fix_first[f], cnt = fix_cnt[f];
    for (int q = 0; q < cnt; ++q) {
        const T* src = E + ((int64_t)nbox + s0 + q) * block + e;
        v0 += src[0], v1 += src[1], v2 += src[2], v3 += src[3];
    }
    dst[0] = v0, dst[1] = v1, dst[2] = v2, dst[3] = v3;
}

// FP32 L2P as a GEMM per (work item = leaf and <= 64 of its panels, chunk of
// RW = 16, 32 or 64 rows r): Y[j][r] += coef * sum_m S_j[m] L[leaf][r][m],
// S_j[m] = wx[a] wy[b] wz[c] (the centroid's separable weights), or S_j = Wt[j]
// (times a_j if mul_area) when explicit weights are given.
// 256 threads; thread (tj, tr) holds panels 4 tj .. 4 tj + 3 and rows
// RT tr .. RT tr + RT - 1, RT = RW / 16; nodes are staged 32 at a time.
template <int N, int RW>
__global__ void __launch_bounds__(256, kMinCtas<N>())
    k_l2p32(DevPlan p, const float* __restrict__ L, const float* __restrict__ Wt, bool mul_area,
            double* __restrict__ Y, int R, int Rb, double coef) {
    constexpr int N3 = Ord<N>::n3, NS = Ord<N>::ns, RT = RW / 16;
    constexpr int JP = kItemPanels, MK = 32, SW = 64 + 4, LW = RW + 4;
    const int it = blockIdx.x;
    const int t = p.item_leaf[it], r0 = p.item_row0[it];
    const int rc = blockIdx.y * RW;
    const int64_t lb = p.leaf_begin[t];
    const int64_t jb = lb + r0;
    const int cnt = (int)min((int64_t)JP, p.leaf_begin[t + 1] - jb);
    const float* src = L + ((int64_t)(p.leaf_box0 + t) * Rb + rc) * NS;
    __shared__ float wv[JP][3 * N];
    __shared__ __align__(16) float Ss[MK][SW];  // [node][panel]
    __shared__ __align__(16) float Ls[MK][LW];  // [node][row]
    const int tid = threadIdx.x, tj = tid >> 4, tr = tid & 15;
    if (!Wt)
        for (int e = tid; e < JP * 3 * N; e += 256) {
            const int jj = e / (3 * N);
            wv[jj][e % (3 * N)] = jj < cnt ? (float)p.w1d[jb * 3 * N + e] : 0.f;
        }
    float acc[4][RT];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < RT; ++q) acc[i][q] = 0.f;
    for (int m0 = 0; m0 < N3; m0 += MK) {
        __syncthreads();
        for (int e = tid; e < JP * MK; e += 256) {
            const int jj = e / MK, mm = e % MK, m = m0 + mm;
            float v = 0.f;
            if (m < N3 && jj < cnt) {
                v = Wt ? Wt[(jb + jj) * NS + m] : wv[jj][m / (N * N)] * wv[jj][N + (m / N) % N] * wv[jj][2 * N + m % N];
                if (mul_area) v *= (float)p.area[jb + jj];
            }
            Ss[mm][jj] = v;
        }
        for (int e = tid; e < RW * MK; e += 256) {
            const int mm = e % MK, r = e / MK;
            Ls[mm][r] = (m0 + mm < N3 && rc + r < R) ? src[(int64_t)r * NS + m0 + mm] : 0.f;
        }
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < MK; ++k) {
            const float4 av = *reinterpret_cast<const float4*>(&Ss[k][4 * tj]);
            const float a[4] = {av.x, av.y, av.z, av.w};
            float b[RT];
#pragma unroll
            for (int q = 0; q < RT; ++q) b[q] = Ls[k][RT * tr + q];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int q = 0; q < RT; ++q) acc[i][q] += a[i] * b[q];
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int jj = 4 * tj + i;
        if (jj >= cnt) continue;
        double* y = Y + (jb + jj) * R + rc + RT * tr;
        if (RT == 4 && rc + RT * tr + 3 < R) {  // R is a multiple of 4: 16-byte aligned pairs
            double2 y0 = *reinterpret_cast<double2*>(y), y1 = *reinterpret_cast<double2*>(y + 2);
            y0.x += coef * (double)acc[i][0], y0.y += coef * (double)acc[i][RT > 1 ? 1 : 0];
            y1.x += coef * (double)acc[i][RT > 2 ? 2 : 0], y1.y += coef * (double)acc[i][RT > 3 ? 3 : 0];
            *reinterpret_cast<double2*>(y) = y0;
            *reinterpret_cast<double2*>(y + 2) = y1;
        } else {
#pragma unroll
            for (int q = 0; q < RT; ++q)
                if (rc + RT * tr + q < R) y[q] += coef * (double)acc[i][q];
        }
    }
}

template <int N, int RW>
void run_p2m32(Ctx& c, const DevPlan& p, const int32_t* slot, const float* X, const FarWeights<float>& w, float* E,
               int R, int Rb) {
    k_p2m32<N, RW><<<dim3(p.nitems, (Rb + RW - 1) / RW), 256, 0, c.stream>>>(p, slot, X, w.src, w.src_area, E, R, Rb);
    GPX_LAUNCH_CHECK();
    c.launches += 1;
}

template <int N, int RW>
void run_l2p32(Ctx& c, const DevPlan& p, const float* L, const FarWeights<float>& w, double* Y, int R, int Rb,
               double coef) {
    k_l2p32<N, RW><<<dim3(p.nitems, (R + RW - 1) / RW), 256, 0, c.stream>>>(p, L, w.tgt, w.tgt_area, Y, R, Rb, coef);
    GPX_LAUNCH_CHECK();
    c.launches += 1;
}

// Column tile of the FP32 kernels for Rb = rhs_pad32(R) rows.
template <class F>
void by_rows32(int Rb, F&& run) {
    if (Rb == 16)
        run(std::integral_constant<int, 16>());
    else if (Rb == 32)
        run(std::integral_constant<int, 32>());
    else
        run(std::integral_constant<int, 64>());
}

// Rows of right-hand sides per M2M / L2L block.
template <class T, int N>
constexpr int tree_rc() {
    return (sizeof(T) == 8 && N >= 6) ? 4 : 8;
}
template <class T, int N>
constexpr size_t tree_smem() {
    return sizeof(T) * (size_t)(4 + 2) * tree_rc<T, N>() * Ord<N>::n3;
}

// 1-D operators of the three axes: m[axis][bit][m * n + k] (m parent node, k
// child node).  A kernel argument, so that every multiply-add takes its
// coefficient from the constant bank: held in registers (50 values at order 5)
// they left one FP64 CTA per SM, read from shared memory they cost a load each.
template <class T, int N>
struct TreeOps {
    T m[3][2][N * N];
};
// From the plan's per-octant table mat[(o*3+axis)*n*n + m*n + k].
template <class T, int N>
TreeOps<T, N> tree_ops(const double* mat) {
    TreeOps<T, N> o;
    for (int axis = 0; axis < 3; ++axis)
        for (int bit = 0; bit < 2; ++bit)
            for (int mk = 0; mk < N * N; ++mk)  // any octant with this bit on this axis
                o.m[axis][bit][mk] = (T)mat[((bit << axis) * 3 + axis) * N * N + mk];
    return o;
}

// M2M, one CTA per (parent box, chunk of RC rows r); children are contiguous
// (Morton order).  With A[oct] the child of octant oct (zero if absent),
// B[q] = sum_oz Z_oz A[q | oz<<2] (q = ox | oy<<1); C[ox] = sum_oy Y_oy B;
// E_par = sum_ox X_ox C[ox].  The parent row is overwritten (the parent has
// no other contribution), padding nodes written as zero.
// Each stage runs one 1-D line per thread (the n values along the contracted
// axis).  The first stage reads the children's lines straight from global
// memory: along z a line is n consecutive values, so a warp reads a contiguous
// stretch, and shared memory holds only B and C (24 KB in FP32 at order 5, eight
// CTAs an SM; staging the children took 56 KB, three CTAs, a clearing pass and
// an element-wise copy).  Bound: L2 latency and the lines' shared-memory reads.
template <class T, int N>
__global__ void __launch_bounds__(256) k_m2m_tree(const __grid_constant__ TreeOps<T, N> ops,
                                                  const int32_t* __restrict__ octant, int pb0,
                                                  const int32_t* __restrict__ child_first,
                                                  const int32_t* __restrict__ child_count, T* __restrict__ E, int Rb) {
    constexpr int N3 = Ord<N>::n3, NS = Ord<N>::ns, RC = tree_rc<T, N>(), NN = N * N;
    const int pb = pb0 + blockIdx.x;
    const int r0 = blockIdx.y * RC;
    const int rc = min(RC, Rb - r0);
    extern __shared__ __align__(16) unsigned char tree_smem_raw[];
    T* B = reinterpret_cast<T*>(tree_smem_raw);  // [RC][4][N3]
    T* C = B + 4 * RC * N3;                      // [RC][2][N3]
    __shared__ int child[8];  // by octant, -1 if absent
    if (threadIdx.x < 8) child[threadIdx.x] = -1;
    __syncthreads();
    const int cf = child_first[pb], cc = child_count[pb];  // cc <= 8 (octree)
    if (threadIdx.x < cc) child[octant[cf + threadIdx.x]] = cf + threadIdx.x;
    __syncthreads();
    // z: B[r][q][(a,b,c')] = sum_oz sum_c Z_oz[c'][c] A[q|oz<<2][r][(a,b,c)]
    for (int e = threadIdx.x; e < rc * 4 * NN; e += 256) {
        const int r = e / (4 * NN), q = (e / NN) & 3, ab = e % NN;
        const int c0 = child[q], c1 = child[q | 4];
        T x0[N], x1[N];
#pragma unroll
        for (int c = 0; c < N; ++c) x0[c] = x1[c] = (T)0;
        if (c0 >= 0) {
            const T* a = E + ((int64_t)c0 * Rb + r0 + r) * NS + ab * N;
#pragma unroll
            for (int c = 0; c < N; ++c) x0[c] = a[c];
        }
        if (c1 >= 0) {
            const T* a = E + ((int64_t)c1 * Rb + r0 + r) * NS + ab * N;
#pragma unroll
            for (int c = 0; c < N; ++c) x1[c] = a[c];
        }
        T* out = B + (r * 4 + q) * N3 + ab * N;
#pragma unroll
        for (int cp = 0; cp < N; ++cp) {
            T s = (T)0;
#pragma unroll
            for (int c = 0; c < N; ++c) s += ops.m[2][0][cp * N + c] * x0[c] + ops.m[2][1][cp * N + c] * x1[c];
            out[cp] = s;
        }
    }
    __syncthreads();
    // y: C[r][ox][(a,b',c)] = sum_oy sum_b Y_oy[b'][b] B[r][ox|oy<<1][(a,b,c)]
    for (int e = threadIdx.x; e < rc * 2 * NN; e += 256) {
        const int r = e / (2 * NN), ox = (e / NN) & 1, ac = e % NN, a = ac / N, c = ac % N;
        const T* b0 = B + (r * 4 + ox) * N3 + a * NN + c;
        const T* b1 = B + (r * 4 + (ox | 2)) * N3 + a * NN + c;
        T x0[N], x1[N];
#pragma unroll
        for (int b = 0; b < N; ++b) {
            x0[b] = b0[b * N];
            x1[b] = b1[b * N];
        }
        T* out = C + (r * 2 + ox) * N3 + a * NN + c;
#pragma unroll
        for (int bp = 0; bp < N; ++bp) {
            T s = (T)0;
#pragma unroll
            for (int b = 0; b < N; ++b) s += ops.m[1][0][bp * N + b] * x0[b] + ops.m[1][1][bp * N + b] * x1[b];
            out[bp * N] = s;
        }
    }
    __syncthreads();
    // x: E_par[r][(a',b,c)] = sum_ox sum_a X_ox[a'][a] C[r][ox][(a,b,c)]; padding nodes zero
    T* dst = E + ((int64_t)pb * Rb + r0) * NS;
    for (int e = threadIdx.x; e < rc * NN; e += 256) {
        const int r = e / NN, bc = e % NN;
        const T* c0 = C + r * 2 * N3 + bc;
        const T* c1 = c0 + N3;
        T x0[N], x1[N];
#pragma unroll
        for (int a = 0; a < N; ++a) {
            x0[a] = c0[a * NN];
            x1[a] = c1[a * NN];
        }
#pragma unroll
        for (int ap = 0; ap < N; ++ap) {
            T s = (T)0;
#pragma unroll
            for (int a = 0; a < N; ++a) s += ops.m[0][0][ap * N + a] * x0[a] + ops.m[0][1][ap * N + a] * x1[a];
            dst[(int64_t)r * NS + ap * NN + bc] = s;
        }
    }
    if constexpr (NS > N3)
        for (int e = threadIdx.x; e < rc * (NS - N3); e += 256) {
            const int r = e / (NS - N3), m = N3 + e % (NS - N3);
            dst[(int64_t)r * NS + m] = (T)0;
        }
}

// L2L, one CTA per (parent box, chunk of RC rows r): the transposed tree.
// C[ox] = X_ox^T L_par; B[ox|oy<<1] = Y_oy^T C[ox]; child of octant oct:
// L_child += Z_oz^T B[oct & 3].  As in M2M the first stage reads the parent's
// lines and the last one updates the children's in global memory, contiguous
// over a warp; shared memory holds C and B.
template <class T, int N>
__global__ void __launch_bounds__(256) k_l2l_tree(const __grid_constant__ TreeOps<T, N> ops,
                                                  const int32_t* __restrict__ octant, int pb0,
                                                  const int32_t* __restrict__ child_first,
                                                  const int32_t* __restrict__ child_count, T* __restrict__ L, int Rb) {
    constexpr int N3 = Ord<N>::n3, NS = Ord<N>::ns, RC = tree_rc<T, N>(), NN = N * N;
    const int pb = pb0 + blockIdx.x;
    const int cf = child_first[pb], cc = child_count[pb];  // cc <= 8 (octree)
    if (cc == 0) return;
    const int r0 = blockIdx.y * RC;
    const int rc = min(RC, Rb - r0);
    extern __shared__ __align__(16) unsigned char tree_smem_raw[];
    T* B = reinterpret_cast<T*>(tree_smem_raw);  // [RC][4][N3]
    T* C = B + 4 * RC * N3;                      // [RC][2][N3]
    __shared__ int oct_s[8];
    if (threadIdx.x < cc) oct_s[threadIdx.x] = octant[cf + threadIdx.x];
    // x: C[r][ox][(a,b,c)] = sum_a' X_ox[a'][a] P[r][(a',b,c)]  (one line per thread)
    const T* src = L + ((int64_t)pb * Rb + r0) * NS;
    for (int e = threadIdx.x; e < rc * NN; e += 256) {
        const int r = e / NN, bc = e % NN;
        T x[N];
#pragma unroll
        for (int ap = 0; ap < N; ++ap) x[ap] = src[(int64_t)r * NS + ap * NN + bc];
#pragma unroll
        for (int ox = 0; ox < 2; ++ox) {
            T* out = C + (r * 2 + ox) * N3 + bc;
#pragma unroll
            for (int a = 0; a < N; ++a) {
                T s = (T)0;
#pragma unroll
                for (int ap = 0; ap < N; ++ap) s += ops.m[0][ox][ap * N + a] * x[ap];
                out[a * NN] = s;
            }
        }
    }
    __syncthreads();
    // y: B[r][q][(a,b,c)] = sum_b' Y_oy[b'][b] C[r][ox][(a,b',c)],  q = ox | oy<<1
    for (int e = threadIdx.x; e < rc * 2 * NN; e += 256) {
        const int r = e / (2 * NN), ox = (e / NN) & 1, ac = e % NN, a = ac / N, c = ac % N;
        const T* cr = C + (r * 2 + ox) * N3 + a * NN + c;
        T x[N];
#pragma unroll
        for (int bp = 0; bp < N; ++bp) x[bp] = cr[bp * N];
#pragma unroll
        for (int oy = 0; oy < 2; ++oy) {
            T* out = B + (r * 4 + (ox | (oy << 1))) * N3 + a * NN + c;
#pragma unroll
            for (int b = 0; b < N; ++b) {
                T s = (T)0;
#pragma unroll
                for (int bp = 0; bp < N; ++bp) s += ops.m[1][oy][bp * N + b] * x[bp];
                out[b * N] = s;
            }
        }
    }
    __syncthreads();
    // z, straight into each existing child: L_child[r][(a,b,c)] += sum_c' Z_oz[c'][c] B[r][oct&3][(a,b,c')]
    for (int e = threadIdx.x; e < cc * RC * NN; e += 256) {
        const int k = e / (RC * NN), r = (e / NN) % RC, ab = e % NN;
        if (r >= rc) continue;
        const int oc = oct_s[k], q = oc & 3, oz = oc >> 2;
        T* dst = L + ((int64_t)(cf + k) * Rb + r0 + r) * NS + ab * N;
        T old[N];
#pragma unroll
        for (int c = 0; c < N; ++c) old[c] = dst[c];
        const T* br = B + (r * 4 + q) * N3 + ab * N;
        T x[N];
#pragma unroll
        for (int cp = 0; cp < N; ++cp) x[cp] = br[cp];
        auto line = [&](const T* m) {
#pragma unroll
            for (int c = 0; c < N; ++c) {
                T s = (T)0;
#pragma unroll
                for (int cp = 0; cp < N; ++cp) s += m[cp * N + c] * x[cp];
                dst[c] = old[c] + s;
            }
        };
        if (oz)  // a branch, so that the coefficients' addresses are constants
            line(ops.m[2][1]);
        else
            line(ops.m[2][0]);
    }
}

// FP64 M2L with dense operators: CTA per target box, 64 (m) x 64 (r) tile,
// 4x4 register tile per thread, operator and source tiles of 32 along the
// contraction in shared memory.  K table: 343 x n3 x n3; E, L: node stride ns.
__global__ void __launch_bounds__(256) k_m2l64(DevPlan p, int b0, double* __restrict__ L, const double* __restrict__ E,
                                               int R, double scale) {
    const int tb = b0 + blockIdx.x;
    const int n3 = p.n3, ns = p.ns;
    __shared__ double Ks[32][65];  // [l][m]
    __shared__ double Ms[32][65];  // [l][r]
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int64_t s0 = p.m2l_off[tb], s1 = p.m2l_off[tb + 1];
    if (s0 == s1) return;
    for (int mc = 0; mc < n3; mc += 64) {
        for (int rcn = 0; rcn < R; rcn += 64) {
            double acc[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;
            for (int64_t e = s0; e < s1; ++e) {
                const double* K = p.m2l_K + (int64_t)p.m2l_slot[e] * n3 * n3;
                const double* Es = E + (int64_t)p.m2l_src[e] * R * ns;
                for (int lc = 0; lc < n3; lc += 32) {
                    __syncthreads();
                    for (int idx = threadIdx.x; idx < 32 * 64; idx += 256) {
                        const int a = idx >> 5, b = idx & 31;  // a: m or r (64), b: l (32)
                        Ks[b][a] = (mc + a < n3 && lc + b < n3) ? K[(int64_t)(mc + a) * n3 + lc + b] : 0.0;
                        Ms[b][a] = (rcn + a < R && lc + b < n3) ? Es[(int64_t)(rcn + a) * ns + lc + b] : 0.0;
                    }
                    __syncthreads();
#pragma unroll 4
                    for (int l = 0; l < 32; ++l) {
                        double kv[4], mv[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) kv[i] = Ks[l][ty + 16 * i];
#pragma unroll
                        for (int j = 0; j < 4; ++j) mv[j] = Ms[l][tx + 16 * j];
#pragma unroll
                        for (int i = 0; i < 4; ++i)
#pragma unroll
                            for (int j = 0; j < 4; ++j) acc[i][j] += kv[i] * mv[j];
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int mm = mc + ty + 16 * i, rr = rcn + tx + 16 * j;
                    if (mm < n3 && rr < R) L[((int64_t)tb * R + rr) * ns + mm] += scale * acc[i][j];
                }
        }
    }
}

inline unsigned cdiv(int64_t a, int64_t b) { return (unsigned)((a + b - 1) / b); }

template <class T, int N>
void far_field_n(Ctx& c, const DevPlan& p, const FarLaunch& f, const T* X, const FarWeights<T>& w, double* Y, int R,
                 int Rb, T* E, T* L, double coef, const M2LLevelFn<T>& m2l, bool m2l_all, const P2MSplit* p2m_tc,
                 bool l_written) {
    cudaStream_t s = c.stream;
    constexpr int N3 = Ord<N>::n3, NS = Ord<N>::ns, RC = tree_rc<T, N>();
    constexpr size_t smem = tree_smem<T, N>();
    const int Lv = p.L;
    const double wb = (double)sizeof(T);
    const double box_bytes = wb * N3 * R;
    const unsigned rchunks_tree = cdiv(Rb, RC);
    if (!l_written)
        launch_zero(c, L, (size_t)p.nbox * NS * Rb * sizeof(T));  // a kernel: also valid inside a device-side loop
    {
        KTimer t(c, prec_tag<T>(K_P2M), (double)p.N * (wb * R + wb * N3 + 8.0) + (p.nleaf + 2.0 * f.npart) * box_bytes,
                 2.0 * (double)p.N * N3 * R);
        if constexpr (sizeof(T) == 8) {
            by_chunk<N>(R, [&](auto nt) { run_p2m64<N, nt>(c, p, f.p2m_slot, X, w, E, R); });
        } else if (p2m_tc && (N == 4 || N == 5)) {
            launch_p2m_tc(c, p, f.p2m_slot, p2m_tc->whi, p2m_tc->wlo, p2m_tc->xhi, p2m_tc->xlo, E, R, Rb, p2m_tc->err);
        } else {
            by_rows32(Rb, [&](auto rw) { run_p2m32<N, rw>(c, p, f.p2m_slot, X, w, E, R, Rb); });
        }
        if (f.nfix > 0) {
            const int64_t block = (int64_t)Rb * NS;
            k_p2m_fix<T><<<dim3(f.nfix, cdiv(block, 1024)), 256, 0, s>>>(p.nbox, p.leaf_box0, f.fix_leaf, f.fix_first,
                                                                         f.fix_cnt, E, block);
            GPX_LAUNCH_CHECK();
            c.launches += 1;
        }
    }
    const TreeOps<T, N> ops = tree_ops<T, N>(f.m2m1d);
    if (smem > 40 * 1024) {  // with the static part above the 48 KB default
        set_smem_once(k_m2m_tree<T, N>, (int)smem);
        set_smem_once(k_l2l_tree<T, N>, (int)smem);
    }
    for (int l = Lv; l >= 3; --l) {
        const int pb0 = f.lvl_off[l - 1], npb = f.lvl_off[l] - pb0, nch = f.lvl_off[l + 1] - f.lvl_off[l];
        if (npb == 0) continue;
        KTimer t(c, prec_tag<T>(K_M2M), (double)(npb + nch) * box_bytes, 2.0 * 14.0 * N * N3 * R * (double)npb);
        k_m2m_tree<T, N><<<dim3(npb, rchunks_tree), 256, smem, s>>>(ops, p.box_octant, pb0, f.child_first,
                                                                    f.child_count, E, Rb);
        GPX_LAUNCH_CHECK();
        c.launches += 1;
    }
    if (m2l_all && Lv >= 2) {
        const int b0 = f.lvl_off[2], nb = f.lvl_off[Lv + 1] - b0;
        const double pairs = (double)(f.m2l_off[b0 + nb] - f.m2l_off[b0]);
        if (pairs > 0) {
            KTimer t(c, prec_tag<T>(K_M2L), 2.0 * nb * box_bytes, 2.0 * (double)N3 * N3 * R * pairs);
            m2l(-1, b0, nb, 0.0);
            c.launches += 1;
        }
    } else {
        for (int l = 2; l <= Lv; ++l) {
            const int b0 = f.lvl_off[l], nb = f.lvl_off[l + 1] - b0;
            if (nb == 0) continue;
            const double pairs = (double)(f.m2l_off[b0 + nb] - f.m2l_off[b0]);
            if (pairs == 0) continue;
            KTimer t(c, prec_tag<T>(K_M2L), 2.0 * nb * box_bytes, 2.0 * (double)N3 * N3 * R * pairs);
            m2l(l, b0, nb, 1.0 / f.lvl_half[l]);
            c.launches += 1;
        }
    }
    for (int l = 2; l < Lv; ++l) {
        const int pb0 = f.lvl_off[l], npb = f.lvl_off[l + 1] - pb0, ncb = f.lvl_off[l + 2] - f.lvl_off[l + 1];
        if (ncb == 0) continue;
        KTimer t(c, prec_tag<T>(K_L2L), (double)(npb + 2 * ncb) * box_bytes, 2.0 * 14.0 * N * N3 * R * (double)npb);
        k_l2l_tree<T, N><<<dim3(npb, rchunks_tree), 256, smem, s>>>(ops, p.box_octant, pb0, f.child_first,
                                                                    f.child_count, L, Rb);
        GPX_LAUNCH_CHECK();
        c.launches += 1;
    }
    {
        KTimer t(c, prec_tag<T>(K_L2P), (double)p.N * (16.0 * R + 24.0 * N) + p.nleaf * box_bytes, 2.0 * (double)p.N * N3 * R);
        if constexpr (sizeof(T) == 8) {
            by_chunk<N>(R, [&](auto nt) { run_l2p64<N, nt>(c, p, L, w, Y, R, coef); });
        } else if (p2m_tc && p2m_tc->shi && (N == 4 || N == 5)) {
            launch_l2p_tc(c, p, L, p2m_tc->shi, p2m_tc->slo, Y, R, Rb, coef, p2m_tc->err);
        } else {
            by_rows32(Rb, [&](auto rw) { run_l2p32<N, rw>(c, p, L, w, Y, R, Rb, coef); });
        }
    }
}

}  // namespace

template <class T>
void launch_far_field(Ctx& c, const DevPlan& p, const FarLaunch& f, const T* X, const FarWeights<T>& w, double* Y,
                      int R, int Rb, T* E, T* L, double coef, const M2LLevelFn<T>& m2l, bool m2l_all,
                      const P2MSplit* p2m_tc, bool l_written) {
    switch (p.n) {
        case 2: far_field_n<T, 2>(c, p, f, X, w, Y, R, Rb, E, L, coef, m2l, m2l_all, p2m_tc, l_written); break;
        case 3: far_field_n<T, 3>(c, p, f, X, w, Y, R, Rb, E, L, coef, m2l, m2l_all, p2m_tc, l_written); break;
        case 4: far_field_n<T, 4>(c, p, f, X, w, Y, R, Rb, E, L, coef, m2l, m2l_all, p2m_tc, l_written); break;
        case 5: far_field_n<T, 5>(c, p, f, X, w, Y, R, Rb, E, L, coef, m2l, m2l_all, p2m_tc, l_written); break;
        case 6: far_field_n<T, 6>(c, p, f, X, w, Y, R, Rb, E, L, coef, m2l, m2l_all, p2m_tc, l_written); break;
        default: throw Error(GPX_ERR_INVALID_ARG, "far field runs Chebyshev orders 2 to 6");
    }
}

void launch_m2l64(Ctx& c, const DevPlan& p, int b0, int nb, double* L, const double* E, int R, double scale) {
    k_m2l64<<<nb, 256, 0, c.stream>>>(p, b0, L, E, R, scale);
    GPX_LAUNCH_CHECK();
}

template void launch_far_field<double>(Ctx&, const DevPlan&, const FarLaunch&, const double*,
                                       const FarWeights<double>&, double*, int, int, double*, double*, double,
                                       const M2LLevelFn<double>&, bool, const P2MSplit*, bool);
template void launch_far_field<float>(Ctx&, const DevPlan&, const FarLaunch&, const float*, const FarWeights<float>&,
                                      double*, int, int, float*, float*, double, const M2LLevelFn<float>&, bool,
                                      const P2MSplit*, bool);

}  // namespace gpx
