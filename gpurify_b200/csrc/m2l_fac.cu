// Factored M2L for low-rank (compressed) operators K_o = U_o Vt_o, in two
// GEMM phases over every level:
//   phase 1, per source box s: for every column c = (pair e, k) of the
//     source's outgoing pairs, T[t_e][col(e,k)][r] = sum_l Vt_o[k][l] E_s[r][l];
//   phase 2, per target box t: L_t[r][m] = scale * sum_c T_t[c][r] Ut[c][m],
//     the contraction running over the concatenated ranks of t's pairs.
// T is stored target-major and column-major (Kp_t columns of R values per
// target, Kp_t = the summed ranks rounded up to 4): phase 1 writes each column
// as contiguous rows of R, phase 2 reads contiguous K-chunks.  The lists hold
// one entry per pair; each CTA expands its pairs into columns in shared memory
// (as many as 17 per pair at order 5, so uploading columns would take most of
// the plan's upload).
//
// FP64 runs on mma.sync (dmma.cuh) with column tiles that follow R, FP32 on
// the CUDA cores with 16-, 32- or 64-column tiles (13,846 box pairs: 96, 137
// and 216 us per FP32 apply; with operands read one at a time from shared
// memory 113, 172 and 279).  One FP64 apply (both phases), against the
// 64-column FMA tiles it replaced:
//   order 5, R = 64, 62,802 box pairs:  0.96 ms (1.98 before; 0.8 at the FP64 rate)
//   order 6, R = 24, 96,750 box pairs:  1.38 ms (6.23)
//   order 5, R = 16, 31,940 box pairs:  0.22 ms (0.95)
//   order 4, R = 4, 4,528 box pairs:    34 us (135)
// Both phases start the items with most columns first (the host sorts them):
// in the order of the boxes the first of these took 1.09 ms, 12 to 14 % of the
// SM cycles idle behind the last long items.
#include "dmma.cuh"
#include "farfield.cuh"

namespace gpx {

namespace {

// FP32: contraction steps per stage, and stages of phase 1 and phase 2
constexpr int kFac32Chunk = 32, kV32Stages = 2, kU32Stages = 3;

inline unsigned cdiv(int64_t a, int64_t b) { return (unsigned)((a + b - 1) / b); }

// Columns of a source item: the Vt row (slot * kFacMaxRank + k) and the T row
// each one writes.
template <class T>
__device__ __forceinline__ void expand_source(const FacM2L<T>& f, const FacItem& it, int32_t* col_vt, int64_t* col_t) {
    const int64_t c0 = f.src_col[it.p0];
    for (int p = it.p0 + threadIdx.x; p < it.p1; p += blockDim.x) {
        const int slot = f.src_slot[p], r = f.rank[slot], c = (int)(f.src_col[p] - c0);
        const int64_t row = f.src_trow[p];
        for (int k = 0; k < r; ++k) {
            col_vt[c + k] = slot * kFacMaxRank + k;
            col_t[c + k] = row + k;
        }
    }
}

// Ut row (slot * kFacMaxRank + k) of every column of target box t.
template <class T>
__device__ __forceinline__ void expand_target(const FacM2L<T>& f, int t, uint16_t* col_ut) {
    const int64_t e1 = f.m2l_off[t + 1];
    for (int64_t e = f.m2l_off[t] + threadIdx.x; e < e1; e += blockDim.x) {
        const int slot = f.m2l_slot[e], r = f.rank[slot], c = f.tgt_col[e];
        for (int k = 0; k < r; ++k) col_ut[c + k] = (uint16_t)(slot * kFacMaxRank + k);
    }
}

// Phase 1, FP64.  One CTA of four warps per (source item, chunk of 8 NT
// right-hand sides).  The source expansion (8 NT rows of ns nodes) is staged
// once in shared memory; each warp takes blocks of 8 MT columns and reads
// their Vt rows, which no other warp of the item needs, straight into
// registers, two 8-node steps ahead.  The row pitch ns + 4 puts the 4 nodes of
// 4 rows in distinct banks.  Nodes are contracted in ascending order (see the
// near apply in kernels.cu).
// Bound: FP64 tensor rate at R = 64 (per column 2 n^3 R flop against 8 n^3
// bytes of Vt from L2); L2 at R <= 16.
template <int NT, int MT>
__global__ void __launch_bounds__(128) k_fac_v64(FacM2L<double> f, const FacItem* __restrict__ items,
                                                 const double* __restrict__ E, int R, int ksteps) {
    const FacItem it = items[blockIdx.x];
    const int rc = blockIdx.y * (8 * NT);
    const int rows = min(8 * NT, R - rc), ns = f.ns, pitch = ns + 4;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* Es = reinterpret_cast<double*>(smem_raw);                       // [8 NT][pitch]
    int64_t* col_t = reinterpret_cast<int64_t*>(Es + 8 * NT * pitch);       // [kFacItemCols]
    int32_t* col_vt = reinterpret_cast<int32_t*>(col_t + kFacItemCols);     // [kFacItemCols]
    const double* src = E + ((int64_t)it.src * R + rc) * ns;
    const int pieces = ns / 2;
    for (int e = threadIdx.x; e < 8 * NT * pieces; e += blockDim.x) {
        const int r = e / pieces, l = 2 * (e - r * pieces);
        cp_async_16(Es + r * pitch + l, r < rows ? src + (int64_t)r * ns + l : src, r < rows);
    }
    cp_async_fence();
    expand_source(f, it, col_vt, col_t);
    const int ncols = (int)(f.src_col[it.p1] - f.src_col[it.p0]);
    cp_async_wait_for<0>();
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = lane >> 2, q = lane & 3;
    const double* eb = Es + row * pitch + q;
    for (int c0 = warp * 8 * MT; c0 < ncols; c0 += 4 * 8 * MT) {
        const double* a_ptr[MT];
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            const int c = min(c0 + 8 * i + row, ncols - 1);  // rows past the end repeat the last column, never stored
            a_ptr[i] = f.Vt + (int64_t)col_vt[c] * ns + q;
        }
        double acc[MT][NT][2];
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
        double a[2][MT][2];  // the next two 8-node steps (rows hold ns >= 32 nodes, so step 1 is readable)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                a[h][i][0] = __ldg(a_ptr[i] + 8 * h);
                a[h][i][1] = __ldg(a_ptr[i] + 8 * h + 4);
            }
#pragma unroll 2
        for (int s = 0; s < ksteps; ++s) {
            double cur[MT][2];
            const int nx = min(s + 2, ksteps - 1);
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    cur[i][h] = a[0][i][h];
                    a[0][i][h] = a[1][i][h];
                    a[1][i][h] = __ldg(a_ptr[i] + 8 * nx + 4 * h);
                }
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const double b = eb[8 * j * pitch + 8 * s + 4 * h];
#pragma unroll
                    for (int i = 0; i < MT; ++i) dmma(acc[i][j], cur[i][h], b);
                }
        }
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            const int c = c0 + 8 * i + row;
            if (c >= ncols) continue;
            double* dst = f.Tm + col_t[c] * R + rc + 2 * q;
#pragma unroll
            for (int j = 0; j < NT; ++j)
                if (8 * j + 2 * q < rows) *reinterpret_cast<double2*>(dst + 8 * j) = make_double2(acc[i][j][0], acc[i][j][1]);
        }
    }
}

// Phase 2, FP64.  One CTA per (target box, chunk of 8 NT right-hand sides),
// one warp per 32 nodes (ns / 32 warps); the contraction streams KC columns of
// T and their gathered Ut rows per stage through a four-stage cp.async ring.
// The pitches (8 NT + 4 and ns + 4 doubles, both 4 more than a multiple of 8)
// keep the four contraction rows of a fragment read in distinct banks.  L is
// written, not added to (boxes without pairs get zero), so the caller clears
// nothing.  Bound: FP64 tensor rate at R = 64, L2 (Ut rows) at R <= 16.
template <int NT, int NS>
struct FacU64 {
    static constexpr int KC = NT >= 3 ? 8 : 16;  // short tiles: fewer barriers per flop
    static constexpr int kStages = 4;
    static constexpr int TP = 8 * NT + 4, UP = NS + 4;
    static constexpr int kSmem = (int)sizeof(double) * kStages * KC * (TP + UP);  // + the column list
    // 64-column tiles would take 183 registers and leave two CTAs an SM at
    // order 5; three need at most 168 (phase 2 of the 64-net window 707 us with
    // two, 540 with three, 490 with the longest boxes first)
    static constexpr int kMinCtas = NS == 128 ? 3 : NS < 128 ? 4 : 1;
};
template <int NT, int NS>
__global__ void __launch_bounds__(NS, (FacU64<NT, NS>::kMinCtas))
    k_fac_u64(FacM2L<double> f, int b0, double* __restrict__ L, int R) {
    using C = FacU64<NT, NS>;
    constexpr int KC = C::KC, S = C::kStages, TP = C::TP, UP = C::UP, ns = NS;
    const int t = f.tgt_order[b0 + blockIdx.x], rc = blockIdx.y * (8 * NT);
    const int rows = min(8 * NT, R - rc);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
    const int K = (int)(f.tgt_col_off[t + 1] - f.tgt_col_off[t]);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* Ts = reinterpret_cast<double*>(smem_raw);           // [S][KC][TP]
    double* Us = Ts + S * KC * TP;                              // [S][KC][UP]
    uint16_t* col = reinterpret_cast<uint16_t*>(Us + S * KC * UP);
    double* out = L + ((int64_t)t * R + rc + g) * ns + 32 * warp + 2 * q;
    double acc[NT][4][2];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    if (K > 0) {
        expand_target(f, t, col);
        __syncthreads();
        const double* Tt = f.Tm + f.tgt_base[t] * R + rc;
        const int nst = (K + KC - 1) / KC;
        constexpr int tp = 4 * NT, up = ns / 2;  // 16-byte pieces of a T row and a Ut row
        auto issue = [&](int s) {
            if (s < nst) {
                const int k0 = s * KC;
                double* ts = Ts + (s % S) * KC * TP;
                double* us = Us + (s % S) * KC * UP;
#pragma unroll
                for (int e = threadIdx.x; e < KC * tp; e += NS) {
                    const int k = e / tp, r = 2 * (e - k * tp);
                    const bool ok = k0 + k < K && r < rows;
                    cp_async_16(ts + k * TP + r, ok ? Tt + (int64_t)(k0 + k) * R + r : f.Tm, ok);
                }
#pragma unroll
                for (int e = threadIdx.x; e < KC * up; e += NS) {
                    const int k = e / up, m = 2 * (e - k * up);
                    const bool ok = k0 + k < K;
                    cp_async_16(us + k * UP + m, ok ? f.Ut + (int64_t)col[k0 + k] * ns + m : f.Ut, ok);
                }
            }
            cp_async_fence();
        };
#pragma unroll
        for (int s = 0; s < S - 1; ++s) issue(s);
        for (int s = 0; s < nst; ++s) {
            cp_async_wait_for<S - 2>();
            __syncthreads();
            issue(s + S - 1);
            const double* ts = Ts + (s % S) * KC * TP + q * TP + g;
            const double* us = Us + (s % S) * KC * UP + q * UP + 32 * warp + g;
#pragma unroll
            for (int k = 0; k < KC; k += 4) {
                double b[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = us[k * UP + 8 * j];
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    const double a = ts[k * TP + 8 * i];
#pragma unroll
                    for (int j = 0; j < 4; ++j) dmma(acc[i][j], a, b[j]);
                }
            }
        }
        cp_async_wait_for<0>();
    }
    const double sc = f.box_scale[t];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        if (8 * i + g >= rows) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            *reinterpret_cast<double2*>(out + (int64_t)(8 * i) * ns + 8 * j) =
                make_double2(sc * acc[i][j][0], sc * acc[i][j][1]);
    }
}

// Phase 1, FP32: a GEMM per (source item, 8 RI right-hand sides), C[c][r] =
// sum_l Vt_c[l] E_s[r][l].  E_s is staged once per item; the gathered Vt rows
// of each CT-column sub-block stream through a cp.async ring over the ns
// nodes.  CT threads, 8 x RI outputs per thread (columns ty + (CT/8) i, rows
// tx + 8 j).  Both tiles are contiguous along the contraction, so a thread
// reads four nodes of a row at once: 10 shared reads for 64 FMAs at RI = 2,
// where one node at a time took 40 and bound the kernel.  Pitches of 4 more
// than a multiple of 32 words keep the reads free of bank conflicts.  Nodes are
// added in ascending order.
template <int CT, int RI>
__global__ void __launch_bounds__(CT) k_fac_v32(FacM2L<float> f, const FacItem* __restrict__ items,
                                                const float* __restrict__ E, int R) {
    constexpr int V = 4, KC = kFac32Chunk, S = kV32Stages, PP = KC + V;
    constexpr int CS = CT / 8;  // column stride of a thread's tile
    const int ns = f.ns;
    const FacItem it = items[blockIdx.x];
    const int rc = blockIdx.y * (8 * RI);
    const int rows = min(8 * RI, R - rc), BP = ns + V;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float(*As)[CT][PP] = reinterpret_cast<float(*)[CT][PP]>(smem_raw);  // [S][CT][PP]: [c][l]
    int64_t* col_t = reinterpret_cast<int64_t*>(smem_raw + sizeof(float) * S * CT * PP);
    int32_t* col_vt = reinterpret_cast<int32_t*>(col_t + kFacItemCols);
    float* Bs = reinterpret_cast<float*>(col_vt + kFacItemCols);  // [8 RI][BP]: [r][l]
    expand_source(f, it, col_vt, col_t);
    const int ncols = (int)(f.src_col[it.p1] - f.src_col[it.p0]);
    __syncthreads();
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
    const int nch = ns / KC;                 // node chunks per sub-block
    const int nsub = (ncols + CT - 1) / CT;  // CT-column sub-blocks
    const int nsteps = nsub * nch;
    auto issue = [&](int step) {
        if (step < nsteps) {
            const int sub = step / nch, ch = step % nch;
            const int nc = min(CT, ncols - CT * sub);
            const int k0 = ch * KC, buf = step % S;
#pragma unroll
            for (int q = 0; q < KC / V; ++q) {
                const int id = tid + CT * q, row = id / (KC / V), kc = (id % (KC / V)) * V;
                const bool ok = row < nc;
                cp_async_16(&As[buf][row][kc], ok ? f.Vt + (int64_t)col_vt[CT * sub + row] * ns + k0 + kc : f.Vt, ok);
            }
        }
        cp_async_fence();
    };
    const float* Es = E + ((int64_t)it.src * R + rc) * ns;
    for (int e = tid; e < 8 * RI * (ns / V); e += CT) {
        const int r = e / (ns / V), l = (e % (ns / V)) * V;
        cp_async_16(Bs + r * BP + l, r < rows ? Es + (int64_t)r * ns + l : Es, r < rows);
    }
#pragma unroll
    for (int s = 0; s < S - 1; ++s) issue(s);
    float acc[8][RI];
    for (int step = 0; step < nsteps; ++step) {
        const int sub = step / nch, ch = step % nch;
        if (ch == 0) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < RI; ++j) acc[i][j] = 0.f;
        }
        cp_async_wait_for<S - 2>();
        __syncthreads();
        issue(step + S - 1);
        const int buf = step % S;
#pragma unroll 2
        for (int kk = 0; kk < KC; kk += V) {
            float4 b[RI];
#pragma unroll
            for (int j = 0; j < RI; ++j)
                b[j] = *reinterpret_cast<const float4*>(Bs + (tx + 8 * j) * BP + ch * KC + kk);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(&As[buf][ty + CS * i][kk]);
#pragma unroll
                for (int j = 0; j < RI; ++j) {
                    acc[i][j] += a.x * b[j].x;
                    acc[i][j] += a.y * b[j].y;
                    acc[i][j] += a.z * b[j].z;
                    acc[i][j] += a.w * b[j].w;
                }
            }
        }
        if (ch == nch - 1) {
            const int nc = min(CT, ncols - CT * sub);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int c = ty + CS * i;
                if (c >= nc) continue;
                float* dst = f.Tm + col_t[CT * sub + c] * R + rc;
#pragma unroll
                for (int j = 0; j < RI; ++j) {
                    const int r = tx + 8 * j;
                    if (r < rows) dst[r] = acc[i][j];
                }
            }
        }
    }
}

// Phase 2, FP32: CTA per (target box, 8 RI rows r, MW nodes m), a warp per 32
// nodes and all rows, 2 RI x 4 outputs per thread (rows 16 h + 4 ry + {0..3},
// nodes 32 warp + 4 nx + {0..3}); the contraction over the target's
// concatenated ranks streams A = T rows and B = gathered Ut rows through a
// cp.async ring, both contiguous along a thread's outputs, which it reads 16
// bytes at a time.  Shared reads bound it at few rows: with warps of 128 nodes x
// 4 rows five wavefronts fed 16 FMAs at RI = 2, with 32 x 16 two do.  L is
// written, not added to.
template <int MW, int RI>
__global__ void __launch_bounds__(MW) k_fac_u32(FacM2L<float> f, int b0, float* __restrict__ L, int R) {
    constexpr int V = 4, KC = kFac32Chunk, S = kU32Stages, XP = MW + V, RW = 8 * RI, AP = RW + V, RT = RW / 4;
    const int ns = f.ns;
    const int t = f.tgt_order[b0 + blockIdx.x];
    const int rc = blockIdx.y * RW;
    const int m0 = blockIdx.z * MW;
    const int K = (int)(f.tgt_col_off[t + 1] - f.tgt_col_off[t]);
    const float sc = (float)f.box_scale[t];
    const float* A = f.Tm + f.tgt_base[t] * R + rc;  // column-major: A[c][r] at c * R + r
    const int m = min(RW, R - rc);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float(*As)[KC][AP] = reinterpret_cast<float(*)[KC][AP]>(smem_raw);                             // [S][KC][AP]: [c][r]
    float(*Bs)[KC][XP] = reinterpret_cast<float(*)[KC][XP]>(smem_raw + sizeof(float) * S * KC * AP);  // [S][KC][XP]
    uint16_t* col = reinterpret_cast<uint16_t*>(smem_raw + sizeof(float) * S * KC * (AP + XP));
    const int tid = threadIdx.x, nx = tid & 7, ry = (tid & 31) >> 3, node = 32 * (tid >> 5) + V * nx;
    const int nchunk = (K + KC - 1) / KC;
    auto issue = [&](int cch) {
        if (cch < nchunk) {
            const int k0 = cch * KC, buf = cch % S;
            for (int id = tid; id < KC * (RW / V); id += MW) {
                const int kk = id / (RW / V), rr = (id % (RW / V)) * V;
                const bool ok = k0 + kk < K && rr < m;
                cp_async_16(&As[buf][kk][rr], ok ? A + (int64_t)(k0 + kk) * R + rr : f.Tm, ok);
            }
            for (int id = tid; id < KC * (MW / V); id += MW) {
                const int kk = id / (MW / V), cc = (id % (MW / V)) * V;
                const bool ok = k0 + kk < K && m0 + cc < ns;
                cp_async_16(&Bs[buf][kk][cc], ok ? f.Ut + (int64_t)col[k0 + kk] * ns + m0 + cc : f.Ut, ok);
            }
        }
        cp_async_fence();
    };
    float acc[RT][4];
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    if (K > 0) {
        expand_target(f, t, col);
        __syncthreads();
#pragma unroll
        for (int s = 0; s < S - 1; ++s) issue(s);
    }
    for (int cch = 0; cch < nchunk; ++cch) {
        cp_async_wait_for<S - 2>();
        __syncthreads();
        issue(cch + S - 1);
        const int buf = cch % S;
#pragma unroll 4
        for (int kk = 0; kk < KC; ++kk) {
            const float4 b = *reinterpret_cast<const float4*>(&Bs[buf][kk][node]);
#pragma unroll
            for (int i = 0; i < RT; i += 4) {
                const float4 a4 = *reinterpret_cast<const float4*>(&As[buf][kk][4 * i + 4 * ry]);
                const float a[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    acc[i + q][0] += a[q] * b.x;
                    acc[i + q][1] += a[q] * b.y;
                    acc[i + q][2] += a[q] * b.z;
                    acc[i + q][3] += a[q] * b.w;
                }
            }
        }
    }
    if (m0 + node >= ns) return;  // ns is a multiple of 4
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        const int r = 16 * (i / 4) + 4 * ry + i % 4;
        if (r >= m) continue;
        *reinterpret_cast<float4*>(L + ((int64_t)t * R + rc + r) * ns + m0 + node) =
            make_float4(sc * acc[i][0], sc * acc[i][1], sc * acc[i][2], sc * acc[i][3]);
    }
}

template <int NT, int NS>
void run_fac_u64(Ctx& c, const FacM2L<double>& f, int b0, int nb, double* L, int R) {
    const int smem = FacU64<NT, NS>::kSmem + 2 * ((f.max_cols + 7) & ~7);
    set_smem_once(k_fac_u64<NT, NS>, smem);
    k_fac_u64<NT, NS><<<dim3(nb, cdiv(R, 8 * NT)), NS, smem, c.stream>>>(f, b0, L, R);
    GPX_LAUNCH_CHECK();
}

template <int NT>
void run_fac64(Ctx& c, const FacM2L<double>& f, int b0, int nb, double* L, const double* E, int R, int n3) {
    constexpr int MT = NT >= 6 ? 2 : NT == 5 ? 3 : 4;  // at most 16 accumulator tiles a warp
    if (f.nitems > 0) {
        const int smem = (int)(sizeof(double) * 8 * NT * (f.ns + 4) + 12 * kFacItemCols);
        set_smem_once(k_fac_v64<NT, MT>, smem);
        k_fac_v64<NT, MT><<<dim3(f.nitems, cdiv(R, 8 * NT)), 128, smem, c.stream>>>(f, f.items, E, R, (n3 + 7) / 8);
        GPX_LAUNCH_CHECK();
    }
    switch (f.ns) {
        case 32: run_fac_u64<NT, 32>(c, f, b0, nb, L, R); break;
        case 64: run_fac_u64<NT, 64>(c, f, b0, nb, L, R); break;
        case 128: run_fac_u64<NT, 128>(c, f, b0, nb, L, R); break;
        default:
            if constexpr (NT <= 4) run_fac_u64<NT, 224>(c, f, b0, nb, L, R);
    }
}

template <int RI>
void run_fac32(Ctx& c, const FacM2L<float>& f, int b0, int nb, float* L, const float* E, int R) {
    constexpr int V = 4, KC = kFac32Chunk, CT = 128, RW = 8 * RI;
    if (f.nitems > 0) {
        const int smem = (int)(sizeof(float) * (kV32Stages * CT * (KC + V) + RW * (f.ns + V)) + 12 * kFacItemCols);
        set_smem_once(k_fac_v32<CT, RI>, smem);
        k_fac_v32<CT, RI><<<dim3(f.nitems, cdiv(R, RW)), CT, smem, c.stream>>>(f, f.items, E, R);
        GPX_LAUNCH_CHECK();
    }
    const int cols = 2 * ((f.max_cols + 7) & ~7);
    if (f.ns >= 128) {
        constexpr int MW = 128;
        const int smem = (int)(sizeof(float) * kU32Stages * KC * (RW + V + MW + V)) + cols;
        set_smem_once(k_fac_u32<MW, RI>, smem);
        k_fac_u32<MW, RI><<<dim3(nb, cdiv(R, RW), cdiv(f.ns, MW)), MW, smem, c.stream>>>(f, b0, L, R);
    } else {
        constexpr int MW = 64;
        const int smem = (int)(sizeof(float) * kU32Stages * KC * (RW + V + MW + V)) + cols;
        set_smem_once(k_fac_u32<MW, RI>, smem);
        k_fac_u32<MW, RI><<<dim3(nb, cdiv(R, RW), cdiv(f.ns, MW)), MW, smem, c.stream>>>(f, b0, L, R);
    }
    GPX_LAUNCH_CHECK();
}

}  // namespace

// Chunks of at most 64 right-hand sides, 32 at order 6, whose 224-node rows
// would otherwise leave one CTA per SM.
template <>
void launch_m2l_fac<double>(Ctx& c, const FacM2L<double>& f, int b0, int nb, double* L, const double* E, int R, int n3) {
    switch (rhs_chunk(R, f.ns > 128 ? 32 : 64) / 8) {
        case 1: run_fac64<1>(c, f, b0, nb, L, E, R, n3); break;
        case 2: run_fac64<2>(c, f, b0, nb, L, E, R, n3); break;
        case 3: run_fac64<3>(c, f, b0, nb, L, E, R, n3); break;
        case 4: run_fac64<4>(c, f, b0, nb, L, E, R, n3); break;
        case 5: run_fac64<5>(c, f, b0, nb, L, E, R, n3); break;
        case 6: run_fac64<6>(c, f, b0, nb, L, E, R, n3); break;
        case 7: run_fac64<7>(c, f, b0, nb, L, E, R, n3); break;
        default: run_fac64<8>(c, f, b0, nb, L, E, R, n3); break;
    }
    c.launches += 1;  // the caller counts the other one
}

// R: rows per box, padded to 16, 32 or a multiple of 64 (rhs_pad32).
template <>
void launch_m2l_fac<float>(Ctx& c, const FacM2L<float>& f, int b0, int nb, float* L, const float* E, int R, int) {
    if (R <= 16)
        run_fac32<2>(c, f, b0, nb, L, E, R);
    else if (R <= 32)
        run_fac32<4>(c, f, b0, nb, L, E, R);
    else
        run_fac32<8>(c, f, b0, nb, L, E, R);
    c.launches += 1;  // the caller counts the other one
}

}  // namespace gpx
