// M2L on the 5th-generation tensor cores (tcgen05, kind::tf32, FP32
// accumulation in tensor memory) for expansions of order 4 (64 nodes) and
// order 5 (125 nodes, stored with a node stride of 128).
//
// For one offset o every target box t with a source s = t + o needs
//     L_t^T (R x NS) += E_s^T (R x NS) * K_o^T (NS x NS).
// A CTA owns G target boxes of one octant class (so their interaction lists
// use the same offsets) with RB right-hand sides each: four boxes of 16 or 32,
// two of 64 (a 64-wide chunk of them for more).  It owns one accumulator D
// (128 x NS, FP32, in TMEM) whose rows are the boxes' right-hand sides, D =
// the stacked E_s(g)^T (A operand) times K_o^T (NS x NS, B operand),
// accumulated over the union of the boxes' offsets.  Expansions are stored
// E[box][r][node] and the operator table K[o][m][l] (target node m, source
// node l), both with node stride NS, so every A row (one right-hand side) and
// every B row (one target node) is a contiguous K-major row: the contraction
// over source nodes runs in atoms of 32 TF32 (one 128-byte swizzle atom per
// row), one or two of them per pipeline stage.
// One thread copies each stage with TMA (a tile per box and one of the
// operator; a box without a source at the offset reads rows past the end of E,
// which are zero) and one thread of another warp waits for the stage's bytes,
// issues its MMAs and commits them to the stage's `empty` mbarrier, on which
// the copies of the next pass wait.  No block-wide barrier in the main loop.
// The work is a stream of tiles from L2 (0.3 to 0.8 GB per apply), so what
// counts is bytes in flight and copies issued: cp.async by 128 threads, each
// arriving on the stage's barrier, took 0.4 us per 24 KB stage whatever was in
// flight, and TMA takes 0.06 us per tile, hence both atoms in one tile where
// they fit.  At 16 columns (21,195-panel bus, depth 5) cp.async over eight
// boxes and two stages took 150 us an apply, this takes 66; at 64 columns (64-
// net window) 134 us and 95.
// The tensor cores read FP32 operands as TF32 (the operator table is stored
// rounded to TF32, the expansions are truncated by the hardware).
// Every mbarrier wait is bounded; on expiry the kernel records an error code,
// drains (bounded) its own MMAs and copies, frees its TMEM and returns.
#include "farfield.cuh"
#include "tma.cuh"

namespace gpx {

namespace {

constexpr int kThreads = 128;  // warp 0 copies, warp 1 multiplies, all four store the accumulator
constexpr int kWaitLimit = 1 << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor: 128 B swizzle, K-major, 8-row groups 1024 B apart.
__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;             // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024u >> 4) << 32;  // stride byte offset
    d |= (uint64_t)1 << 46;             // descriptor version (sm_100)
    d |= (uint64_t)2 << 61;             // SWIZZLE_128B
    return d;
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (int i = 0; i < kWaitLimit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}

template <int NS, int RB>
struct TcCfg {
    static constexpr int kMaxStages = 8;
    static constexpr int kGroup = tc_group(RB);  // boxes
    // Column atoms (32 source nodes) per stage: two where the accumulator's 128
    // rows hold both atoms' rows of every box, so that one copy brings both.
    static constexpr int kAtoms = 2 * kGroup * RB <= 128 ? 2 : 1;
    static constexpr uint32_t kBox = kAtoms * RB * 128;           // one box's operand rows, atom-major
    static constexpr uint32_t kATile = kGroup * kBox;
    static constexpr uint32_t kBTile = kAtoms * NS * 128;
    static constexpr uint32_t kStage = kATile + kBTile;           // multiple of 1024
    // The MMA reads 128 A rows from an atom's start: those that are not its
    // boxes' are the other atom's, other stage memory and past the last stage
    // this pad.  They only reach accumulator rows that are never read.
    static constexpr uint32_t kRead = (kAtoms - 1) * RB * 128 + 128 * 128;
    static constexpr uint32_t kPad = kStage < kRead ? kRead - kStage : 0;
    static constexpr uint32_t smem(int stages) {
        return stages * kStage + kPad + 1024 + 256;  // + alignment slack + barriers
    }
    static constexpr uint32_t kTmemCols = NS;                  // FP32 columns
    static constexpr int kChunks = NS / (32 * kAtoms);         // contraction chunks (stages) per entry
    // Instruction descriptor: D F32, A/B TF32, both K-major, N = NS, M = 128.
    static constexpr uint32_t kIdesc =
        (1u << 4) | (2u << 7) | (2u << 10) | (((uint32_t)NS >> 3) << 17) | ((128u >> 4) << 24);
};

template <int NS, int RB>
__global__ void __launch_bounds__(kThreads) k_m2l_tc(TcLevel lv, const __grid_constant__ CUtensorMap E,
                                                     const __grid_constant__ CUtensorMap K32, float* __restrict__ L,
                                                     int R, int erows, float scale,
                                                     const double* __restrict__ box_scale, int* __restrict__ err,
                                                     int S) {
    using C = TcCfg<NS, RB>;
    constexpr int G = C::kGroup;
    static_assert(C::kAtoms * G * RB <= 128, "one accumulator of 128 rows");
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* sbase = smem_raw + (base - raw);
    uint64_t* bars = reinterpret_cast<uint64_t*>(sbase + S * C::kStage + C::kPad);  // full[S], empty[S]
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 2 * S);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int item = blockIdx.x;
    const int r0 = blockIdx.y * RB;
    const int e0 = lv.item_off[item], e1 = lv.item_off[item + 1];
    const int total = (e1 - e0) * C::kChunks;

    uint64_t* full = bars;
    uint64_t* empty = bars + S;
    __shared__ int s_bad;
    if (tid == 0) {
        for (int k = 0; k < S; ++k) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&full[k])), "r"(1));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&empty[k])));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_bad = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(C::kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = *tslot;

    int issued = 0;  // chunks copied (copy thread), chunks whose MMAs were committed (MMA thread)
    if (tid == 0) {
        // Chunk (entry e, source nodes 32 kc ..) into stage st: A rows RB g ..
        // RB g + RB - 1 from target g's source (rows past the end of E, which
        // read as zero, where a target has no source at this offset); B rows =
        // the operator's target nodes.  The indices of entry e + 1 are read
        // while entry e is copied.
        int cur[G], slot = 0, st = 0, round = 0;  // stage and pass of the ring
        auto fetch = [&](int e, int (&srcs)[G], int& sl) {
#pragma unroll
            for (int g = 0; g < G; ++g) srcs[g] = lv.src[(int64_t)e * G + g];
            sl = lv.slot[e];
        };
        if (e0 < e1) fetch(e0, cur, slot);
        bool stop = false;
        for (int e = e0; e < e1 && !stop; ++e) {
            int next[G], nslot;
            fetch(min(e + 1, e1 - 1), next, nslot);
#pragma unroll
            for (int kc = 0; kc < C::kChunks; ++kc) {
                if ((round > 0 && !mbar_wait(smem_u32(&empty[st]), (uint32_t)((round - 1) & 1))) ||
                    *(volatile int*)&s_bad) {
                    atomicExch(&s_bad, 1);
                    stop = true;
                    break;
                }
                const uint32_t a = base + (uint32_t)st * C::kStage, bar = smem_u32(&full[st]);
                mbar_expect(bar, C::kStage);
#pragma unroll
                for (int g = 0; g < G; ++g)
                    tma_load_atoms(a + g * C::kBox, &E, kc * C::kAtoms, cur[g] >= 0 ? cur[g] * R + r0 : erows, bar);
                tma_load_atoms(a + C::kATile, &K32, kc * C::kAtoms, slot * NS, bar);
                ++issued;
                if (++st == S) {
                    st = 0;
                    ++round;
                }
            }
#pragma unroll
            for (int g = 0; g < G; ++g) cur[g] = next[g];
            slot = nslot;
        }
        // no copy may be in flight when the block ends
        for (int q = issued > S ? issued - S : 0; q < issued; ++q)
            if (!mbar_wait(smem_u32(&full[q % S]), (uint32_t)((q / S) & 1))) atomicExch(&s_bad, 1);
    } else if (tid == 32) {
        int st = 0, round = 0;
        for (int q = 0; q < total; ++q) {
            if (!mbar_wait(smem_u32(&full[st]), (uint32_t)(round & 1))) {
                atomicExch(&s_bad, 1);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t abase = base + (uint32_t)st * C::kStage, bbase = abase + C::kATile;
#pragma unroll
            for (int i = 0; i < 4 * C::kAtoms; ++i) {
                const uint32_t at = i / 4, k = i % 4;
                const uint64_t bd = desc_sw128(bbase + at * (NS * 128) + k * 32u);
                const uint32_t acc = (q > 0 || i > 0) ? 1u : 0u;
                const uint64_t ad = desc_sw128(abase + at * (RB * 128) + k * 32u);
                asm volatile(
                    "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                    "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
                    "l"(ad), "l"(bd), "r"(C::kIdesc), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&empty[st]))
                         : "memory");
            issued = q + 1;
            if (++st == S) {
                st = 0;
                ++round;
            }
        }
        // Drain: the last commit covers every MMA issued before it (after an
        // expired wait too, so the TMEM is idle before it is freed).
        if (issued > 0) {
            const int last = issued - 1;
            if (!mbar_wait(smem_u32(&empty[last % S]), (uint32_t)((last / S) & 1))) atomicExch(&s_bad, 1);
        }
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (s_bad) {
        if (tid == 0) atomicExch(err, 1);
    } else if (total > 0) {
        // Epilogue: warp w (0..3) reads TMEM lanes 32w..32w+31 = rows of D.
        const int row = warp * 32 + lane;
        const int g = row / (C::kAtoms * RB), rr = row % (C::kAtoms * RB);
        const int t = g < G && rr < RB ? lv.item_t[(int64_t)item * G + g] : -1;
        float* dst = (t >= 0) ? L + ((int64_t)t * R + r0 + rr) * NS : nullptr;
        const float sc = (t >= 0 && box_scale) ? (float)box_scale[t] : scale;
#pragma unroll
        for (int cb = 0; cb < NS / 16; ++cb) {
            uint32_t v[16];
            tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(cb * 16), v);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (dst) {
#pragma unroll
                for (int k = 0; k < 16; k += 4) {
                    const float4 o = make_float4(sc * __uint_as_float(v[k]), sc * __uint_as_float(v[k + 1]),
                                                 sc * __uint_as_float(v[k + 2]), sc * __uint_as_float(v[k + 3]));
                    *reinterpret_cast<float4*>(dst + cb * 16 + k) = o;
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::kTmemCols));
}

// Stages: what the CTAs that share an SM leave each other of its shared memory
// (227 KB, 1 KB of it reserved per CTA), four CTAs at most, since the grids of
// many items fill the copy path with four CTAs of two stages.
template <int NS, int RB>
void launch_rb(Ctx& c, const TcLevel& lv, const float* E, int64_t nbox, float* L, const float* K32, int R,
              float scale, const double* box_scale, int* err) {
    using Cf = TcCfg<NS, RB>;
    const int64_t ctas = (int64_t)lv.nitems * (R / RB);
    const int per_sm = (int)std::min<int64_t>(4, (ctas + c.sm_count - 1) / c.sm_count);
    const int room = 227 * 1024 / per_sm - 1024;
    int S = Cf::kMaxStages;
    while (S > 2 && (int)Cf::smem(S) > room) --S;
    set_smem_once(k_m2l_tc<NS, RB>, (int)Cf::smem(S));
    k_m2l_tc<NS, RB><<<dim3(lv.nitems, R / RB), kThreads, Cf::smem(S), c.stream>>>(
        lv, tma_map_f32(E, nbox * R, NS, RB, Cf::kAtoms), tma_map_f32(K32, (int64_t)343 * NS, NS, NS, Cf::kAtoms), L, R, (int)(nbox * R),
        scale, box_scale, err, S);
    GPX_LAUNCH_CHECK();
}

template <int NS>
void launch_ns(Ctx& c, const TcLevel& lv, const float* E, int64_t nbox, float* L, const float* K32, int R,
               float scale, const double* box_scale, int* err) {
    if (R == 16)
        launch_rb<NS, 16>(c, lv, E, nbox, L, K32, R, scale, box_scale, err);
    else if (R == 32)
        launch_rb<NS, 32>(c, lv, E, nbox, L, K32, R, scale, box_scale, err);
    else
        launch_rb<NS, 64>(c, lv, E, nbox, L, K32, R, scale, box_scale, err);
}

}  // namespace

void launch_m2l_tc(Ctx& c, const TcLevel& lv, int ns, const float* E, int64_t nbox, float* L, const float* K32, int R,
                   float scale, const double* box_scale, int* err) {
    if (lv.nitems == 0) return;
    if (R != 16 && R != 32 && R % 64 != 0)
        throw Error(GPX_ERR_INTERNAL, "tensor-core M2L needs 16, 32 or a multiple of 64 rows per box");
    if (nbox * R > INT32_MAX - 128) throw Error(GPX_ERR_INTERNAL, "expansion rows past 32-bit tile coordinates");
    if (ns == 64)
        launch_ns<64>(c, lv, E, nbox, L, K32, R, scale, box_scale, err);
    else if (ns == 128)
        launch_ns<128>(c, lv, E, nbox, L, K32, R, scale, box_scale, err);
    else
        throw Error(GPX_ERR_INTERNAL, "tensor-core M2L runs node strides 64 and 128 (orders 4 and 5)");
}

}  // namespace gpx
