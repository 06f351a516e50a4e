// NVFP4 MoE expert down-projection (GEMM2 of the routed experts), the weighted top-k combine, and the tensor-parallel
// reduction that follows, in one kernel for sm_100a.
//
//   y[token, k]   = bf16( (sum over f of act[slot, f] * W2[e, :, f]) * g2[e] )        e = ids[token, k] local to the rank
//   out[token]    = bf16( sum over k in list order of weight[token, k] * y[token, k] )  (+ shared -> bf16)
//   then out is this rank's partial of the all-reduce (experts are split whole across ranks).
//
// Arithmetic follows the reference's statement of the TRT-LLM-gen MoE roundings, dlmrt/ops/triton/nvfp4_moe.py:107-150
// (FP32 dot of E2M1 x E4M3-per-16 operands, times g2, BF16 per (token, expert); FP32 combine in list order); the entry
// point replaces dlmrt/quantization/nvfp4.py:280-306 (`trtllm_moe`) plus the add and reduce of
// dlmrt/models/llada2/model.py:354-362,437-438.
//
// Work item = (entry, 128 output features), entry = (active local expert, block of at most `rows_cap` of its rows). W2's
// [128 x F] slab sits on the MMA's M axis, the entry's rows (padded to 16) on its N axis. Every CTA takes one contiguous
// run of items, so that consecutive items mostly share their entry and the entry's rows are fetched once per run, not
// once per item; what streams is the weights alone:
//   warp 0   TMA: per 256-element k-block the 16 KB code slab of W2 (one bulk copy of a pre-tiled slab, or one box) and
//            its 2 KB of pre-interleaved 128 x 4 scale atoms (one bulk copy)
//   warp 2   TMA, once per entry: its activation rows, all of K (boxes of 8 rows x 128 bytes)
//   warp 3   once per entry: the rows' linear E4M3 scales, rewritten into scale atoms
//   warp 1   per entry: tcgen05.cp the rows' scale atoms into tensor memory, where they stay for all its items (where they
//            fit, else again per k-block); per k-block: tcgen05.cp W2's atoms, then up to four
//            tcgen05.mma.kind::mxf4nvf4.block_scale (K = 64) into the FP32 accumulator
//   warps 4-11  two groups of four, one accumulator buffer each, alternate items: tcgen05.ld, times g2, BF16, scatter
//            rows to Y[pair] through the expert's slot map
// (GEMM1 with a very long K streams the rows with the weights instead, see moe_layout.)
// The kernel is bound by the HBM weight stream if nothing else holds it up, and what held it up was the chain behind each
// k-block: one thread issuing eight scale copies, four MMAs and a commit (the commit alone waits ~340 ns behind eight
// copies), and small copies of activation rows and scales repeated for every item. Rows kept per entry halve the scale
// copies and leave two bulk copies per k-block.
// When all CTAs are through their items (arrival counter), rows of the output are combined from Y in FP32 and pushed
// into the owner ranks' receive slots, and the reduction phases of comm.cuh follow.
//
// The same pipeline, instantiated with GATE_UP, is GEMM1 of the experts (the step in front of the down-projection,
// dlmrt/ops/triton/nvfp4_moe.py:69-104 `_gate_up`): W13 [2F x hidden] streams instead of W2, its rows interleaved
// (row 2i = gate feature i, row 2i + 1 = up feature i) so that a gate value and its up value sit in neighbouring lanes
// of the accumulator; the expert's rows are the NVFP4-quantised tokens routed to it. The epilogue scales by g1, applies
// SwiGLU or GeGLU in FP32, re-quantises to NVFP4 against 1 / a2 (per 16 features: E4M3 scale, E2M1 codes, the
// approximate-reciprocal recipe of nvfp4_moe.py:36-47) and writes codes and scales straight into the expert-major
// slots the down-projection reads. It ends there: no combine, no reduction.
#include "kernels.cuh"

namespace dlm {

namespace {

constexpr int kMoeThreads = kFusedThreads;
constexpr int kCodeTileW = 128 * 128;  // 128 rows x 128 bytes (256 FP4) of W2 codes
constexpr int kBoxRows = 8;            // activation rows per TMA box (one 1 KB swizzle atom)
constexpr int kAtom = 512;             // one 128-row x 4-scale atom
constexpr int kStepsPerBlock = 4;      // K = 64 instructions per 256-element k-block
constexpr int kStageBytes = kCodeTileW + kStepsPerBlock * kAtom;  // 18 KB: a k-block's codes and scale atoms
constexpr int kMaxRowsCap = 128;       // rows of one entry: the MMA's N
// Tensor memory: two accumulators of rows_cap columns, then the scales of the MMAs' operands, four columns per K = 64 step.
// Nothing orders a scale copy behind MMAs issued before it that still read the columns it overwrites (copy before MMA is
// an ordered pair, MMA before copy is not), so every set of columns belongs to the shared memory it is copied from and
// is overwritten only after that has been refilled, which waits for those MMAs: W2's scales have a set per ring stage,
// the entry's row scales all of its steps per row buffer (`resident`) or, where these do not fit, a set per stage too.
constexpr int kTmemCols = 512, kScaleCols = 4 * kStepsPerBlock;
constexpr int kMaxLocalExperts = 256;
constexpr int kMaxEntries = 2 * kMaxLocalExperts;  // one per active expert + one per 16 rows of 4096 pairs at most
constexpr int kMoeStages = 12;
constexpr int kMoeSmemBudget = 222 * 1024;

struct MoeSmem {
    uint64_t full[kMoeStages];
    uint64_t empty[kMoeStages];
    uint64_t a_full[2];
    uint64_t a_empty[2];
    uint64_t acc_full[2];
    uint64_t acc_empty[2];
    uint32_t tmem_base;
    int n_active, epoch, gen, failed;
    int warp_count[8];
    int counted[kMaxLocalExperts];  // GATE_UP: rows of each local expert
    float scratch[64];
    short active[kMaxEntries];  // expert | row block << 8
    short rows[kMaxEntries];    // rows of that block
};

// Shared memory of one entry's rows: codes [k-blocks][rows_cap][128 bytes], then one scale atom per K = 64 step.
__host__ __device__ int entry_bytes(int rows_cap, int k) {
    return (k + 255) / 256 * rows_cap * 128 + (k / 64 + 1) / 2 * (2 * kAtom);  // a multiple of 1 KB
}

// The same for one k-block of the rows, as a ring stage holds it where rows are streamed with the weights.
__host__ __device__ int row_stage_bytes(int rows_cap) { return rows_cap * 128 + kStepsPerBlock * kAtom; }

}  // namespace

// Picks rows_cap, the number of row buffers and the ring's stages for experts of `k` inputs and at most `m_max` rows, of
// which an expert gets `mean_rows` on average. Two buffers hide the fetch of the next entry's rows; the ring wants six
// stages (108 KB in flight per SM cover HBM's latency at full rate), four at least. More rows per entry mean fewer
// passes over an expert's weights (the later ones come out of L2), so the largest cap that leaves the ring its stages is
// taken; where experts have many more rows than that on average, one larger buffer beats two small ones.
// Where K is so long that one buffer holds 16 rows only (above 6400), rows are not kept at all but streamed: each ring
// stage brings the entry's rows of its k-block along with the weights, `most` of them, again for every item. GEMM1 of two
// layers with 1024 features, us with 16 rows kept and streamed: K = 8192, 64 experts of 32 rows 424 and 234, 8 of 256
// 325 and 133, 64 of one 143 and 143; K = 6656, 128 of 8 303 and 311. Up to 6400 32 rows or more are kept: K = 4096, 64
// experts of 32 rows 124 and 156, 16 of 128 96 and 128, 8 of 256 96 and 102; K = 6144 the same three 227 and 213, 149 and
// 167, 147 and 128.
MoeLayout moe_layout(int k, int m_max, int mean_rows) {
    int most = (m_max + 15) / 16 * 16;
    if (most > kMaxRowsCap) most = kMaxRowsCap;
    auto stages_of = [&](int cap, int buffers) { return (kMoeSmemBudget - buffers * entry_bytes(cap, k)) / kStageBytes; };
    MoeLayout best{0, 0, 0, false};
    for (int want = 6; want >= 4; --want) {
        for (int cap = most; cap >= 16; cap -= 16) {
            if (stages_of(cap, 2) < want) continue;
            best = {cap, 2, stages_of(cap, 2), false};
            break;
        }
        if (best.buffers == 2 && (best.rows_cap >= 32 || best.rows_cap == most)) break;
    }
    if (best.buffers == 0 || mean_rows > best.rows_cap) {
        for (int cap = most; cap > best.rows_cap; cap -= 16) {
            if (stages_of(cap, 1) < 4) continue;
            best = {cap, 1, stages_of(cap, 1), false};
            break;
        }
    }
    if (best.buffers < 2 && best.rows_cap < 32 && best.rows_cap < most)
        best = {most, 0, kMoeSmemBudget / (kStageBytes + row_stage_bytes(most)), false};
    if (best.stages > kMoeStages) best.stages = kMoeStages;
    auto tmem_cols = [&](int stages, bool resident) {
        const int rows = resident ? best.buffers * (k / 64) * 4 : stages * kScaleCols;
        return 2 * best.rows_cap + stages * kScaleCols + rows;
    };
    // A stage less, out of six or more, costs less than copying the row scales again for every item.
    if (best.buffers > 0 && best.stages > 5 && tmem_cols(best.stages, true) > kTmemCols &&
        tmem_cols(best.stages - 1, true) <= kTmemCols)
        --best.stages;
    best.resident = best.buffers > 0 && tmem_cols(best.stages, true) <= kTmemCols;
    while (!best.resident && tmem_cols(best.stages, false) > kTmemCols) --best.stages;
    return best;
}

static int moe_smem_bytes(const MoeDev& d) {
    const int rows = d.buffers > 0 ? d.buffers * entry_bytes(d.rows_cap, d.f) : d.stages * row_stage_bytes(d.rows_cap);
    return d.stages * kStageBytes + rows + static_cast<int>(sizeof(MoeSmem)) + 1024;
}

// A token's expert list for the combine step, eight entries at a time: local expert index (or -1) and routing weight.
constexpr int kCombineBatch = 8;
struct CombineMeta {
    int e[kCombineBatch];
    float w[kCombineBatch];
};

// Entries [k0, k0 + 8) of row `row`: all loads are independent, so they cost one round trip, and they depend on
// nothing this launch computes (callers issue them before waiting for the expert outputs).
__device__ __forceinline__ CombineMeta combine_meta(const MoeDev& g, int row, int k0) {
    CombineMeta m;
#pragma unroll
    for (int j = 0; j < kCombineBatch; ++j) {
        const bool have = k0 + j < g.top_k;
        const int e = have ? g.ids[row * g.top_k + k0 + j] - g.lo : -1;
        m.e[j] = e >= 0 && e < g.e_local ? e : -1;
        m.w[j] = have ? g.weights[row * g.top_k + k0 + j] : 0.f;
    }
    return m;
}

// One output row of the combine step for thread t's eight columns: FP32 sum over the token's expert list, in list
// order, of weight * y (fused multiply-add; experts of other ranks contribute 0 * 0), rounded to BF16, then the
// shared expert's BF16 row added and rounded again (dlmrt/ops/triton/nvfp4_moe.py:134-150). `first` holds entries
// [0, 8) of the row, fetched early; the expert outputs of a batch are loaded together and added in list order.
__device__ __forceinline__ uint4 combine_row(const MoeDev& g, int row, int t, const CombineMeta& first) {
    float acc[kVec] = {};
    for (int k0 = 0; k0 < g.top_k; k0 += kCombineBatch) {
        const CombineMeta m = k0 == 0 ? first : combine_meta(g, row, k0);
        uint4 raw[kCombineBatch];
#pragma unroll
        for (int j = 0; j < kCombineBatch; ++j) {
            raw[j] = make_uint4(0, 0, 0, 0);
            if (m.e[j] >= 0)
                raw[j] = __ldcg(reinterpret_cast<const uint4*>(g.y + static_cast<size_t>(row * g.top_k + k0 + j) * g.n) + t);
        }
#pragma unroll
        for (int j = 0; j < kCombineBatch; ++j) {
            if (k0 + j < g.top_k) {
                const float w = m.e[j] >= 0 ? m.w[j] : 0.f;
                const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&raw[j]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 f = __bfloat1622float2(b[i]);
                    acc[2 * i] = fmaf(w, f.x, acc[2 * i]);
                    acc[2 * i + 1] = fmaf(w, f.y, acc[2 * i + 1]);
                }
            }
        }
    }
    uint4 packed = pack_bf16x8(acc);
    if (g.shared) {
        float v[kVec] = {};
        add_bf16x8(v, packed);
        add_bf16x8(v, *(reinterpret_cast<const uint4*>(g.shared + static_cast<size_t>(row) * g.n) + t));
        packed = pack_bf16x8(v);
    }
    return packed;
}

// Single rank: combine each owned row and finish it (residual + RMSNorm by mode, store into OUT) in one go.
template <int MODE>
__device__ __forceinline__ void combine_and_finish(const MoeDev& g, const CommDev& c, int block, int blocks, float* scratch,
                                                   const CombineMeta& first) {
    const int t = threadIdx.x, threads = g.n / kVec;
    const bool active = t < threads;
    const int col = (active ? t : 0) * kVec;
    uint4 wraw = make_uint4(0, 0, 0, 0);
    if (MODE != kReduce && active) wraw = *reinterpret_cast<const uint4*>(c.weight + col);
    for (int row = block; row < g.m; row += blocks) {
        const size_t off = static_cast<size_t>(row) * c.n + col;
        uint4 hraw = make_uint4(0, 0, 0, 0);
        if (MODE == kReduceNormResidual && active) hraw = *reinterpret_cast<const uint4*>(c.h + off);
        float v[kVec] = {};
        if (active) {  // +0.0f + partial: the rank-ordered sum over one rank
            add_bf16x8(v, combine_row(g, row, t, row == block ? first : combine_meta(g, row, 0)));
        }
        finish_row<MODE>(c, v, hraw, wraw, off, active, true, scratch, threads);
    }
}

// ---- NVFP4 re-quantisation of the activation (nvfp4_moe.py:20-47) --------------------------------------------------
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// FP32 -> FP8 E4M3 bits (round to nearest even, saturating) and back.
__device__ __forceinline__ uint32_t f32_to_e4m3(float x) {
    uint16_t pair;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(pair) : "f"(0.f), "f"(x));
    return pair & 0xFFu;
}
__device__ __forceinline__ float e4m3_to_f32(uint32_t bits) {
    uint32_t h2;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(static_cast<uint16_t>(bits)));
    return __half2float(__ushort_as_half(static_cast<unsigned short>(h2 & 0xFFFFu)));
}

// One byte of two E2M1 codes (nearest, ties to the even code, saturating at 6): `lo` in the low nibble.
__device__ __forceinline__ uint32_t e2m1x2(float lo, float hi) {
    uint32_t out;
    asm("{\n.reg .b8 t;\ncvt.rn.satfinite.e2m1x2.f32 t, %1, %2;\ncvt.u32.u8 %0, t;\n}" : "=r"(out) : "f"(hi), "f"(lo));
    return out;
}

__device__ __forceinline__ float gated_activation(float gate, float up, int kind) {
    if (kind == 0) return gate * (1.f / (1.f + __expf(-gate))) * up;  // SwiGLU: g * sigmoid(g) * u
    const float inner = 0.7978845608028654f * (gate + 0.044715f * gate * gate * gate);
    return 0.5f * gate * (1.f + tanhf(inner)) * up;                  // GeGLU with the tanh GELU
}

// GEMM1's epilogue for 16 token rows x 32 tile rows (one warp): activation and NVFP4 re-quantisation. Tile row 2i holds
// gate feature i, row 2i + 1 its up feature, so lanes l and l ^ 1 hold a feature's two halves, each for all 16 rows
// (`r`). They swap half of them: the even lane then has both halves of rows 0-7, the odd lane of rows 8-15, and each
// activation is computed once. The warp's 16 features are one scale block of each row, so a row's block maximum runs over
// the 16 lanes of one parity; the maxima of eight rows are reduced together, every step halving the rows a lane still
// carries, after which each lane holds the maximum of one row and computes that row's scale alone. One row at a time,
// as one chain of shuffles and conversions with everything computed in two lanes, a row took 340 ns and an expert
// with 32 rows 11 us per tile, longer than its weights take to stream.
__device__ __forceinline__ void requantise_chunk(const MoeDev& g, const uint32_t (&r)[16], float g1, float a2i, int lane,
                                                 int rows, int slot, int ft, int quarter) {
    const bool odd = lane & 1;
    float act[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float lower = __uint_as_float(r[j]) * g1, upper = __uint_as_float(r[j + 8]) * g1;
        const float other = __shfl_xor_sync(0xffffffff, odd ? lower : upper, 1);
        act[j] = gated_activation(odd ? other : lower, odd ? upper : other, g.act_kind);
    }
    // Lane bits 4, 3, 2 choose the row each lane ends up with: `mine` = bit 4 * 4 + bit 3 * 2 + bit 2.
    float m4[4], m2[2], amax;
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float lo = fabsf(act[j]), hi = fabsf(act[j + 4]);
        m4[j] = fmaxf(b4 ? hi : lo, __shfl_xor_sync(0xffffffff, b4 ? lo : hi, 16));
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
        m2[j] = fmaxf(b3 ? m4[j + 2] : m4[j], __shfl_xor_sync(0xffffffff, b3 ? m4[j] : m4[j + 2], 8));
    amax = fmaxf(b2 ? m2[1] : m2[0], __shfl_xor_sync(0xffffffff, b2 ? m2[0] : m2[1], 4));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffff, amax, 2));
    const uint32_t sf = f32_to_e4m3(a2i * (amax * rcp_approx(6.f)));
    const float scale = amax != 0.f ? rcp_approx(e4m3_to_f32(sf) * rcp_approx(a2i)) : 0.f;
    const int mine = (lane & 16 ? 4 : 0) + (lane & 8 ? 2 : 0) + (lane & 4 ? 1 : 0) + (odd ? 8 : 0);
    const int groups = g.f_out / 16, half_f = g.f_out / 2;
    if (!(lane & 2) && mine < rows)
        g.as_out[static_cast<size_t>(slot + mine) * groups + ft * 4 + quarter] = static_cast<uint8_t>(sf);
    // Codes: the feature's neighbour (lane ^ 2) has the other nibble of each byte. The even feature's lane assembles the
    // bytes of rows 0-3 of its eight, the odd feature's lane those of rows 4-7.
    const bool second = lane & 2;
    float y[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
        y[j] = act[j] * __shfl_sync(0xffffffff, scale, (lane & 1) | (j & 4 ? 16 : 0) | (j & 2 ? 8 : 0) | (j & 1 ? 4 : 0));
    uint8_t* codes = g.aq_out + ft * 32 + quarter * 8 + (lane >> 2);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float other = __shfl_xor_sync(0xffffffff, second ? y[j] : y[j + 4], 2);
        const uint32_t byte = second ? e2m1x2(other, y[j + 4]) : e2m1x2(y[j], other);
        const int row = (odd ? 8 : 0) + (second ? 4 : 0) + j;
        if (row < rows) codes[static_cast<size_t>(slot + row) * half_f] = static_cast<uint8_t>(byte);
    }
}

// STREAMED: rows come with the weights, k-block by k-block (GEMM1 only: the down-projection takes no K that long).
template <int NR, bool GATE_UP, bool STREAMED>
__global__ void __launch_bounds__(kMoeThreads, 1) moe_kernel(const __grid_constant__ MoeParams<NR> p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const int slot = NR == 1 ? 0 : static_cast<int>(blockIdx.y);
    const MoeDev& g = p.g[slot];
    const CommDev& c = p.c[slot];
    const int warp = uniform(static_cast<int>(threadIdx.x >> 5)), lane = threadIdx.x & 31;
    const int block = static_cast<int>(blockIdx.x), blocks = static_cast<int>(gridDim.x);
    if (c.stamps && threadIdx.x == 0) c.stamps[block * kStampSlots + 7] = globaltimer();

    const int feature_tiles = g.n / kBlockF;
    const int steps = g.f / 64;                  // K = 64 instructions per item
    const int nkb = (steps + kStepsPerBlock - 1) / kStepsPerBlock;
    const int scale_row = g.f / 16;              // bytes of scales per activation row
    const int row_tile = g.rows_cap * 128;       // bytes of one k-block of an entry's rows
    const int rows_bytes = STREAMED ? row_stage_bytes(g.rows_cap) : entry_bytes(g.rows_cap, g.f);

    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    // The ring's codes, then its scale atoms, then the entries' rows: everything the MMAs read swizzled is 1 KB aligned.
    uint8_t* ring_scales = tiles + g.stages * kCodeTileW;
    uint8_t* entry_rows = tiles + g.stages * kStageBytes;
    MoeSmem* sm = reinterpret_cast<MoeSmem*>(entry_rows + (STREAMED ? g.stages : g.buffers) * rows_bytes);

    if (threadIdx.x == 0) {
        for (int i = 0; i < g.stages; ++i) {
            mbar_init(&sm->full[i], STREAMED ? 34 : 1);  // the weights' expect_tx arrival (and the rows', as in a_full)
            mbar_init(&sm->empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sm->a_full[i], 33);  // the TMA producer's expect_tx arrival and the scale loader's 32 lanes
            mbar_init(&sm->a_empty[i], 1);
            mbar_init(&sm->acc_full[i], 1);
            mbar_init(&sm->acc_empty[i], 4);  // one arrival per epilogue warp of the buffer's group
        }
        fence_barrier_init();
        if (!g.w_tiles) tma_prefetch_descriptor(&g.tm_w);
        tma_prefetch_descriptor(&g.tm_a);
    }
    if (warp == 2) tmem_alloc(&sm->tmem_base, kTmemCols);
    // The next kernel of the stream may be set up from now on (its blocks move in as this kernel's blocks leave).
    pdl_launch_dependents();
    if (GATE_UP) {
        // The kernel in front of this one (moe_prepare_kernel) triggers only after it has itself waited for everything
        // before it, so the packed top-k may be read already: the rows of each expert are counted from it here, and the
        // weight stream starts while that kernel is still quantising rows into their slots. The roles that touch the
        // slots wait for it. Four layers of 32 tokens, 256 experts: 274 us waiting first, 262 this way.
        for (int e = threadIdx.x; e < kMaxLocalExperts; e += kMoeThreads) sm->counted[e] = 0;
        __syncthreads();
        const int pairs = g.m * g.top_k;
        for (int first = threadIdx.x; first < pairs; first += 4 * kMoeThreads) {
            int word[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (first + u * kMoeThreads < pairs) word[u] = __ldcg(g.packed + first + u * kMoeThreads);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = first + u * kMoeThreads < pairs ? (word[u] >> 16) - g.lo : -1;
                if (e >= 0 && e < g.e_local) atomicAdd(&sm->counted[e], 1);
            }
        }
        __syncthreads();
    } else {
        // Routing (counts, slots, activations) comes from the previous kernels of the stream: nothing of it may be read
        // before they are complete.
        pdl_wait();
    }
    // Compact list of (expert, block of rows_cap rows) entries that have rows, in expert order.
    {
        const int e = threadIdx.x;
        const int total_rows = e < g.e_local ? min(GATE_UP ? sm->counted[e] : g.counts[g.lo + e], g.m_max) : 0;
        int early = 0;  // the invocation counters, fetched in the same round trip as the counts
        if (!GATE_UP) {
            if (threadIdx.x == 352 && p.fused) early = c.epochs[block];
            if (threadIdx.x == 353) early = g.gen[block];
            if (threadIdx.x == 354 && p.fused) early = comm_failed(c);
        }
        const int nb = (total_rows + g.rows_cap - 1) / g.rows_cap;
        int incl = nb;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffff, incl, o);
            if (lane >= o) incl += up;
        }
        if (warp < 8 && lane == 31) sm->warp_count[warp] = incl;
        tcgen05_fence_before();
        __syncthreads();
        tcgen05_fence_after();
        if (warp < 8) {
            int base = 0;
            for (int wv = 0; wv < warp; ++wv) base += sm->warp_count[wv];
            for (int j = 0; j < nb && base + incl - nb + j < kMaxEntries; ++j) {
                sm->active[base + incl - nb + j] = static_cast<short>(e | (j << 8));
                sm->rows[base + incl - nb + j] = static_cast<short>(min(total_rows - j * g.rows_cap, g.rows_cap));
            }
            if (threadIdx.x == 0) {
                int total = 0;
                for (int wv = 0; wv < 8; ++wv) total += sm->warp_count[wv];
                sm->n_active = min(total, kMaxEntries);
            }
        }
        if (threadIdx.x == 352) sm->epoch = early;
        if (threadIdx.x == 353) sm->gen = early;
        if (threadIdx.x == 354) sm->failed = early;
        __syncthreads();
    }
    if (c.stamps && threadIdx.x == 0) c.stamps[block * kStampSlots + 0] = globaltimer();
    const uint32_t tmem = uniform(sm->tmem_base);
    const int n_items = uniform(sm->n_active) * feature_tiles;
    const long long deadline = globaltimer() + (c.timeout_ns > 0 ? c.timeout_ns : kDefaultTimeoutNs);

    // This CTA's run of items, and its position in it: entry and feature tile advance together.
    struct Cursor {
        int entry, ft;
        __device__ void next(int feature_tiles) {
            if (++ft == feature_tiles) ft = 0, ++entry;
        }
    };
    const int i0 = static_cast<int>(static_cast<long long>(block) * n_items / blocks);
    const int i1 = static_cast<int>(static_cast<long long>(block + 1) * n_items / blocks);
    const int first_entry = i0 / feature_tiles;
    const int last_entry = i1 > i0 ? (i1 - 1) / feature_tiles : first_entry - 1;
    const Cursor start{first_entry, i0 - first_entry * feature_tiles};

    bool bad = false;  // a wait of this thread ran out: its block announces, pushes and stores nothing
    // Warps 0 to 2 run as whole warps on uniform values, one elected lane issuing (see uniform()).
    if (warp == 0) {
        const bool leader = elect_one();
        int st = 0;
        uint32_t phase = 1;  // waiting for parity 1 on a fresh barrier returns at once: the first lap is free
        Cursor at = start;
        for (int i = i0; i < i1; ++i, at.next(feature_tiles)) {
            const int e = uniform(sm->active[at.entry] & 0xFF);
            const size_t tile = static_cast<size_t>(e) * feature_tiles + at.ft;
            const uint8_t* codes = g.w_tiles + tile * nkb * kCodeTileW;
            const uint8_t* scales = g.w_scales + tile * steps * kAtom;
            for (int kb = 0; kb < nkb; ++kb) {
                if (!mbar_wait_warp(&sm->empty[st], phase, deadline)) {
                    if (leader) report(c.status, kErrTimeout, st, kPhasePipeline, 0);
                    i = i1;
                    break;
                }
                const uint32_t scale_bytes = static_cast<uint32_t>(min(kStepsPerBlock, steps - kb * kStepsPerBlock)) * kAtom;
                if (leader) {
                    mbar_expect_tx(&sm->full[st], kCodeTileW + scale_bytes);
                    if (g.w_tiles)  // one contiguous 16 KB run of HBM, already in the swizzled shared-memory order
                        bulk_load(tiles + st * kCodeTileW, codes + kb * kCodeTileW, kCodeTileW, &sm->full[st], kEvictFirst);
                    else
                        tma_load_2d(tiles + st * kCodeTileW, &g.tm_w, &sm->full[st], kb * 128, e * g.n + at.ft * kBlockF,
                                    kEvictFirst);
                    bulk_load(ring_scales + st * kStepsPerBlock * kAtom, scales + kb * kStepsPerBlock * kAtom, scale_bytes,
                              &sm->full[st], kEvictFirst);
                }
                if (++st == g.stages) st = 0, phase ^= 1;
            }
        }
        __syncwarp();
    } else if (warp == 2 || warp == 3) {
        // The entries' rows: codes by TMA (warp 2, one thread), scales by asynchronous copies straight into the atoms
        // (warp 3): atom byte (r % 32) * 16 + (r / 32) * 4 + j of step s holds scale 4 s + j of row r (< 128). A buffer is
        // refilled once the MMAs of the entry it held have completed. Streamed rows go into the ring's stages instead.
        const bool leader = elect_one();
        if (GATE_UP) pdl_wait();  // the slots are filled by the kernel in front
        // K-blocks [kb0, kb0 + kbs) of an entry's rows into `codes` and `atoms`, announced on `bar`.
        auto fetch = [&](int entry, int kb0, int kbs, uint8_t* codes, uint8_t* atoms, uint64_t* bar) {
            const int what = uniform(static_cast<int>(sm->active[entry])), cnt = uniform(static_cast<int>(sm->rows[entry]));
            const int row0 = (what & 0xFF) * g.m_max + (what >> 8) * g.rows_cap;  // first slot of the entry
            if (warp == 2) {
                const int boxes = (cnt + kBoxRows - 1) / kBoxRows;
                if (leader) {
                    mbar_expect_tx(bar, static_cast<uint32_t>(kbs * boxes * kBoxRows * 128));
                    for (int kb = 0; kb < kbs; ++kb)
                        for (int b = 0; b < boxes; ++b)
                            tma_load_2d(codes + kb * row_tile + b * kBoxRows * 128, &g.tm_a, bar, (kb0 + kb) * 128,
                                        row0 + b * kBoxRows, kEvictLast);
                }
            } else {
                const int step0 = kb0 * kStepsPerBlock, count = min(steps - step0, kbs * kStepsPerBlock);
                const uint8_t* from = g.a_scales + static_cast<size_t>(row0) * scale_row + step0 * 4;
                // A warp copies 2^lg rows of 32 / 2^lg steps at a time. The steps of one row all go to one bank (atoms are
                // 512 bytes apart), so as many rows as there are share an instruction. With one row per instruction, 128
                // rows of K = 2048 took longer than their codes: 8 experts of 134 rows, whole call, 54 us and 36 this way;
                // 8 of 256 at hidden 2816 99 and 60; four layers of 256 experts under Zipf routing 215 and 196.
                const int lg = min(5, 32 - __clz(cnt - 1));
                for (int r = lane & ((1 << lg) - 1); r < cnt; r += 1 << lg) {
                    const uint8_t* src = from + static_cast<size_t>(r) * scale_row;
                    uint8_t* dst = atoms + (r % 32) * 16 + (r / 32) * 4;
#pragma unroll 4
                    for (int s2 = lane >> lg; s2 < count; s2 += 32 >> lg) cp_async_4(dst + s2 * kAtom, src + s2 * 4);
                }
                cp_async_arrive(bar);
            }
        };
        int at_ring = 0;
        uint32_t phase = 1;
        if (STREAMED) {
            Cursor at = start;
            for (int i = i0; i < i1; ++i, at.next(feature_tiles)) {
                for (int kb = 0; kb < nkb; ++kb) {
                    if (!mbar_wait_warp(&sm->empty[at_ring], phase, deadline)) {
                        if (leader) report(c.status, kErrTimeout, at_ring, kPhasePipeline, 5);
                        i = i1;
                        break;
                    }
                    uint8_t* rows = entry_rows + at_ring * rows_bytes;
                    fetch(at.entry, kb, 1, rows, rows + row_tile, &sm->full[at_ring]);
                    if (++at_ring == g.stages) at_ring = 0, phase ^= 1;
                }
            }
        } else {
            for (int entry = first_entry; entry <= last_entry; ++entry) {
                if (!mbar_wait_warp(&sm->a_empty[at_ring], phase, deadline)) {
                    if (leader) report(c.status, kErrTimeout, at_ring, kPhasePipeline, 5);
                    break;
                }
                uint8_t* rows = entry_rows + at_ring * rows_bytes;
                fetch(entry, 0, nkb, rows, rows + nkb * row_tile, &sm->a_full[at_ring]);
                if (++at_ring == g.buffers) at_ring = 0, phase ^= 1;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // One lane feeds the tensor pipe.
        const bool leader = elect_one();
        const uint64_t desc_hi = umma_desc_k128(tiles) & 0xFFFFFFFF00000000ull;     // swizzled operand tiles
        const uint64_t sf_hi = utccp_desc(tiles) & 0xFFFFFFFF00000000ull;           // scale atoms
        auto operand = [&](uint32_t address) { return desc_hi | ((address & 0x3FFFF) >> 4); };
        auto atom = [&](uint32_t address) { return sf_hi | ((address & 0x3FFFF) >> 4); };
        const uint32_t ring = smem_u32(tiles), scales = smem_u32(ring_scales), rows0 = smem_u32(entry_rows);
        // Columns of the scales: W2's by ring stage, the entry's rows by row buffer and step, or by ring stage.
        const uint32_t tmem_sfa = tmem + 2 * g.rows_cap, tmem_sfb = tmem_sfa + g.stages * kScaleCols;
        const bool resident = g.resident;
        int st = 0, buf = -1;
        uint32_t phase = 0, a_phase = 1;
        uint32_t rows = 0, row_scales = 0, idesc = 0;
        bool alive = true;
        Cursor at = start;
        for (int i = i0; i < i1 && alive; ++i, at.next(feature_tiles)) {
            const int item = i - i0, acc_buf = item & 1;
            if (item == 0 || at.ft == 0)  // a new entry
                idesc = umma_idesc_nvfp4(kBlockF, (uniform(static_cast<int>(sm->rows[at.entry])) + 15) & ~15);
            if (!STREAMED && (item == 0 || at.ft == 0)) {
                if (leader && buf >= 0) umma_commit(&sm->a_empty[buf]);
                if (++buf == g.buffers) buf = 0;
                if (buf == 0) a_phase ^= 1;
                if (!mbar_wait_warp(&sm->a_full[buf], a_phase, deadline)) {
                    if (leader) report(c.status, kErrTimeout, buf, kPhasePipeline, 6);
                    break;
                }
                fence_proxy_async();  // the scale atoms were written through the generic proxy
                tcgen05_fence_after();
                rows = rows0 + buf * rows_bytes;
                row_scales = tmem_sfb + buf * steps * 4;
                if (resident && leader)
                    for (int s2 = 0; s2 < steps; ++s2)
                        utccp_128x4(row_scales + 4 * s2, atom(rows + nkb * row_tile + s2 * kAtom));
            }
            // The accumulator buffer must have been read out by the epilogue of two items ago.
            if (item >= 2 && !mbar_wait_warp(&sm->acc_empty[acc_buf], ((item >> 1) - 1) & 1, deadline)) {
                if (leader) report(c.status, kErrTimeout, 0, kPhasePipeline, 4);
                break;
            }
            tcgen05_fence_after();
            const uint32_t acc = tmem + acc_buf * g.rows_cap;
            for (int kb = 0; kb < nkb; ++kb) {
                if (!mbar_wait_warp(&sm->full[st], phase, deadline)) {
                    if (leader) report(c.status, kErrTimeout, st, kPhasePipeline, 1);
                    alive = false;
                    break;
                }
                if (STREAMED) fence_proxy_async();  // as for the entry's scale atoms above
                tcgen05_fence_after();
                const uint32_t row_codes = STREAMED ? rows0 + st * rows_bytes : rows + kb * row_tile;
                const uint64_t dw = operand(ring + st * kCodeTileW), da = operand(row_codes);
                const uint64_t fa = atom(scales + st * kStepsPerBlock * kAtom);
                const uint32_t sfa = tmem_sfa + st * kScaleCols;
                const uint32_t sfb = resident ? row_scales + kb * kScaleCols : tmem_sfb + st * kScaleCols;
                const int nsteps = min(kStepsPerBlock, steps - kb * kStepsPerBlock);
                if (leader) {
                    if (!resident) {
                        const uint64_t fb = atom(STREAMED ? row_codes + row_tile : rows + nkb * row_tile + kb * kStepsPerBlock * kAtom);
                        for (int s2 = 0; s2 < nsteps; ++s2) utccp_128x4(sfb + 4 * s2, fb + s2 * (kAtom >> 4));
                    }
                    if (nsteps == kStepsPerBlock) {
#pragma unroll
                        for (int s2 = 0; s2 < kStepsPerBlock; ++s2) utccp_128x4(sfa + 4 * s2, fa + s2 * (kAtom >> 4));
#pragma unroll
                        for (int s2 = 0; s2 < kStepsPerBlock; ++s2)
                            umma_nvfp4(acc, dw + 2 * s2, da + 2 * s2, idesc, sfa + 4 * s2, sfb + 4 * s2, (kb | s2) != 0);
                    } else {
                        for (int s2 = 0; s2 < nsteps; ++s2) utccp_128x4(sfa + 4 * s2, fa + s2 * (kAtom >> 4));
                        for (int s2 = 0; s2 < nsteps; ++s2)
                            umma_nvfp4(acc, dw + 2 * s2, da + 2 * s2, idesc, sfa + 4 * s2, sfb + 4 * s2, (kb | s2) != 0);
                    }
                    umma_commit(&sm->empty[st]);
                }
                if (++st == g.stages) st = 0, phase ^= 1;
            }
            if (alive && leader) umma_commit(&sm->acc_full[acc_buf]);
        }
        __syncwarp();
    } else {
        // Epilogue: lane = output feature of the tile, registers = the entry's rows. Group 0 takes the run's even items,
        // group 1 the odd ones. What it needs from global memory (the expert's scale, the destination rows) changes with
        // the entry only.
        const int quarter = warp & 3, group = (warp - 4) >> 2;
        if (GATE_UP) pdl_wait();  // the slots written below may still be read by the kernels before
        int entry = -1, cnt = 0, slot0 = 0;
        float g2 = 0.f, a2i = 0.f;
        int dest[kMaxRowsCap / 32];  // destination of row 32 q + lane
        Cursor at = start;
        if (group == 1) at.next(feature_tiles);
        for (int i = i0 + group; i < i1; i += 2, at.next(feature_tiles), at.next(feature_tiles)) {
            if (at.entry != entry) {
                entry = at.entry;
                const int what = sm->active[entry], e = what & 0xFF, row0 = (what >> 8) * g.rows_cap;
                cnt = sm->rows[entry];
                g2 = g.g2[e];
                if (GATE_UP) {
                    a2i = g.a2_inv[e];
                    slot0 = e * g.m_max + row0;
                } else {
                    const int* slots = g.amap + static_cast<size_t>(g.lo + e) * g.m_max + row0;
#pragma unroll
                    for (int q = 0; q < kMaxRowsCap / 32; ++q) dest[q] = q * 32 + lane < cnt ? slots[q * 32 + lane] : -1;
                }
            }
            if (!mbar_wait(&sm->acc_full[group], ((i - i0) >> 1) & 1, deadline)) {
                report(c.status, kErrTimeout, 0, kPhasePipeline, 2);
                bad = true;
                break;
            }
            tcgen05_fence_after();
            const int col = at.ft * kBlockF + quarter * 32 + lane;
            const uint32_t acc = tmem + group * g.rows_cap + (static_cast<uint32_t>(quarter * 32) << 16);
#pragma unroll
            for (int chunk = 0; chunk < kMaxRowsCap / 16; ++chunk) {
                if (chunk * 16 >= cnt) break;
                uint32_t r[16];
                tmem_load_16(acc + chunk * 16, r);
                tmem_load_wait();
                if (GATE_UP) {
                    requantise_chunk(g, r, g2, a2i, lane, cnt - chunk * 16, slot0 + chunk * 16, at.ft, quarter);
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const int pair = __shfl_sync(0xffffffff, dest[chunk / 2], (chunk & 1) * 16 + j);
                        if (pair >= 0)
                            g.y[static_cast<size_t>(pair) * g.n + col] = __float2bfloat16_rn(__uint_as_float(r[j]) * g2);
                    }
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm->acc_empty[group]);
        }
    }
    // Every Y row this CTA produced is written; announce it and wait for the rest of the grid (the combine reads rows
    // written by other CTAs). Counters are banked by launch generation as in the BF16 kernel.
    tcgen05_fence_before();
    bad = __syncthreads_or(bad);
    if (c.stamps && threadIdx.x == 0) c.stamps[block * kStampSlots + 4] = globaltimer();
    if (warp == 2) {
        tcgen05_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
    if (GATE_UP) return;  // the activation slots are written; the down-projection launch that follows does the rest
    CommCtx x{};
    if (p.fused) x = comm_begin(c, block, blocks, sm->epoch, sm->failed);
    // The expert list of this CTA's first output row is fetched now, ahead of the wait for the experts' outputs.
    CombineMeta first;
    if (block < g.m) first = combine_meta(g, block, 0);
    {
        const int gen = sm->gen + 1;
        int* counter = g.counters + (gen & 1) * kMaxTiles;
        if (threadIdx.x == 0) {
            if (block == 0) g.counters[((gen + 1) & 1) * kMaxTiles] = 0;
            __threadfence();  // after the block barrier: orders every thread's Y stores before the announce
            // Rows that never came out of the pipeline are not announced: whoever combines them runs out of time in turn.
            if (!bad) atomicAdd(counter, 1);
            // Only CTAs that have output rows to combine need the others' Y rows; polling is paced so that the
            // arrivals of the rest of the grid are not queued behind a storm of loads on the same word.
            while (block < g.m) {
                int seen;
                asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
                if (seen >= blocks) break;
                if (globaltimer() > deadline) {
                    report(c.status, kErrTimeout, 0, kPhasePipeline, 3);
                    bad = true;
                    break;
                }
                __nanosleep(100);
            }
            for (int j = block; j < kEpochSlots; j += blocks) g.gen[j] = gen;
        }
        bad = __syncthreads_or(bad);
    }
    if (c.stamps && threadIdx.x == 0) c.stamps[block * kStampSlots + 5] = globaltimer();
    // Combine: out[row] = bf16(sum over k in list order of w_k * y_k), experts of other ranks contribute 0 * 0.
    // With one rank the sum over ranks is the identity and the CTA that combines a row is also its owner (rows block,
    // block + blocks, ... in both roles), so the row is finished here and never travels through the receive slots.
    // After a failure, of this launch or of an earlier one of the group, no row is written any more: neither the output
    // nor the residual stream (x.dead is false in an unfused launch, and push_store looks at it itself).
    const bool local_rows = p.fused && c.world == 1;
    const bool write = !bad && !(local_rows && x.dead);
    if (write && local_rows) {
        if (c.mode == kReduce) combine_and_finish<kReduce>(g, c, block, blocks, sm->scratch, first);
        else if (c.mode == kReduceNorm) combine_and_finish<kReduceNorm>(g, c, block, blocks, sm->scratch, first);
        else combine_and_finish<kReduceNormResidual>(g, c, block, blocks, sm->scratch, first);
    } else if (write) {
        const int t = threadIdx.x, threads = g.n / kVec;
        for (int row = block; row < g.m; row += blocks) {
            if (t < threads) {
                const uint4 packed = combine_row(g, row, t, row == block ? first : combine_meta(g, row, 0));
                if (p.fused) {
                    push_store(c, x, row, t * kVec, packed);
                } else {
                    store_v4(g.out + static_cast<size_t>(row) * g.ldo + t * kVec, packed);
                }
            }
        }
    }
    if (p.fused) {
        stamp(c, x, 1);
        if (local_rows) {  // no slot was written: nothing to re-arm, the invocation counters stay where they are
            stamp(c, x, 2);
            stamp(c, x, 3);
        } else {
            rearm_early(c, x);
            own_and_collect(c, x, sm->scratch);  // re-arms late shares between its own and collect phases
            comm_end(c, x);
        }
    }
}

template <int NR, bool GATE_UP, bool STREAMED = false>
static int launch_impl(const MoeParams<NR>& p, dim3 grid, const LaunchOpts& o) {
    int smem = moe_smem_bytes(p.g[0]);
    for (unsigned i = 1; i < grid.y; ++i) smem = max(smem, moe_smem_bytes(p.g[i]));  // emulated ranks may differ in f
    static bool raised[64] = {};
    cudaError_t err = cudaSuccess;
    int dev = 0;
    (void)cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !raised[dev]) {
        err = cudaFuncSetAttribute(moe_kernel<NR, GATE_UP, STREAMED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   kMoeSmemBudget + static_cast<int>(sizeof(MoeSmem)) + 1024);
        raised[dev] = err == cudaSuccess;
    }
    if (err == cudaSuccess) {
        cudaLaunchConfig_t config{};
        config.gridDim = grid;
        config.blockDim = dim3(kMoeThreads);
        config.dynamicSmemBytes = static_cast<size_t>(smem);
        config.stream = o.stream;
        cudaLaunchAttribute attrs[2];
        int n = 0;
        if (o.pdl) {
            attrs[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attrs[n].val.programmaticStreamSerializationAllowed = 1;
            ++n;
        }
        if (o.cooperative) {
            attrs[n].id = cudaLaunchAttributeCooperative;
            attrs[n].val.cooperative = 1;
            ++n;
        }
        config.attrs = attrs;
        config.numAttrs = n;
        err = cudaLaunchKernelEx(&config, moe_kernel<NR, GATE_UP, STREAMED>, p);
    }
    if (err != cudaSuccess) {
        g_last_cuda_error = static_cast<int>(err);
        (void)cudaGetLastError();
        return -6;
    }
    ++g_launches;
    return 0;
}

int launch_moe(const MoeParams<1>& p, int grid, const LaunchOpts& o) { return launch_impl<1, false>(p, dim3(grid), o); }

int launch_moe_gate_up(const MoeParams<1>& p, int grid, const LaunchOpts& o) {
    return p.g[0].buffers > 0 ? launch_impl<1, true>(p, dim3(grid), o) : launch_impl<1, true, true>(p, dim3(grid), o);
}

int launch_moe_loopback(const MoeParams<kMaxWorld>& p, int grid, int nranks, const LaunchOpts& o) {
    return launch_impl<kMaxWorld, false>(p, dim3(grid, nranks), o);
}

}  // namespace dlm
