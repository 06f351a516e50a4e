// Stand-alone fused tensor-parallel reduction of a given BF16 partial: push reduce-scatter, rank-ordered FP32 sum
// (+ residual + RMSNorm), multicast all-gather, in-band arrival detection. One launch per call; every CTA pushes its
// share of the partial, re-arms its share of the stale buffers, then owns rows r = block, block + grid, ...
// Replaces reduce_kernel<NORM, RESIDUAL> of the reference (dlmrt/ops/csrc/tp_comm.cu:138-275) bit for bit.
#include "kernels.cuh"

namespace dlm {

int g_last_cuda_error = 0;
long long g_launches = 0;

// NR = 1: one rank per GPU (production). NR = 8: up to eight ranks emulated by one launch on one GPU, rank slot =
// blockIdx.y; the grid is launched cooperatively so that all ranks' CTAs are resident together.
// MAXT: 512 for hidden sizes up to 4096 (blocks of hidden / 8 threads), where the compiler may then use 128 registers
// per thread; 1024 for the rest.
template <int NR, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) reduce_kernel(const __grid_constant__ ReduceParams<NR> p) {
    const int slot = NR == 1 ? 0 : static_cast<int>(blockIdx.y);
    const CommDev& c = p.c[slot];
    __shared__ float scratch[64];
    pdl_launch_dependents();  // the next kernel may be set up while this one runs; it waits before it reads our output
    pdl_wait();
    const CommCtx x = comm_begin(c, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x), c.epochs[blockIdx.x],
                                 comm_failed(c));
    stamp(c, x, 0);
    push_partial(c, x, p.partial[slot]);
    stamp(c, x, 1);
    rearm_early(c, x);
    own_and_collect<(MAXT <= 512)>(c, x, scratch);  // re-arms late shares between its own and collect phases
    comm_end(c, x);
}

// The reduction with one rank: the sum over ranks is the partial itself (added to +0.0f), so nothing travels through the
// receive slots, nothing is polled and nothing re-armed; what is left is a row kernel: residual add, RMSNorm, BF16
// rounding. Bound by memory latency for small blocks and by L2 bandwidth for large ones, so each row is one block (256
// rows of 8192 columns are resident at once, two blocks of 512 threads per SM) and a thread has all its loads in flight
// before it uses the first. VPT: 16-byte vectors per thread, t and t + blockDim.x; the block-wide sum keeps the tree of
// block_sum over the row's n / 8 lanes, so the values are those of the many-rank kernel bit for bit. Against that
// kernel run with one rank: 9.4 -> 4.1 us per [256, 8192] reduction in a graph (16.8 MB through L2).
template <int MODE, int VPT>
__global__ void __launch_bounds__(512) finish_kernel(const __grid_constant__ ReduceParams<1> p) {
    __shared__ float scratch[32];
    const CommDev& c = p.c[0];
    const int t = static_cast<int>(threadIdx.x), warp = t >> 5, lane = t & 31;
    const int vecs = c.n / kVec;
    pdl_launch_dependents();
    pdl_wait();
    if (c.stamps && t == 0) c.stamps[blockIdx.x * kStampSlots] = globaltimer();
    const int failed = comm_failed(c);  // sticky: after a time-out of this group nothing is written any more
    for (int row = static_cast<int>(blockIdx.x); row < c.rows; row += static_cast<int>(gridDim.x)) {
        uint4 raw[VPT], hraw[VPT], wraw[VPT];
        bool active[VPT];
        const size_t base = static_cast<size_t>(row) * c.n;
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            const int vec = t + i * static_cast<int>(blockDim.x);
            active[i] = vec < vecs;
            raw[i] = hraw[i] = wraw[i] = make_uint4(0, 0, 0, 0);
            if (active[i]) {
                raw[i] = *reinterpret_cast<const uint4*>(p.partial[0] + base + vec * kVec);
                if (MODE == kReduceNormResidual) hraw[i] = *reinterpret_cast<const uint4*>(c.h + base + vec * kVec);
                if (MODE != kReduce) wraw[i] = *reinterpret_cast<const uint4*>(c.weight + vec * kVec);
            }
        }
        float v[VPT][kVec] = {};
#pragma unroll
        for (int i = 0; i < VPT; ++i) add_bf16x8(v[i], raw[i]);  // +0.0f + partial: -0.0 becomes +0.0 as in any sum
        if (MODE != kReduce) {
#pragma unroll
            for (int i = 0; i < VPT; ++i) {
                if (MODE == kReduceNormResidual) {
                    add_bf16x8(v[i], hraw[i]);
                    if (active[i] && !failed)
                        store_v4(c.h + base + (t + i * static_cast<int>(blockDim.x)) * kVec, pack_bf16x8(v[i]));
                }
                float ss = 0.f;
#pragma unroll
                for (int j = 0; j < kVec; ++j) ss = fmaf(v[i][j], v[i][j], ss);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffff, ss, o);
                if (lane == 0) scratch[warp + i * static_cast<int>(blockDim.x >> 5)] = ss;
            }
            __syncthreads();
            float ss = lane < (vecs >> 5) ? scratch[lane] : 0.f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffff, ss, o);
            __syncthreads();  // scratch is reused by the next row
            const float rs = rsqrtf(ss / c.n + c.eps) * c.scale;
#pragma unroll
            for (int i = 0; i < VPT; ++i) {
                const __nv_bfloat162* w = reinterpret_cast<const __nv_bfloat162*>(&wraw[i]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 f = __bfloat1622float2(w[j]);
                    v[i][2 * j] = v[i][2 * j] * rs * f.x;
                    v[i][2 * j + 1] = v[i][2 * j + 1] * rs * f.y;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            if (active[i] && !failed) {
                const size_t at = base + (t + i * static_cast<int>(blockDim.x)) * kVec;
                if (c.out_mc) multicast_store(c.out_mc + at, pack_bf16x8(v[i]));
                else store_v4(c.out_peers[0] + at, pack_bf16x8(v[i]));
            }
        }
    }
    if (c.stamps && t == 0) c.stamps[blockIdx.x * kStampSlots + 3] = globaltimer();
}

template <int VPT>
static cudaError_t launch_finish(const ReduceParams<1>& p, const cudaLaunchConfig_t& config) {
    if (p.c[0].mode == kReduce) return cudaLaunchKernelEx(&config, finish_kernel<kReduce, VPT>, p);
    if (p.c[0].mode == kReduceNorm) return cudaLaunchKernelEx(&config, finish_kernel<kReduceNorm, VPT>, p);
    return cudaLaunchKernelEx(&config, finish_kernel<kReduceNormResidual, VPT>, p);
}

// All-gather of a small block of bytes (row statistics and the like) in the same barrier-free style: every rank stores
// its block into slot [e % 3][rank] of every rank's receive buffer (one multimem.st per 16 bytes, or one store per
// rank), re-arms the buffer peers write two invocations from now, and copies each slot into its own OUT
// [world][bytes] as the slot's vectors arrive. A vector has arrived once none of its four 32-bit words is all-ones,
// so the payload may be FP32, FP16 or BF16 values (arithmetic never produces those bit patterns) but not arbitrary
// integers. `c.n` is the block's size in 2-byte units (a multiple of 8), `c.rows` is 1.
template <int NR>
__global__ void __launch_bounds__(256, 1) gather_kernel(const __grid_constant__ ReduceParams<NR> p) {
    const int slot = NR == 1 ? 0 : static_cast<int>(blockIdx.y);
    const CommDev& c = p.c[slot];
    if (NR == 1 && c.world == 1) {  // one rank: its block is the result, no slots in between
        pdl_launch_dependents();
        pdl_wait();
        const int stride = static_cast<int>(gridDim.x * blockDim.x);
        if (!comm_failed(c))
            for (int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x); i < c.n / kVec; i += stride)
                store_v4(c.out + static_cast<size_t>(i) * kVec,
                         *reinterpret_cast<const uint4*>(p.partial[slot] + static_cast<size_t>(i) * kVec));
        return;
    }
    pdl_wait();
    const CommCtx x = comm_begin(c, static_cast<int>(blockIdx.x), static_cast<int>(gridDim.x), c.epochs[blockIdx.x],
                                 comm_failed(c));
    const int vecs = c.n / kVec;
    const int stride = x.blocks * blockDim.x;
    const int first = x.block * blockDim.x + threadIdx.x;
    for (int i = first; i < vecs; i += stride) {
        const uint4 v = *reinterpret_cast<const uint4*>(p.partial[slot] + static_cast<size_t>(i) * kVec);
        push_store(c, x, 0, i * kVec, v);
    }
    rearm(c, x, x.block, x.blocks);
    pdl_launch_dependents();
    const __nv_bfloat16* mine = c.recv[c.rank] + x.buf * x.buf_elems;
    for (int i = first; i < vecs * c.world; i += stride) {  // slot s = i / vecs, vector i % vecs
        const __nv_bfloat16* src = mine + static_cast<size_t>(i) * kVec;
        uint4 v;
        bool ok = !x.dead;
        while (ok) {
            v = load_volatile(src);
            if (v.x != 0xFFFFFFFFu && v.y != 0xFFFFFFFFu && v.z != 0xFFFFFFFFu && v.w != 0xFFFFFFFFu) break;
            if (globaltimer() > x.deadline) {
                report(c.status, kErrTimeout, i / vecs, kPhaseReceive, x.e);
                ok = false;
                break;
            }
        }
        if (ok) store_v4(c.out + static_cast<size_t>(i) * kVec, v);
    }
    comm_end(c, x);
}

template <int NR>
static int launch_gather_impl(const ReduceParams<NR>& p, dim3 grid, const LaunchOpts& o) {
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = dim3(256);
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
    const cudaError_t err = cudaLaunchKernelEx(&config, gather_kernel<NR>, p);
    if (err != cudaSuccess) {
        g_last_cuda_error = static_cast<int>(err);
        (void)cudaGetLastError();
        return -6;
    }
    ++g_launches;
    return 0;
}

int launch_gather(const ReduceParams<1>& p, int grid, const LaunchOpts& o) { return launch_gather_impl<1>(p, dim3(grid), o); }

int launch_gather_loopback(const ReduceParams<kMaxWorld>& p, int grid, int nranks, const LaunchOpts& o) {
    return launch_gather_impl<kMaxWorld>(p, dim3(grid, nranks), o);
}

template <int NR>
static int launch_impl(const ReduceParams<NR>& p, dim3 grid, int threads, const LaunchOpts& o) {
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = dim3(static_cast<unsigned>(threads));
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
    const cudaError_t err = threads <= 512 ? cudaLaunchKernelEx(&config, reduce_kernel<NR, 512>, p)
                                           : cudaLaunchKernelEx(&config, reduce_kernel<NR, 1024>, p);
    if (err != cudaSuccess) {
        g_last_cuda_error = static_cast<int>(err);
        (void)cudaGetLastError();
        return -6;
    }
    ++g_launches;
    return 0;
}

int launch_reduce(const ReduceParams<1>& p, int grid, int threads, const LaunchOpts& o) {
    return launch_impl<1>(p, dim3(grid), threads, o);
}

int launch_reduce_single(const ReduceParams<1>& p, int grid, const LaunchOpts& o) {
    const int vecs = p.c[0].n / kVec;
    const bool two = vecs > 512;  // 512 threads hold the widest row in two vectors each
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(static_cast<unsigned>(grid));
    config.blockDim = dim3(static_cast<unsigned>(two ? (vecs / 2 + 31) / 32 * 32 : vecs));
    config.stream = o.stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &attr;
    config.numAttrs = o.pdl ? 1 : 0;
    const cudaError_t err = two ? launch_finish<2>(p, config) : launch_finish<1>(p, config);
    if (err != cudaSuccess) {
        g_last_cuda_error = static_cast<int>(err);
        (void)cudaGetLastError();
        return -6;
    }
    ++g_launches;
    return 0;
}

int launch_reduce_loopback(const ReduceParams<kMaxWorld>& p, int grid, int nranks, int threads, const LaunchOpts& o) {
    return launch_impl<kMaxWorld>(p, dim3(grid, nranks), threads, o);
}

}  // namespace dlm
