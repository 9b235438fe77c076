// Dequant-linear for a server's batch of tokens (more than the matrix-vector kernels take, up to 128 rows of
// x; also fewer whose x is too large for those kernels' shared memory) on the stream or the kernel layout of the packed weight:
//   y[M,N] = x[M,K] * W[N,K]^T, replacing F.linear on the dequantized weight (project_quant/modeling.py:629).
//
// At these sizes every weight is decoded once and used for a few dozen tokens, so the work is the decode, not
// the multiply.  The weight tile is therefore the A operand and lives in TENSOR MEMORY: a transcoder thread owns
// one weight row (a TMEM lane), decodes its codes with the byte-permute tables of decode.cuh straight into
// the registers that one tcgen05.st writes, and the tensor core multiplies them with x from shared memory
// (B operand, N = the tokens rounded up to 16).  Nothing of the decoded weight passes through shared memory:
// no swizzled stores, no proxy fences, no operand reads of it.
//
//   warp 0        producer of the packed weight: one TMA box per unit, eight chunks of 1152 contiguous bytes (kernel
//                 layout: one box of 128 rows x 64 bytes of codes, swizzled; the scale bytes come through the L1)
//   warp 1        producer of x: one box of tokens x 2 x 64 K per unit (128-byte swizzle)
//   warp 2        TMEM allocation; one lane issues tcgen05.mma (128 weight rows x tokens x 16)
//   warps 4-7     epilogue: accumulators -> y
//   warps 8-23    transcoders: four groups of four warps, group g takes every fourth unit
//
// A unit is 128 weight rows x 128 K.  Work split: a cluster of c CTAs takes a contiguous range of 128-row
// tiles (over up to three weights that share x), and the range's units are cut into c equal contiguous
// runs.  A tile inside one run is stored directly; the partial sums of a tile that runs cut stay in TMEM to the
// end, then go to shared memory (free by then) and are added in rank order over distributed shared memory by the
// CTAs that share the tile (a fixed order: results are deterministic).  No workspace, one launch.
// Every mbarrier wait is bounded and reports through the caller's status word.
//
// Bank conflicts: a thread reads its row's 64 bytes of codes in 16-byte pieces, and rows are 64 bytes apart, so
// consecutive rows would share two of the eight 16-byte units of a bank line.  The chunks therefore sit 1168 bytes apart
// (16 modulo 128; the box is 16 bytes wider than a chunk and the tensor map ends with the chunk, so the copy engine
// writes zeros there), and a warp's lanes take 8 rows of 4 chunks: a quarter-warp reads 2 rows of 4 chunks, eight units.
// The kernel layout's box has no room between chunks: with the 64-byte swizzle (16-byte piece p of row r lies at p ^ (r / 2
// mod 4)) and a row per lane in order a quarter-warp's eight rows cover the eight units as well (4096 x 4096, 48 tokens:
// 14.8 -> 13.8 us; unswizzled it took longer alone than the 128-row tiles, 13.7 us).
//
// The single-warp roles set the pace unless they are lean: measured on gate + up (28672 x 4096, 48 tokens), integer
// divisions in their loops 66 us whatever the decode did, running counters 39 us, one barrier, one box and
// predicated (not branched) issue per unit 30 us, two more A stages 28 us.

#include <string.h>

#include <mutex>

#include "common.cuh"
#include "decode.cuh"
#include "gemm_small.cuh"
#include "gemv_common.cuh"
#include "tcgen05.cuh"

namespace mixfp4 {
namespace {

constexpr int kMaxSegS = 3;
constexpr int kGroups = 4;                          // transcoder groups of four warps
constexpr int kFirstTranscoder = 8;                 // warp index
constexpr int kThreadsS = (kFirstTranscoder + 4 * kGroups) * 32;
constexpr int kTileRows = 128, kUnitK = 128, kMaxCluster = 8;
constexpr int kTileChunks = kTileRows / (int)kChunkRows;
constexpr uint32_t kSlotBytes = kChunkBytes + 16, kUnitBytes = kTileChunks * kSlotBytes;
constexpr int kMaxWStages = 8, kUnitStages = 4;
constexpr uint32_t kTmemColsS = 512;

struct SmallSegment {
    const uint8_t* scales;                          // kernel layout only: [n, kpad / 16]
    const uint4* lut;                               // optional prebuilt decode table
    const float* global_scale;
    void* y;
    int64_t ldy;
    int n;
    int tile_end;                                   // first tile index after this segment's tiles
};
// floor(n r / cluster) = quot r + floor(rem r / cluster) for the n units of a cluster's range
struct RunSplit {
    int quot, rem;
};
struct SmallArgs {
    SmallSegment seg[kMaxSegS];
    int m, np;                                      // tokens, tokens rounded up to 16
    int units;                                      // units along K (kpad / 128)
    int nseg, cluster, out_dtype;
    int per_cluster, extra;                         // tiles per cluster; the first `extra` clusters take one more
    RunSplit split, split_more;
    uint32_t inv_cluster, inv_units;                // 2^16 / cluster (rounded up), 2^32 / units (rounded down)
    int d_cols;                                     // TMEM columns of an accumulator: np rounded up to 32
    int chains;                                     // accumulators per piece (1, 2 or 4), units in turn: see gemm_small
    int slots;                                      // sums of cut tiles kept apart from the rings: 0, 1 or 2
    uint32_t part[2];                               // where they are in the end: a run's first piece, its last one behind others
    int flush;                                      // 0, or units after which a piece's accumulators are added to its sums
    int sum_cols;                                   // flush with more than 16 tokens: TMEM columns of the sums (16: registers)
    int sets;                                       // sets of accumulators: 3, or 2 when no piece has to stay in TMEM
    int a_stages;                                   // A stages (units, with their x): 4, or 2 when the accumulators need the columns
    int x_pair;                                     // x comes in boxes of 2 x 64 K (K a multiple of 64), else one by one
    int w_stages, lut_shift;                        // weight stages (a power of two); 2^lut_shift copies of the decode table
    int* status;
    uint64_t wait_ns;                               // limit of a wait
};
struct SmallMaps {
    CUtensorMap x;
    CUtensorMap w[kMaxSegS];
};
// Weight row (inside a tile) of lane `lane` of the warps that own TMEM lanes 32 q .. 32 q + 31.
template <bool kStream>
__device__ __forceinline__ int tile_row(int q, int lane) {
    return kStream ? (4 * (q >> 1) + (lane & 3)) * 16 + 8 * (q & 1) + (lane >> 2) : q * 32 + lane;
}

// shared-memory map (offsets from a 1024-aligned base)
struct SmallLayout {
    uint32_t x, codes, lut, parts, bars, misc, bytes;
};
__host__ __device__ inline SmallLayout small_layout(int np, int nseg, int w_stages, int a_stages, int lut_shift, int slots) {
    SmallLayout l;
    l.x = 0;
    l.codes = l.x + (uint32_t)a_stages * np * 256;
    l.lut = l.codes + (uint32_t)w_stages * kUnitBytes;
    l.parts = l.lut + (uint32_t)nseg * (4096u << lut_shift);
    l.bars = l.parts + (uint32_t)slots * np * kTileRows * 4u;                  // sums of cut tiles; without slots the rings take them
    l.misc = l.bars + (2 * kMaxWStages + 2 * kUnitStages + 6) * 8;
    l.bytes = l.misc + 16 + 16 + 1024;                   // + alignment slack
    return l;
}

// One lane of the converged warp (always the same).
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p;
}
// The issuing instructions take the elected lane as a predicate instead of a branch: the code around them stays
// uniform and their operands in uniform registers.
__device__ __forceinline__ void expect_if(uint32_t lead, uint32_t bar, uint32_t bytes) {
    asm volatile(
        "{\n\t.reg .pred l;\n\tsetp.ne.u32 l, %0, 0;\n\t"
        "@l mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %2;\n\t}"
        ::"r"(lead), "r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_2d_if(uint32_t lead, uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile(
        "{\n\t.reg .pred l;\n\tsetp.ne.u32 l, %0, 0;\n\t"
        "@l cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%1], [%2, {%4, %5}], [%3];\n\t}"
        ::"r"(lead), "r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma_load_3d_if(uint32_t lead, uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
    asm volatile(
        "{\n\t.reg .pred l;\n\tsetp.ne.u32 l, %0, 0;\n\t"
        "@l cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%1], [%2, {%4, %5, %6}], [%3];\n\t}"
        ::"r"(lead), "r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc], bf16 inputs, fp32 accumulate.
__device__ __forceinline__ void umma_ts_bf16_if(uint32_t lead, uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                                uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, l;\n\t"
        "setp.ne.b32 p, %5, 0;\n\tsetp.ne.u32 l, %0, 0;\n\t"
        "@l tcgen05.mma.cta_group::1.kind::f16 [%1], [%2], %3, %4, p;\n\t}"
        ::"r"(lead), "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit_if(uint32_t lead, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred l;\n\tsetp.ne.u32 l, %0, 0;\n\t"
        "@l tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%1];\n\t}"
        ::"r"(lead), "r"(bar) : "memory");
}
// thread i of the warp writes lane base+i, 32 columns
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
        ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
          "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
          "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, float (&r)[16]) {
    uint32_t v[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) r[i] = __uint_as_float(v[i]);
}
// thread i of the warp writes lane base+i, 16 columns (no wait: tcgen05.wait::st before they are read)
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const float (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
        ::"r"(__float_as_uint(r[0])), "r"(__float_as_uint(r[1])), "r"(__float_as_uint(r[2])), "r"(__float_as_uint(r[3])),
          "r"(__float_as_uint(r[4])), "r"(__float_as_uint(r[5])), "r"(__float_as_uint(r[6])), "r"(__float_as_uint(r[7])),
          "r"(__float_as_uint(r[8])), "r"(__float_as_uint(r[9])), "r"(__float_as_uint(r[10])), "r"(__float_as_uint(r[11])),
          "r"(__float_as_uint(r[12])), "r"(__float_as_uint(r[13])), "r"(__float_as_uint(r[14])), "r"(__float_as_uint(r[15])),
          "r"(taddr)
        : "memory");
}
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, uint32_t rank) {      // the same offset in a CTA of the cluster
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    return remote;
}
__device__ __forceinline__ float4 ld_peer_f32x4(uint32_t remote) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
    return v;
}
// End of the kernel before (nothing to wait for without a dependent launch).  Every role comes here before the first wait
// that x can hold up, so that the time limit of its waits does not run while that kernel does.
__device__ __forceinline__ void wait_previous_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// A millisecond.
__device__ __noinline__ void let_copies_land() {
    const uint64_t t_0 = global_timer_ns();
    while (global_timer_ns() - t_0 < 1000000ull) {}
    __syncthreads();
}
// Wait of a whole warp: the vote makes the result (and what is computed from it) provably uniform, so the loops of
// the single-warp roles run on the uniform datapath, where TMA and MMA instructions take their operands from.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, const WaitCtx& ctx, int code) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    return __all_sync(0xffffffffu, mbar_wait_call(bar, parity, ctx, code));
}
__device__ __forceinline__ void store_y(const SmallSegment& s, int out_dtype, int64_t token, int row, float v) {
    if (out_dtype == MIXFP4_F32) static_cast<float*>(s.y)[token * s.ldy + row] = v;
    else static_cast<__nv_bfloat16*>(s.y)[token * s.ldy + row] = __float2bfloat16_rn(v);
}

// kStream: the weights are in the stream layout, else in the kernel layout.  kSums: pieces are flushed into sums in TMEM (a
// kernel of its own: as one kernel the other form spilled; 28672 x 4096 at 48 tokens 26.9 us as one, 26.6 as two, 4096 x 4096
// at 128 tokens 15.4 and 15.0).
template <bool kStream, bool kSums>
__global__ void __launch_bounds__(kThreadsS, 1) gemm_small_kernel(const __grid_constant__ SmallMaps maps,
                                                                  const __grid_constant__ SmallArgs a) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;            // the same offset in every CTA of the cluster
    uint8_t* gen = smem_raw + (base - raw);
    const SmallLayout L = small_layout(a.np, a.nseg, a.w_stages, a.a_stages, a.lut_shift, a.slots);

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // provably warp-uniform
    const int S = a.units, np = a.np;
    constexpr uint32_t kStageBytes = kStream ? kUnitBytes : kTileChunks * kChunkCodeBytes;

    // the cluster's tiles and this CTA's run of their units (the quotients come from the host: an integer division
    // costs more here than anything else before the first load)
    int cl;
    asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(cl));
    const int rank = (int)cluster_ctarank();
    const bool more = cl < a.extra;                          // the first clusters take one tile more
    const int t0 = cl * a.per_cluster + min(cl, a.extra);
    const RunSplit split = more ? a.split_more : a.split;
    auto run_start = [&](int r) { return split.quot * r + (int)(((uint32_t)(split.rem * r) * a.inv_cluster) >> 16); };
    const int ua = run_start(rank), ub = run_start(rank + 1), cnt = ub - ua;
    auto div_units = [&](int u) {                            // u / S
        int q = (int)__umulhi((uint32_t)u, a.inv_units);
        while (q * S > u) --q;
        while ((q + 1) * S <= u) ++q;
        return q;
    };
    const uint32_t w_mask = (uint32_t)a.w_stages - 1;        // a power of two

    auto seg_of = [&](int tile) { return (tile >= a.seg[0].tile_end) + (tile >= a.seg[1].tile_end); };
    auto seg_first = [&](int s) { return s == 0 ? 0 : a.seg[s - 1].tile_end; };

    const uint32_t bars = base + L.bars;
    auto full_w = [&](int s) { return bars + 8u * s; };
    auto empty_w = [&](int s) { return bars + 8u * (kMaxWStages + s); };
    auto full_a = [&](int s) { return bars + 8u * (2 * kMaxWStages + s); };
    auto empty_a = [&](int s) { return bars + 8u * (2 * kMaxWStages + kUnitStages + s); };
    auto full_d = [&](int s) { return bars + 8u * (2 * kMaxWStages + 2 * kUnitStages + s); };
    auto empty_d = [&](int s) { return bars + 8u * (2 * kMaxWStages + 2 * kUnitStages + 3 + s); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + L.misc);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + L.misc + 4);
    volatile int* sharer = reinterpret_cast<volatile int*>(gen + L.misc + 16);     // first and last CTA of the run's cut tiles
    const WaitCtx ctx{abort_flag, a.status, a.wait_ns};

    // The next kernel in the stream may set itself up from here on; it waits for this grid's end before it
    // reads this one's outputs.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (warp == 0) {
        if (elect_one()) {
            for (int s = 0; s < kMaxWStages; ++s) { mbar_init(full_w(s), 1); mbar_init(empty_w(s), 4); }
            *abort_flag = 0;                     // both producers write it: neither waits for the other's set-up
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            fence_async_proxy();
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            for (int s = 0; s < kUnitStages; ++s) { mbar_init(full_a(s), 5); mbar_init(empty_a(s), 1); }
            for (int s = 0; s < 3; ++s) { mbar_init(full_d(s), 1); mbar_init(empty_d(s), 4); }
            *abort_flag = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            fence_async_proxy();
        }
        __syncwarp();
    } else if (warp == 2) {
        tmem_alloc(base + L.misc, kTmemColsS);
    }

    // The roles below walk over the run's units with running counters: an integer division costs a lone warp more
    // time than a unit's share of the decode.
    const int tile_first = div_units(ua), sub_first = ua - tile_first * S;      // first tile inside the cluster's range, unit in it

    const uint32_t lead = elect_one();               // the lane that issues for a single-warp role
    int w_issued = 0, w_sub = sub_first, w_tile = t0 + tile_first, w_seg = seg_of(w_tile);
    int w_row = (w_tile - seg_first(w_seg)) * kTileChunks;             // row tile of 16 inside the segment
    uint32_t w_stage = 0;
    auto load_w = [&]() {
        const uint32_t dst = base + L.codes + w_stage * kStageBytes;
        if constexpr (kStream) {
            expect_if(lead, full_w(w_stage), kUnitBytes);
            tma_load_3d_if(lead, dst, &maps.w[w_seg], full_w(w_stage), 0, w_sub, w_row);
        } else {
            expect_if(lead, full_w(w_stage), kTileChunks * kChunkCodeBytes);
            tma_load_2d_if(lead, dst, &maps.w[w_seg], full_w(w_stage), w_sub * (kUnitK / 2), w_row * (int)kChunkRows);
        }
        w_stage = (w_stage + 1) & w_mask;
        ++w_issued;
        if (++w_sub == S) {
            w_sub = 0;
            w_row += kTileChunks;
            if (++w_tile == a.seg[w_seg].tile_end) { ++w_seg; w_row = 0; }
        }
    };
    // the (format, scale) -> magnitudes tables of the segments this run touches, 2^lut_shift copies of every
    // entry: with eight, a quarter-warp's look-ups never share a bank.  Two threads per entry.
    if (warp >= kFirstTranscoder) {
        const int e = (threadIdx.x - kFirstTranscoder * 32) >> 1, half = threadIdx.x & 1;
        const int s_lo = seg_of(t0 + tile_first), s_hi = seg_of(t0 + div_units(ub - 1));
        for (int sg = s_lo; sg <= s_hi; ++sg) {
            uint4* dst = reinterpret_cast<uint4*>(gen + L.lut + (uint32_t)sg * (4096u << a.lut_shift)) + ((uint32_t)e << a.lut_shift);
            const uint4 v = a.seg[sg].lut ? __ldg(a.seg[sg].lut + e) : make_lut_entry(e & 127, e >> 7, *a.seg[sg].global_scale);
            for (int c = half; c < 1 << a.lut_shift; c += 2) dst[c] = v;
        }
    }
    // The producers need nothing from the other warps: they arrive and go on.
    tcgen05_fence_before();
    if (warp < 2) asm volatile("barrier.cta.arrive 1, %0;" ::"n"(kThreadsS) : "memory");
    else asm volatile("barrier.cta.sync 1, %0;" ::"n"(kThreadsS) : "memory");
    tcgen05_fence_after();
    const uint32_t tmem_base = warp < 2 ? 0u : __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const uint32_t d_cols = (uint32_t)a.d_cols;               // TMEM: sets of accumulators | sums (flush) | A stages
    const uint32_t sum_base = tmem_base + a.sets * a.chains * d_cols, a_base = sum_base + a.sum_cols;
    // accumulator set of a run's piece p and how often it has been used before: two sets in turn, or three, where the
    // first piece may be a cut tile that has to stay in its own
    auto d_of = [&](int p) { return a.sets == 2 ? p & 1 : p == 0 ? 0 : 1 + ((p - 1) & 1); };
    auto d_use = [&](int p) { return a.sets == 2 ? p >> 1 : p == 0 ? 0 : (p - 1) >> 1; };
    const int npieces = div_units(ub - 1) - tile_first + 1;
    auto piece_whole = [&](int p) {
        const int tile = tile_first + p;
        return tile * S >= ua && (tile + 1) * S <= ub;
    };
    // 16 tokens of a finished piece: its accumulators added up (a short piece does not use all of them)
    auto load_piece = [&](int p, int c, float (&v)[16]) {
        const int lo = (tile_first + p) * S, len = min(lo + S, ub) - max(lo, ua);
        const uint32_t src = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(d_of(p) * a.chains) * d_cols + c;
        tmem_ld_32x16(src, v);
        for (int i = 1; i < min(a.chains, len); ++i) {
            float w[16];
            tmem_ld_32x16(src + i * d_cols, w);
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] += w[j];
        }
    };

    // Unit u uses A / x stage u modulo a_stages and barrier pair u modulo 4 (its transcoder group's own); the stage is
    // free once the MMAs of unit u - a_stages are done.
    auto wait_stage = [&](int u) {
        return a.a_stages == 4 ? warp_wait(empty_a(u & 3), ((u >> 2) & 1) ^ 1, ctx, 5)
                               : (u < 2 || warp_wait(empty_a((u - 2) & 3), ((u - 2) >> 2) & 1, ctx, 5));
    };

    if (warp == 0) {
        bool ok = true;
        uint32_t parity = 1;                                        // of the stage's last release
        while (w_issued < cnt && ok) {
            if (w_stage == 0 && w_issued > 0) parity ^= 1;
            if (w_issued == a.w_stages) wait_previous_grid();
            if (w_issued >= a.w_stages) ok = warp_wait(empty_w(w_stage), parity, ctx, 7);
            if (ok) load_w();
        }
        // never leave with a copy still writing into this CTA's shared memory
        for (int u = max(0, w_issued - a.w_stages); u < w_issued && ok; ++u) ok = warp_wait(full_w(u & w_mask), (u / a.w_stages) & 1, ctx, 8);
    } else if (warp == 1) {
        // x (and nothing else this kernel reads) may come from the kernel launched just before
        wait_previous_grid();
        asm volatile("fence.proxy.async.global;" ::: "memory");
        const uint32_t box = (uint32_t)np * 128u;
        int sub = sub_first;
        bool ok = true;
        for (int u = 0; u < cnt && ok; ++u) {
            ok = wait_stage(u);
            if (!ok) break;
            const uint32_t bar = full_a(u & 3), dst = base + L.x + (uint32_t)(u & (a.a_stages - 1)) * 2 * box;
            expect_if(lead, bar, 2 * box);
            if (a.x_pair) {
                tma_load_3d_if(lead, dst, &maps.x, bar, 0, 0, 2 * sub);
            } else {
                tma_load_2d_if(lead, dst, &maps.x, bar, sub * kUnitK, 0);
                tma_load_2d_if(lead, dst + box, &maps.x, bar, sub * kUnitK + 64, 0);
            }
            if (++sub == S) sub = 0;
        }
        // copies still in flight: the stages' MMAs wait for them, and the epilogue for the MMAs
    } else if (warp == 2) {
        // kind::f16: D fp32, A and B bf16, both K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(np >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint32_t box16 = (uint32_t)np * 128u >> 4;                   // 64 K of x, in descriptor units
        const uint64_t x_desc0 = make_smem_desc(base + L.x);
        uint32_t d_set = tmem_base;
        int piece = 0, done = 0, left = min(S - sub_first, cnt);    // units of the piece done (since the last flush) and left
        int set = 0, set_par = 1;                                   // flushing: sets in turn
        bool ok = true;
        wait_previous_grid();
        for (int u = 0; u < cnt; ++u) {
            ok = warp_wait(full_a(u & 3), (u >> 2) & 1, ctx, 4);
            if (!ok) break;
            tcgen05_fence_after();
            const uint32_t st = (uint32_t)(u & (a.a_stages - 1));
            const uint32_t a_tmem = a_base + st * 64;
            const uint64_t db = x_desc0 + st * 2 * box16;
            const uint32_t d_tmem = d_set + (uint32_t)(done & (a.chains - 1)) * d_cols, accumulate = done >= a.chains;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                umma_ts_bf16_if(lead, d_tmem, a_tmem + k * 8, db + (k >> 2) * box16 + 2u * (k & 3), idesc, k == 0 ? accumulate : 1u);
            umma_commit_if(lead, empty_a(u & 3));
            ++done;
            --left;
            if (a.flush) {
                if (left == 0 || done == a.flush) {
                    umma_commit_if(lead, full_d(set));
                    if (left == 0) left = min(S, cnt - (u + 1));
                    done = 0;
                    if (++set == a.sets) { set = 0; set_par ^= 1; }
                    d_set = tmem_base + (uint32_t)(set * a.chains) * d_cols;
                    if (u + 1 < cnt && !warp_wait(empty_d(set), set_par, ctx, 10)) break;
                }
            } else if (left == 0) {                                   // the piece is complete; the next one's accumulators
                umma_commit_if(lead, full_d(d_of(piece)));
                ++piece;
                left = min(S, cnt - (u + 1));
                done = 0;
                d_set = tmem_base + (uint32_t)(d_of(piece) * a.chains) * d_cols;
                if (d_use(piece) > 0 && left > 0 && !warp_wait(empty_d(d_of(piece)), (d_use(piece) & 1) ^ 1, ctx, 10)) break;
            }
        }
    } else if (warp == 3) {
        // who shares the tiles that this run's first and last piece are cut from (off everyone's way)
        if (lane < 2) {
            const int lo = (tile_first + (lane == 0 ? 0 : npieces - 1)) * S, hi = lo + S;
            int wf = rank, wl = rank;
            while (run_start(wf) > lo) --wf;
            while (run_start(wl + 1) < hi) ++wl;
            sharer[lane] = wf | (wl << 8) | ((run_start(wf) < lo ? 1 : 0) << 16);
        }
        __syncwarp();
    } else if (warp >= 4 && warp < 8) {
        // epilogue of the tiles this run holds from end to end
        const int q = warp & 3, row = tile_row<kStream>(q, lane);
        int set = 0, par = 0;
        wait_previous_grid();
        for (int p = 0; !kSums && a.flush && p < npieces; ++p) {      // 16 tokens at most: the sums fit in registers
            float sum[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) sum[j] = 0.0f;
            const int lo = (tile_first + p) * S;
            int len = min(lo + S, ub) - max(lo, ua);
            bool ok = true;
            for (; len > 0 && ok; len -= a.flush) {
                ok = warp_wait(full_d(set), par, ctx, 6);
                if (!ok) break;
                tcgen05_fence_after();
                for (int i = 0; i < min(a.chains, len); ++i) {
                    float v[16];
                    tmem_ld_32x16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(set * a.chains + i) * d_cols, v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) sum[j] += v[j];
                }
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(empty_d(set));
                if (++set == a.sets) { set = 0; par ^= 1; }
            }
            if (!ok) break;
            if (piece_whole(p)) {
                const int tile = t0 + tile_first + p, sg = seg_of(tile);
                const SmallSegment& seg = a.seg[sg];
                const int n0 = (tile - seg_first(sg)) * kTileRows + row;
                if (n0 < seg.n)
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (j < a.m) store_y(seg, a.out_dtype, j, n0, sum[j]);
            } else {
                float* part = reinterpret_cast<float*>(gen + a.part[p > 0]) + q * 32 + lane;
#pragma unroll
                for (int j = 0; j < 16; ++j) part[j * kTileRows] = sum[j];
            }
        }
        // more tokens: the sums of a piece longer than the flush interval lie in TMEM between its parts
        for (int p = 0; kSums && p < npieces; ++p) {
            const bool whole = piece_whole(p);
            const int tile = t0 + tile_first + p, sg = seg_of(tile);
            const SmallSegment& seg = a.seg[sg];
            const int n0 = (tile - seg_first(sg)) * kTileRows + row;
            float* part = reinterpret_cast<float*>(gen + a.part[p > 0]) + q * 32 + lane;
            const bool stays = !whole && a.part[p > 0] == 0;        // goes where the rings are: in TMEM until they are free
            const uint32_t lanes = (uint32_t)(q * 32) << 16;
            const int lo = (tile_first + p) * S;
            bool ok = true, first = true;
            for (int len = min(lo + S, ub) - max(lo, ua); len > 0 && ok; len -= a.flush) {
                ok = warp_wait(full_d(set), par, ctx, 6);
                if (!ok) break;
                tcgen05_fence_after();
                const bool last = len <= a.flush;
#pragma unroll 1
                for (int c = 0; c < np; c += 16) {
                    float v[16];
                    tmem_ld_32x16(tmem_base + lanes + (uint32_t)set * d_cols + c, v);
                    if (!first) {
                        float w[16];
                        tmem_ld_32x16(sum_base + lanes + c, w);
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] += w[j];
                    }
                    if (!last || stays) {
                        tmem_st_32x16(sum_base + lanes + c, v);
                    } else if (!whole) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) part[(c + j) * kTileRows] = v[j];
                    } else if (n0 < seg.n) {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (c + j < a.m) store_y(seg, a.out_dtype, c + j, n0, v[j]);
                    }
                }
                if (!last || stays) asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                first = false;
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(empty_d(set));
                if (++set == a.sets) { set = 0; par ^= 1; }
            }
            if (!ok) break;
        }
        for (int p = 0; !kSums && !a.flush && p < npieces; ++p) {
            const int d = d_of(p);
            if (!warp_wait(full_d(d), d_use(p) & 1, ctx, 6)) break;
            const bool whole = piece_whole(p);
            if (!whole && a.slots == 0) continue;                   // stays in TMEM to the end
            tcgen05_fence_after();
            const int tile = t0 + tile_first + p, sg = seg_of(tile);
            const SmallSegment& seg = a.seg[sg];
            const int n0 = (tile - seg_first(sg)) * kTileRows + row;
            for (int c = 0; c < np; c += 16) {
                float v[16];
                load_piece(p, c, v);
                if (!whole) {                                       // a cluster of two: one cut tile per run
                    float* part = reinterpret_cast<float*>(gen + a.part[p > 0]) + c * kTileRows + q * 32 + lane;
#pragma unroll
                    for (int j = 0; j < 16; ++j) part[j * kTileRows] = v[j];
                } else if (n0 < seg.n) {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (c + j < a.m) store_y(seg, a.out_dtype, c + j, n0, v[j]);
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(empty_d(d));
        }
    } else if (warp >= kFirstTranscoder) {
        const int g = (warp - kFirstTranscoder) >> 2, q = warp & 3, row = tile_row<kStream>(q, lane);
        const uint32_t slot_row = (uint32_t)(row >> 4) * (kStream ? kSlotBytes : kChunkCodeBytes);
        const uint32_t spread = kStream ? 0u : ((row >> 1) & 3) * 16;        // 64-byte swizzle of the kernel layout's box
        const uint32_t lut_lane = base + L.lut + (lane & ((1 << a.lut_shift) - 1)) * 16;
        const uint32_t row_lane = (uint32_t)(q * 32) << 16;
        bool ok = true;
        const int w_shift = 31 - __clz(a.w_stages), u_held = g < a.a_stages ? g + kGroups : g;   // first unit whose stage x can hold up
        int tile = t0 + tile_first, sub = sub_first + g;            // of this group's unit
        // kernel layout: the row's eight scale bytes of a unit, fetched while the group's unit before is decoded
        auto fetch_scales = [&](int t, int u_k) {
            while (u_k >= S) { u_k -= S; ++t; }
            const int sg = seg_of(t), r = min((t - seg_first(sg)) * kTileRows + row, a.seg[sg].n - 1);
            return __ldg(reinterpret_cast<const uint2*>(a.seg[sg].scales + ((size_t)r * S + u_k) * (kUnitK / 16)));
        };
        uint2 next = make_uint2(0u, 0u);
        if (!kStream && g < cnt) next = fetch_scales(tile, sub);
        for (int u = g; u < cnt; u += kGroups) {
            const int ws = u & w_mask;
            while (sub >= S) { sub -= S; ++tile; }
            ok = warp_wait(full_w(ws), (u >> w_shift) & 1, ctx, 9);
            if (!ok) break;
            const uint32_t src = base + L.codes + ws * kStageBytes + slot_row;
            uint4 w[4];
#pragma unroll
            for (int p = 0; p < 4; ++p) w[p] = lds128_lut(src + (row & 15) * 64 + ((p * 16) ^ spread));
            uint32_t sc[2];
            if constexpr (kStream) {
                asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(sc[0]), "=r"(sc[1]) : "r"(src + kChunkCodeBytes + (row & 15) * 8));
            } else {
                sc[0] = next.x;
                sc[1] = next.y;
                if (u + kGroups < cnt) next = fetch_scales(tile, sub + kGroups);
            }
            const uint32_t lut_seg = lut_lane + (uint32_t)seg_of(tile) * (4096u << a.lut_shift);
            sub += kGroups;
#pragma unroll
            for (int h = 0; h < 2; ++h) {                           // 64 K elements: 32 TMEM columns
                uint32_t out[32];
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const uint4 tab = lds128_lut(lut_seg + (((sc[h] >> (8 * b)) & 0xffu) << (4 + a.lut_shift)));
                    const uint4 wv = w[2 * h + (b >> 1)];
                    uint32_t p0[4], p1[4];
                    decode8_kl((b & 1) ? wv.z : wv.x, tab, p0);
                    decode8_kl((b & 1) ? wv.w : wv.y, tab, p1);
#pragma unroll
                    for (int j = 0; j < 4; ++j) { out[8 * b + j] = p0[j]; out[8 * b + 4 + j] = p1[j]; }
                }
                if (h == 0) {
                    if (u == u_held) wait_previous_grid();
                    ok = wait_stage(u);
                    if (!ok) break;
                    tcgen05_fence_after();                          // the MMAs that read this stage are done
                }
                tmem_st_32x32(a_base + row_lane + (u & (a.a_stages - 1)) * 64 + h * 32, out);
            }
            if (!ok) break;
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) {
                // released only here, where every word has been used: an arrive right behind the loads was seen to
                // overtake them (rows of a later unit in a few lanes, about one launch in ten)
                mbar_arrive(empty_w(ws));
                mbar_arrive(full_a(g));
            }
        }
    }

    // Every role has stopped issuing.  Without an expired wait all copies have landed and all MMAs are done; after one, copies and
    // MMAs may be in flight whoever gave up, and nothing tells when the last has ended (a role that stopped leaves barriers
    // short of arrivals).  They get a millisecond, hundreds of times what a unit takes, before shared memory is written again,
    // tensor memory is freed or the CTA leaves: a bounded wait, not a proof, and the status word is set by then.
    tcgen05_fence_before();
    __syncthreads();
    if (*abort_flag) let_copies_land();              // (the same for all threads: nobody waits with a limit after the barrier)
    if (a.cluster > 1) {
        // Tiles cut by run boundaries.  The rings are free (the epilogue warps have waited for every piece's MMAs):
        // [token][TMEM lane] fp32 at part[0] (first piece) and part[1] (last).
        // (Sums that have slots are there already.)
        const int tl_index = (warp & 3) * 32 + lane;
        if ((kSums ? a.part[1] == 0 : a.slots == 0) && warp >= 4 && warp < 8) {
            tcgen05_fence_after();
            for (int i = kSums ? 1 : 0; i < 2; ++i) {
                const int p = i == 0 ? 0 : npieces - 1;
                if ((i == 1 && npieces == 1) || piece_whole(p)) continue;
                float* part = reinterpret_cast<float*>(gen + a.part[i]) + tl_index;
                for (int c = 0; c < np; c += 16) {
                    float v[16];
                    if (kSums) tmem_ld_32x16(sum_base + ((uint32_t)((warp & 3) * 32) << 16) + c, v);
                    else load_piece(p, c, v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) part[(c + j) * kTileRows] = v[j];
                }
            }
        }
        __syncwarp();
        cluster_sync_all();
        for (int i = 0; i < 2; ++i) {
            const int p = i == 0 ? 0 : npieces - 1;
            if ((i == 1 && npieces == 1) || piece_whole(p)) continue;
            const int packed = sharer[i], wf = packed & 0xff, share = ((packed >> 8) & 0xff) - wf + 1;
            const int tile = t0 + tile_first + p, sg = seg_of(tile);
            const SmallSegment& seg = a.seg[sg];
            // a thread adds four neighbouring TMEM lanes (stream layout: rows of four chunks, 16 apart) of a token; warps take tokens in turn
            const int n0 = (tile - seg_first(sg)) * kTileRows + tile_row<kStream>(lane >> 3, (lane & 7) * 4);
            uint32_t src[kMaxCluster];                              // the sharers' copies, in rank order
#pragma unroll
            for (int w2 = 0; w2 < kMaxCluster; ++w2)
                if (w2 < share)
                    src[w2] = peer_addr(base + (uint32_t)lane * 16u + a.part[w2 == 0 && (packed >> 16)], (uint32_t)(wf + w2));
            for (int b = (rank - wf) + share * warp; b < a.m; b += share * (kThreadsS / 32)) {
                float4 v[kMaxCluster];
#pragma unroll
                for (int w2 = 0; w2 < kMaxCluster; ++w2)
                    if (w2 < share) v[w2] = ld_peer_f32x4(src[w2] + (uint32_t)b * (kTileRows * 4u));
                float4 sum = v[0];
#pragma unroll
                for (int w2 = 1; w2 < kMaxCluster; ++w2)
                    if (w2 < share) { sum.x += v[w2].x; sum.y += v[w2].y; sum.z += v[w2].z; sum.w += v[w2].w; }
                if (n0 < seg.n) store_y(seg, a.out_dtype, b, n0, sum.x);
                constexpr int kNext = kStream ? 16 : 1;                 // rows from one TMEM lane to the next
                if (n0 + kNext < seg.n) store_y(seg, a.out_dtype, b, n0 + kNext, sum.y);
                if (n0 + 2 * kNext < seg.n) store_y(seg, a.out_dtype, b, n0 + 2 * kNext, sum.z);
                if (n0 + 3 * kNext < seg.n) store_y(seg, a.out_dtype, b, n0 + 3 * kNext, sum.w);
            }
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        tcgen05_fence_before();
        __syncthreads();
    }
    if (warp == 2) {
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, kTmemColsS);
    }
    // peers read this CTA's partial sums until here
    if (a.cluster > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ------------------------------------------------------------------------- host side
constexpr uint32_t kSmemLimitS = 227 * 1024;
// accumulators per piece where nothing is flushed (three sets of them beside the A stages in 512 TMEM columns)
int small_chains(int np) { return np <= 32 ? 4 : np <= 64 ? 2 : 1; }
constexpr int kMaxDevicesS = 64;

// How many clusters of each size the current device runs at once (one CTA per SM), asked once per device.
int max_clusters(int (&out)[kMaxCluster + 1]) {
    static std::mutex lock;
    static int known[kMaxDevicesS][kMaxCluster + 1];
    static bool have[kMaxDevicesS];
    int dev = 0;
    MIXFP4_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevicesS) return MIXFP4_E_UNSUPPORTED;
    std::lock_guard<std::mutex> guard(lock);
    if (!have[dev]) {
        for (const auto kernel : {gemm_small_kernel<true, false>, gemm_small_kernel<true, true>, gemm_small_kernel<false, false>, gemm_small_kernel<false, true>})
            MIXFP4_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimitS));
        for (int c = 1; c <= kMaxCluster; ++c) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)c);
            cfg.blockDim = dim3(kThreadsS);
            cfg.dynamicSmemBytes = kSmemLimitS;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = (unsigned)c;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, gemm_small_kernel<true, false>, &cfg) != cudaSuccess) {
                (void)cudaGetLastError();                    // a cluster size the device does not take
                n = 0;
            }
            known[dev][c] = n;
        }
        have[dev] = true;
    }
    memcpy(out, known[dev], sizeof(out));
    return MIXFP4_OK;
}

}  // namespace

// Work split: the cluster size with the shortest longest run.  In units (about 0.37 us each), an exchange of partial
// sums costs next to nothing between two CTAs and about nine units among four or more; odd sizes lose SMs and start
// late (28672 x 4096, 48 tokens: 30.5, 30.3, 37.7, 31.4, 32.7, 31.6, 36.4, 33.0 us for 1 to 8 CTAs; 4096 x 14336: 44.5,
// 24.3, 19.9, 17.4, 22.8, 18.0, 22.5, 20.4 us), and are left out.  Nine is too much where every cluster has one tile:
//   runs of at most 2048 K whose CTAs leave the next launch of a chain half of the SMs (2048 x 2048, 48 tokens, clusters of 2
//   and 4: 10.3 and 8.7 us alone, 6.4 and 5.5 us in a chain; with more CTAs the chain loses, 4096 x 2048, 96 tokens: 7.7 and 9.1 us);
//   more than 64 tokens, where clusters of two have two A stages as well (4096 x 4096, 128 tokens: 15.1 and 12.4 us alone, 12.8
//   and 11.6 us in a chain);
//   clusters of four on three quarters of the SMs (3000 x 4096, 17 tokens: 12.6 and 9.6 us alone, 8.4 and 8.1 us in a chain).
// With nine there these took longer alone than the 128-row tiles (9.8 us for the first, 11.0 us for the last).
// One decode step of 48 tokens through the linears of eight 8B-shaped decoder layers: 1358 us with the 128-row tiles of
// gemm_kernel (seven launches and up to seven split-K sums a layer), 511 us with four launches of this kernel.  Launches
// in a chain, 48 tokens: 4096 x 4096 8.9 us, 6144 x 4096 in three weights 10.3 us, 28672 x 4096 in two 26.3 us, 4096 x 14336
// 16.9 us.  The decode's byte permutes keep the ALU busy for 476 cycles of a unit.
//
// chain_limit (products, a multiple of 128): a chain of the tensor core's accumulation is no longer than that.  The longest
// piece of a run is cut by the accumulators it has in turn; where that is not enough its accumulators are flushed
// into sums in TMEM (error against fp64 and time, 128 tokens, without the limit and with it: 4096 x 4096 1.72e-6 -> 7.8e-7,
// 14.7 -> 15.0 us; 8192 x 28672 9.2e-6 -> 4.0e-6, 73.5 -> 73.8 us; 12288 x 14336 9.4e-6 -> 4.4e-6, 45.7 -> 46.5 us).
SmallPlan plan_small(int ntiles, int units, int np, int64_t chain_limit, const int* clusters) {
    SmallPlan best = {0, 0, 0};
    double t_best = 1e300;
    const int chains = small_chains(np), limit = chain_limit > kUnitK ? (int)(chain_limit / kUnitK) : 1;
    for (int c = 1; c <= kMaxCluster && c <= units; c += c == 1 ? 1 : 2) {
        if (clusters[c] < 1) continue;
        const int n = ntiles < clusters[c] ? ntiles : clusters[c];
        const int64_t longest = ((int64_t)((ntiles + n - 1) / n) * units + c - 1) / c;
        const int piece = (int)(longest < units ? longest : units);
        const bool flush = np > 16 && (piece + chains - 1) / chains > limit;
        double exchange = c == 1 ? 0.0 : c == 2 ? 1.0 : 9.0;
        if (c > 2 && ntiles <= n) {                          // a tile per cluster
            if (units <= 16) exchange = c * n <= clusters[2] ? 0.5 * c : 9.0;
            else if (np > 64) exchange = 4.0;
            else if (c == 4 && c * n * 2 <= 3 * clusters[2]) exchange = 7.5;
        }
        const double t = (double)longest + exchange;
        if (t < t_best) { t_best = t; best.cluster = c; best.nclusters = n; best.flush = flush ? limit : 0; }
    }
    return best;
}

int gemm_small(const void* x, int64_t m, int64_t ldx, int64_t k, const mixfp4_gemv_segment* segments, int count,
               bool stream_layout, int out_dtype, int64_t chain_limit, uint64_t wait_ns, bool dependent, int* status,
               cudaStream_t st) {
    if (m < 1 || m > (count > 1 ? kSmallMaxGrouped : kSmallMaxTokens) || count < 1 || count > kMaxSegS) return MIXFP4_E_SHAPE;
    if (!aligned(x, 16) || ldx % 8 != 0) return MIXFP4_E_ALIGN;
    EncodeTiledFn encode = encode_tiled_fn();
    if (!encode) return record_error_text("cuTensorMapEncodeTiled is not available from the driver");
    SmallArgs a = {};
    SmallMaps maps;
    memset(&maps, 0, sizeof(maps));
    a.m = (int)m;
    a.np = (int)((m + 15) / 16 * 16);
    a.nseg = count;
    a.out_dtype = out_dtype;
    a.status = status;
    a.wait_ns = wait_ns;
    const int64_t units = padded_k(k) / kUnitK;
    const cuuint32_t estr[3] = {1, 1, 1};
    int64_t tiles = 0;
    for (int s = 0; s < kMaxSegS; ++s) {
        const mixfp4_gemv_segment& in = segments[s < count ? s : count - 1];
        if (s < count) {
            if (in.n <= 0 || in.ldy < in.n) return MIXFP4_E_SHAPE;
            tiles += (in.n + kTileRows - 1) / kTileRows;
            if (tiles * units > 0x0fffffffLL) return MIXFP4_E_SHAPE;
            uint8_t* codes = const_cast<uint8_t*>(in.codes);
            CUresult made;
            if (stream_layout) {
                // whole chunks as rows of 144 eight-byte elements; the box takes two more, which lie outside the map
                const cuuint64_t dims[3] = {kChunkBytes / 8, (cuuint64_t)units, (cuuint64_t)stream_tiles(in.n)};
                const cuuint64_t strides[2] = {kChunkBytes, (cuuint64_t)units * kChunkBytes};
                const cuuint32_t box[3] = {kSlotBytes / 8, 1, kTileChunks};
                made = encode(&maps.w[s], CU_TENSOR_MAP_DATA_TYPE_INT64, 3, codes, dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            } else {
                const cuuint64_t dims[2] = {(cuuint64_t)units * (kUnitK / 2), (cuuint64_t)in.n}, strides[1] = {(cuuint64_t)units * (kUnitK / 2)};
                const cuuint32_t box[2] = {kUnitK / 2, kTileRows};
                made = encode(&maps.w[s], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, codes, dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            }
            if (made != CUDA_SUCCESS) return record_error_text("cuTensorMapEncodeTiled failed for the packed codes");
        }
        a.seg[s] = SmallSegment{in.scales, static_cast<const uint4*>(in.lut), in.global_scale, in.y, in.ldy, (int)in.n,
                                s < count ? (int)tiles : 0x7fffffff};
    }
    a.units = (int)units;
    {
        // boxes of 64 K elements (one swizzle row) by the tokens; two at a time where K is a multiple of 64
        a.x_pair = k % 64 == 0;
        const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)m}, dims3[3] = {64, (cuuint64_t)m, (cuuint64_t)(k / 64)};
        const cuuint64_t strides[2] = {(cuuint64_t)ldx * 2, 128};
        const cuuint32_t box[3] = {64, (cuuint32_t)a.np, 2};
        if (encode(&maps.x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a.x_pair ? 3 : 2, const_cast<void*>(x), a.x_pair ? dims3 : dims,
                   strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return record_error_text("cuTensorMapEncodeTiled failed");
    }
    int clusters[kMaxCluster + 1];
    if (const int rc = max_clusters(clusters)) return rc;
    const SmallPlan plan = plan_small((int)tiles, a.units, a.np, chain_limit, clusters);
    if (plan.cluster < 1) return MIXFP4_E_UNSUPPORTED;
    a.cluster = plan.cluster;
    a.per_cluster = (int)tiles / plan.nclusters;
    a.extra = (int)tiles - a.per_cluster * plan.nclusters;
    const int n0 = a.per_cluster * a.units, n1 = n0 + a.units;
    a.split = RunSplit{n0 / a.cluster, n0 % a.cluster};
    a.split_more = RunSplit{n1 / a.cluster, n1 % a.cluster};
    a.inv_cluster = 65536u / (uint32_t)a.cluster + 1;
    a.inv_units = a.units == 1 ? 0xffffffffu : (uint32_t)((1ull << 32) / (uint32_t)a.units);
    // TMEM (512 columns): two or three sets of accumulators, the sums of flushed ones, 4 or 2 A stages of 64 columns.  The
    // tensor core's accumulation error grows with the number of products in a chain (7.8e-7 of the result after 1024, 1.7e-6
    // after 2048, 3.6e-6 after 4096, 9.3e-6 after 14336 against fp64), so a piece's units go to as many accumulators in turn
    // as there is room for and the sums are added in fp32.
    a.d_cols = (a.np + 31) / 32 * 32;
    a.chains = plan.flush ? 1 : small_chains(a.np);
    // Up to 16 tokens stand in for matrix-vector kernels that split K finely: chains of 256 products at most, added up in
    // the epilogue warps' registers.  More tokens whose pieces exceed the limit: added up in TMEM.
    a.flush = a.np == 16 ? 2 * a.chains : plan.flush;
    a.sum_cols = plan.flush ? a.d_cols : 0;
    // A run has a cut tile at each end at most, in a cluster of two only at one; sums that leave TMEM as soon as their
    // piece is complete free a set of accumulators for two more A stages (28672 x 4096, 48 tokens: about a tenth).
    // (Beyond 64 tokens shared memory has room for one slot, which only flushing needs: a first piece's sums would be in the
    // way of the next one's; the last piece's stay in TMEM.)
    a.slots = a.cluster == 1 ? 0 : a.flush ? (a.np <= 64 ? 2 : 1) : a.cluster == 2 && a.np <= 64 ? 1 : 0;
    a.sets = a.flush || (a.np <= 64 && a.cluster <= 2) ? 2 : 3;
    a.a_stages = a.sets * a.chains * a.d_cols + a.sum_cols + 4 * 64 <= (int)kTmemColsS ? 4 : 2;
    // shared memory: eight weight stages and eight copies of the tables where they fit
    const int choices[6][2] = {{8, 3}, {8, 2}, {4, 3}, {4, 2}, {4, 1}, {4, 0}};
    for (const auto& c : choices) {
        a.w_stages = c[0];
        a.lut_shift = c[1];
        if (small_layout(a.np, count, a.w_stages, a.a_stages, a.lut_shift, a.slots).bytes <= kSmemLimitS) break;
    }
    const SmallLayout L = small_layout(a.np, count, a.w_stages, a.a_stages, a.lut_shift, a.slots);
    const uint32_t part_bytes = (uint32_t)a.np * kTileRows * 4u;
    a.part[0] = a.slots ? L.parts : 0u;
    a.part[1] = a.slots != 1 ? a.part[0] + part_bytes : a.cluster == 2 ? a.part[0] : 0u;
    // (sums of cut tiles without a slot go where the rings were)
    if (L.bytes > kSmemLimitS || (2 - a.slots) * part_bytes > L.lut) return MIXFP4_E_SHAPE;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(plan.cluster * plan.nclusters));
    cfg.blockDim = dim3(kThreadsS);
    cfg.dynamicSmemBytes = L.bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)a.cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent ? 2 : 1;
    const auto kernel = stream_layout ? (plan.flush ? gemm_small_kernel<true, true> : gemm_small_kernel<true, false>)
                                      : (plan.flush ? gemm_small_kernel<false, true> : gemm_small_kernel<false, false>);
    MIXFP4_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, maps, a));
    return check_launch("gemm_small_kernel");
}

}  // namespace mixfp4

using namespace mixfp4;

extern "C" int mixfp4_gemm_grouped(const void* x, int64_t m, int64_t ldx, int64_t k,
                                   const mixfp4_gemv_segment* segments, int count, int layout, int out_dtype,
                                   int* status, int flags, void* stream) {
    if (layout != MIXFP4_LAYOUT_STREAM) return MIXFP4_E_MODE;
    if (!x || !segments) return MIXFP4_E_NULL;
    if (m <= 0 || m > kSmallMaxGrouped || k <= 0 || k > 0x7fffffffLL || ldx < k || count < 1 || count > kMaxSegS)
        return MIXFP4_E_SHAPE;
    if (out_dtype != MIXFP4_F32 && out_dtype != MIXFP4_BF16) return MIXFP4_E_DTYPE;
    for (int s = 0; s < count; ++s) {
        const mixfp4_gemv_segment& in = segments[s];
        if (!in.codes || !in.global_scale || !in.y) return MIXFP4_E_NULL;
        if (in.n <= 0 || in.n > 0x7fffffffLL || in.ldy < in.n) return MIXFP4_E_SHAPE;
        if (!aligned(in.codes, 16) || (in.lut && !aligned(in.lut, 16))) return MIXFP4_E_ALIGN;
    }
    if (!aligned(x, 16) || ldx % 8 != 0) return MIXFP4_E_ALIGN;
    const bool decode = m <= 16;                       // rows that the decode kernels take: their wait limit, their status word
    if (decode && !status) {
        if (const int rc = stream_status_word(&status)) return rc;
    }
    int64_t chain = INT64_MAX;
    for (int s = 0; s < count; ++s) {
        const int64_t c = gemm_tile_chain(m, segments[s].n, k);
        chain = c < chain ? c : chain;
    }
    return gemm_small(x, m, ldx, k, segments, count, true, out_dtype, chain, decode ? wait_limit_ns() : kWaitLimitNs,
                      (flags & MIXFP4_FLAG_OVERLAP_PREVIOUS) != 0, status, static_cast<cudaStream_t>(stream));
}
