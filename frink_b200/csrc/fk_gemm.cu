// Prefill GEMM over resident quantized weights: int8 tensor-core MMA
// (tcgen05.mma kind::i8, accumulators in tensor memory) on q8_1 activations,
// with the exact per-32-run rescale done by the epilogue warps.
//
//   out[t][r] = sum_kb  dw[r][kb] * dx[t][kb] * ( sum_{k in kb} wq[r][k] * xq[t][k] )   (- Q4_K min term)
//
// The inner sum is an exact int32 (one MMA of K = 32 per run kb), so every
// integer this kernel produces equals the GEMV's and the oracle's.  Because the
// weight scale and the activation scale both change every 32 K, an accumulator
// is drained from tensor memory after every K = 32 step and scaled on the CUDA
// cores; that rescale, not the tensor pipe, bounds this kernel.  Accumulators change hands in groups (half of tensor
// memory at a time), not run by run, and the launch overlaps the quantizer in front of it (programmatic serialization):
// with the weight scales decoded by the unpack warps, 8192 x 3072 Q4_K, M = 512 went from 185 to 135 us.
//
// One CTA = 128 weight rows x BN tokens (128, 64 or 32; gemm_plan), warps with fixed roles (Tile<BN>):
//   epilogue    TMEM -> registers (tcgen05.ld), f32 rescale, store
//   unpack      packed weights (global) -> int8 tile in shared memory
//               (128-byte swizzle, the layout the MMA descriptor names)
//   TMA         activation int8 tile + its scale tiles (and the
//               weight tile itself for Q8_0, whose int8 plane needs no unpacking)
//   MMA issuer  one elected lane, + TMEM allocation
// The CTAs of a cluster may share one tile, each on its own part of K; their f32 sums meet in distributed shared memory.
// Stages (K = 128 each) and TMEM accumulators are rings guarded by mbarriers; every mbarrier wait is bounded and raises
// the context's error word instead of spinning forever.  Two waits have no limit of their own: the cluster barriers of a
// split tile, which every CTA reaches because its mbarrier waits end, and tcgen05.alloc, which never has to wait for a
// CTA that waits for others (see the co-residence asserts below Smem).
#include "fk_common.cuh"

#include <math.h>

#include "fk_tc.cuh"

namespace {
using namespace fk_tc;

#ifdef FK_TRACE
__device__ unsigned long long fk_gemm_trace[4][512];
__device__ __forceinline__ unsigned long long gtime_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
#define GTR(k_, i_, who_) do { if ((who_) && blockIdx.x == 0 && blockIdx.y == 0 && (i_) < 512) fk_gemm_trace[k_][i_] = gtime_ns(); } while (0)
#else
#define GTR(k_, i_, who_) do { } while (0)
#endif

constexpr int BM = 128;           // weight rows per CTA (MMA M)
constexpr int KSTAGE = 128;       // K per pipeline stage (4 MMAs of K = 32)
constexpr int NSTAGE = 4;
// Tile shapes.  BN token columns per CTA; an epilogue warp owns CW of them in one TMEM lane quadrant.
template <int BN> struct Tile {
    static constexpr int CW = BN >= 128 ? 32 : 16;
    static constexpr int EPI_WARPS = BN / CW * 4;
    static constexpr int UNPACK_WARPS = BN >= 128 ? 2 : 4;
    static constexpr int THREADS = (EPI_WARPS + UNPACK_WARPS + 2) * 32;
    static constexpr int BLOCKS = BN >= 64 ? 1 : 2;      // resident per SM: what shared and tensor memory are cut for
    static constexpr int NACC = 512 / BLOCKS / BN;       // TMEM accumulators: two groups, one filled while the other is drained
    static constexpr int GROUP = NACC / 2;               // runs that share one hand-over (a commit, a wait, a release)
};
constexpr int MAX_SPLIT = 8;      // CTAs of a cluster that share one tile, each on its own part of K

struct GemmArgs {
    const uint8_t* w;         // matrix 0 of the weight handle
    size_t mat_stride;
    size_t plane_off[4];
    size_t plane_stride[4];
    int rows, cols;
    int mat;                  // dense: the matrix; grouped: ignored
    const int* tile_expert;   // grouped: expert of each token tile (nullptr = dense)
    const int* n_tiles_dev;   // grouped: number of live token tiles (nullptr = all of gridDim.y)
    const int* out_row;       // padded token row -> output row, -1 = padding (nullptr = dense: row t is token t, padding from m on)
    int m;
    int split;                // CTAs per tile along K (the cluster's size in z)
    float* out;
    int32_t* isums;           // test hook: the raw accumulators, [token][rows][cols / run] (nullptr = off)
    int* err;
};

// Shared memory map (offsets from a 1024-byte aligned base).
template <int BN> struct Smem {
    static constexpr int A_BYTES = BM * KSTAGE;          // 16 KB
    static constexpr int B_BYTES = BN * KSTAGE;
    static constexpr int DX_BYTES = 4 * BN * 4;          // [4 runs][BN] f32
    static constexpr int DW_BYTES = 4 * BM * 4;          // [4 runs][BM] f32: weight scales, then (Q4_K) min scales
    static constexpr int DX = A_BYTES + B_BYTES, DW = DX + 2 * DX_BYTES;
    static constexpr int STAGE = DW + 2 * DW_BYTES;
    static constexpr int BARS = NSTAGE * STAGE;          // barrier block
    static constexpr int USED = BARS + 256 + 1024;       // + alignment slack
    static constexpr int TOTAL = BN == 64 && USED < 128 * 1024 ? 128 * 1024 : USED;   // 64: see below
    static_assert(BM * BN * 4 <= BARS, "the partial sums of a split tile reuse the stages");
};

// A CTA of a split tile waits for its cluster while it holds tensor memory.  Were CTAs of two such grids (two contexts, two
// streams) to meet on two SMs whose tensor memory holds one of them, each could hold what the other's cluster waits for, for
// ever.  So CTAs that share an SM must fit its tensor memory together: what does not fit is kept off by its shared memory
// (the 64-token tile asks for 4 KB more than it uses).  Two 32-token tiles fit both; three fit neither.
constexpr int SM_SMEM = 228 * 1024, CTA_RESERVED = 1024, TMEM_COLS = 512;
template <int A, int B> constexpr bool may_share_an_sm() { return Smem<A>::TOTAL + Smem<B>::TOTAL + 2 * CTA_RESERVED <= SM_SMEM; }
template <int BN> constexpr int tmem_cols() { return Tile<BN>::NACC * BN; }
static_assert(!may_share_an_sm<128, 128>() && !may_share_an_sm<128, 64>() && !may_share_an_sm<128, 32>() && !may_share_an_sm<64, 64>() &&
              !may_share_an_sm<64, 32>(), "their accumulators do not fit one SM's tensor memory");
static_assert(may_share_an_sm<32, 32>() && 2 * tmem_cols<32>() <= TMEM_COLS && 3 * (Smem<32>::TOTAL + CTA_RESERVED) > SM_SMEM, "two 32-token tiles, not three");

// The weight scales of one tile row for one stage (runs kb0 .. kb0 + 3): as loaded, and decoded.  The unpack warps load
// them beside the row they belong to and leave them decoded in the stage, so the epilogue -- the kernel's critical path --
// reads one or two words a run.  (Loaded by every epilogue warp for itself they cost each stage a global-memory latency:
// 340 to 1800 cycles out of 2400 to 7000.)
template <int KIND> struct RawScale {
    uint4 hd;        // Q4_K: d, dmin and the packed scales
    uint2 sc;        // Q8_0: four f16; Q6_K: eight int8 (two per run); MXFP4: four exponents in x
    uint16_t d;      // Q6_K
};
struct StageScale { uint32_t sc, mn; float d, dmin; uint2 raw; };

template <int KIND>
__device__ __forceinline__ void load_wscales(const GemmArgs& a, const uint8_t* wb, int wrow0, int r, int st, bool live, RawScale<KIND>& v) {
    v.hd = make_uint4(0, 0, 0, 0);
    v.sc = make_uint2(0, 0);
    v.d = 0;
    const int kb0 = 4 * st, wrow = wrow0 + (KIND == FK_Q6_K ? r >> 1 : r);
    if (!live || wrow >= a.rows) return;
    if (KIND == FK_Q4_K) {
        v.hd = ldg16(wb + ((size_t)wrow * (a.cols >> 8) + (kb0 >> 3)) * 144);
    } else if (KIND == FK_Q8_0) {
        v.sc = __ldg((const uint2*)(wb + a.plane_off[1] + (size_t)wrow * a.plane_stride[1] + 2 * kb0));   // rows are padded to 16 bytes
    } else if (KIND == FK_MXFP4) {
        v.sc.x = __ldg((const uint32_t*)(wb + a.plane_off[1] + (size_t)wrow * a.plane_stride[1] + kb0));
    } else {
        v.d = __ldg((const uint16_t*)(wb + a.plane_off[3] + (size_t)wrow * a.plane_stride[3]) + (kb0 >> 3));
        v.sc = __ldg((const uint2*)(wb + a.plane_off[2] + (size_t)wrow * a.plane_stride[2] + 2 * kb0));
    }
}
template <int KIND>
__device__ __forceinline__ StageScale stage_scales(const RawScale<KIND>& v, int kb0) {
    StageScale t{};
    if (KIND == FK_Q4_K) {
        t.d = fk_h2f((uint16_t)(v.hd.x & 0xFFFF));
        t.dmin = fk_h2f((uint16_t)(v.hd.x >> 16));
        // 6-bit scales and mins of sub-blocks 0..3 or 4..7, one per byte
        t.sc = (kb0 & 4) ? (v.hd.w & 0x0F0F0F0Fu) | ((v.hd.y >> 2) & 0x30303030u) : v.hd.y & 0x3F3F3F3Fu;
        t.mn = (kb0 & 4) ? ((v.hd.w >> 4) & 0x0F0F0F0Fu) | ((v.hd.z >> 2) & 0x30303030u) : v.hd.z & 0x3F3F3F3Fu;
    } else {
        if (KIND == FK_Q6_K) t.d = fk_h2f(v.d);
        t.raw = v.sc;
    }
    return t;
}
// Scale (and, Q4_K, min scale) of run kb0 + j.
template <int KIND>
__device__ __forceinline__ void run_scale(const StageScale& t, int j, int row, float* dw, float* mw) {
    *mw = 0.0f;
    if (KIND == FK_Q4_K) {
        *dw = t.d * (float)((t.sc >> (8 * j)) & 0xFFu);
        *mw = t.dmin * (float)((t.mn >> (8 * j)) & 0xFFu);
    } else if (KIND == FK_Q8_0) {
        *dw = fk_h2f((uint16_t)((j < 2 ? t.raw.x : t.raw.y) >> (16 * (j & 1))));
    } else if (KIND == FK_MXFP4) {
        *dw = e8m0_half((t.raw.x >> (8 * j)) & 0xFFu);
    } else {
        *dw = t.d * (float)(int8_t)((j < 2 ? t.raw.x : t.raw.y) >> (16 * (j & 1) + 8 * (row & 1)));
    }
}

// Packed bytes of one TILE row for stage `st` (K range [128 st, 128 st + 128)), as loaded (nothing decoded yet, so the
// loads of the next stages can be in flight while this stage is written).  Q6_K: tile row r is half r & 1 of weight row
// r >> 1, and takes the 16 bytes of every plane piece that hold its half.
template <int KIND> struct RawRow { uint4 q[KIND == FK_Q6_K ? 3 : 4]; };

template <int KIND>
__device__ __forceinline__ void load_raw(const GemmArgs& a, const uint8_t* wb, int wrow0, int r, int st, bool live, RawRow<KIND>& raw) {
    constexpr int N = KIND == FK_Q6_K ? 3 : 4;
#pragma unroll
    for (int i = 0; i < N; i++) raw.q[i] = make_uint4(0, 0, 0, 0);
    const int k0 = st * KSTAGE;
    const int wrow = wrow0 + (KIND == FK_Q6_K ? r >> 1 : r);
    if (!live || wrow >= a.rows || k0 >= a.cols || KIND == FK_Q8_0) return;
    if (KIND == FK_Q4_K) {
        // 128 weights = 64 quant bytes: two groups of 32 bytes
        const uint8_t* p = wb + ((size_t)wrow * (a.cols >> 8) + (k0 >> 8)) * 144 + 16 + ((k0 >> 7) & 1) * 64;
#pragma unroll
        for (int i = 0; i < 4; i++) raw.q[i] = ldg16(p + 16 * i);
    } else if (KIND == FK_MXFP4) {
        const uint8_t* p = wb + a.plane_off[0] + (size_t)wrow * (a.cols >> 1) + (k0 >> 1);
#pragma unroll
        for (int b = 0; b < 4; b++)
            if (k0 + 32 * b < a.cols) raw.q[b] = ldg16(p + 16 * b);
    } else {  // FK_Q6_K: of the 64 ql bytes and 32 qh bytes of this half super-block, those of bytes 16 h .. 16 h + 15 of every 32
        const int sb = k0 >> 8, hf = (k0 >> 7) & 1, h = 16 * (r & 1);
        const uint8_t* ql = wb + a.plane_off[0] + (size_t)wrow * (a.cols >> 1) + (size_t)sb * 128 + 64 * hf + h;
        const uint8_t* qh = wb + a.plane_off[1] + (size_t)wrow * (a.cols >> 2) + (size_t)sb * 64 + 32 * hf + h;
        raw.q[0] = ldg16(ql);
        raw.q[1] = ldg16(ql + 32);
        raw.q[2] = ldg16(qh);
    }
}

// Decode one tile row's 128 weights of a stage to int8 and write them, eight 16-byte chunks each at their swizzled
// places.  Q6_K: the codes minus 32 with the 16 weights of the OTHER half of every run of 32 zeroed, so that one K = 32
// MMA yields the exact dot of a 16-weight scale group.
template <int KIND>
__device__ __forceinline__ void store_raw(const RawRow<KIND>& raw, int r, uint8_t* a_tile) {
    uint4 o[8];
    if (KIND == FK_Q4_K) {
        // low nibbles are the first 32 weights of a 32-byte group, high nibbles the next 32
#pragma unroll
        for (int g = 0; g < 2; g++) {
            const uint4 q0 = raw.q[2 * g], q1 = raw.q[2 * g + 1];
            o[4 * g + 0] = make_uint4(q0.x & 0x0F0F0F0Fu, q0.y & 0x0F0F0F0Fu, q0.z & 0x0F0F0F0Fu, q0.w & 0x0F0F0F0Fu);
            o[4 * g + 1] = make_uint4(q1.x & 0x0F0F0F0Fu, q1.y & 0x0F0F0F0Fu, q1.z & 0x0F0F0F0Fu, q1.w & 0x0F0F0F0Fu);
            o[4 * g + 2] = make_uint4((q0.x >> 4) & 0x0F0F0F0Fu, (q0.y >> 4) & 0x0F0F0F0Fu, (q0.z >> 4) & 0x0F0F0F0Fu, (q0.w >> 4) & 0x0F0F0F0Fu);
            o[4 * g + 3] = make_uint4((q1.x >> 4) & 0x0F0F0F0Fu, (q1.y >> 4) & 0x0F0F0F0Fu, (q1.z >> 4) & 0x0F0F0F0Fu, (q1.w >> 4) & 0x0F0F0F0Fu);
        }
    } else if (KIND == FK_MXFP4) {
        // bytes come out as (elem j, elem j+16) pairs, the order the activation
        // plane of this kind is stored in; an absent block (past the last column) is zeros
#pragma unroll
        for (int b = 0; b < 4; b++) {
            const uint4 q = raw.q[b];
            o[2 * b] = make_uint4(e2m1x2_4(q.x), e2m1x2_4(q.x >> 16), e2m1x2_4(q.y), e2m1x2_4(q.y >> 16));
            o[2 * b + 1] = make_uint4(e2m1x2_4(q.z), e2m1x2_4(q.z >> 16), e2m1x2_4(q.w), e2m1x2_4(q.w >> 16));
        }
    } else if (KIND == FK_Q6_K) {
        // element e = 32 * qd + 16 * half + l (qd = 0..3): nibble (qd >> 1) of ql piece (qd & 1), qh bits [2 qd, 2 qd + 2)
        const uint32_t hh[4] = {raw.q[2].x, raw.q[2].y, raw.q[2].z, raw.q[2].w};
        const bool odd = r & 1;
#pragma unroll
        for (int qd = 0; qd < 4; qd++) {
            const uint4 l0 = raw.q[qd & 1];
            const uint32_t ll[4] = {l0.x, l0.y, l0.z, l0.w};
            uint32_t v[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t nib = (qd >> 1) ? ((ll[i] >> 4) & 0x0F0F0F0Fu) : (ll[i] & 0x0F0F0F0Fu);
                v[i] = __vsub4(nib | (((hh[i] >> (2 * qd)) & 0x03030303u) << 4), 0x20202020u);
            }
            const uint4 val = make_uint4(v[0], v[1], v[2], v[3]), zero = make_uint4(0, 0, 0, 0);
            o[2 * qd] = odd ? zero : val;
            o[2 * qd + 1] = odd ? val : zero;
        }
    }
    uint8_t* dst = a_tile + r * 128;
#pragma unroll
    for (int c = 0; c < 8; c++) *(uint4*)(dst + ((c ^ (r & 7)) << 4)) = o[c];
}

__device__ __forceinline__ float lds32f(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr, int rank) {
    uint32_t remote;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote));
    return v;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int KIND, int BN, bool DUMP>
__global__ void __launch_bounds__(Tile<BN>::THREADS, Tile<BN>::BLOCKS)
gemm_kernel(const GemmArgs a, const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_dx,
            const __grid_constant__ CUtensorMap map_sx, const __grid_constant__ CUtensorMap map_w) {
    using S = Smem<BN>;
    using T = Tile<BN>;
    constexpr int EPI_WARPS = T::EPI_WARPS, UNPACK_WARPS = T::UNPACK_WARPS, NACC = T::NACC, G = T::GROUP, CW = T::CW, NCH = CW / 16;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32(smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // Only weights (constants) may be read before the quantizer in front of this launch has finished; the grouped form's
    // tile list is the work of the kernels before that.
    const int ttile = blockIdx.y;
    if (a.n_tiles_dev) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (ttile >= *a.n_tiles_dev) return;       // every CTA of the cluster alike
    }
    const int mat = a.tile_expert ? a.tile_expert[ttile] : a.mat;
    const uint8_t* wb = a.w + (size_t)mat * a.mat_stride;
    // Q6_K tile rows are (weight row, half) pairs: 64 weight rows per CTA
    constexpr int WROWS = KIND == FK_Q6_K ? BM / 2 : BM;
    const int wrow0 = blockIdx.x * WROWS;
    const int tok0 = ttile * BN;
    const int nkb = a.cols >> 5;
    const int nst_all = (nkb + 3) >> 2;
    // this CTA's stages: [st0, st0 + nst) of the row, runs kb_lo .. kb_lo + nkl - 1
    const int rank = blockIdx.z, split = a.split;
    const int st0 = (int)((long long)nst_all * rank / split), nst = (int)((long long)nst_all * (rank + 1) / split) - st0;
    const int kb_lo = 4 * st0, nkl = min(nkb - kb_lo, 4 * nst);

    // barriers: full_b[NSTAGE], full_a[NSTAGE], empty[NSTAGE], acc_full[2], acc_empty[2], then the TMEM base word
    const uint32_t bar0 = sbase + S::BARS;
    auto full_b = [&](int s) { return bar0 + 8u * s; };
    auto full_a = [&](int s) { return bar0 + 8u * (NSTAGE + s); };
    auto empty = [&](int s) { return bar0 + 8u * (2 * NSTAGE + s); };
    auto acc_full = [&](int b) { return bar0 + 8u * (3 * NSTAGE + b); };
    auto acc_empty = [&](int b) { return bar0 + 8u * (3 * NSTAGE + 2 + b); };
    uint32_t* tmem_word = (uint32_t*)(smem + S::BARS + 8 * (3 * NSTAGE + 4));

    if (threadIdx.x == 0) {
        for (int s = 0; s < NSTAGE; s++) {
            mbar_init(full_b(s), 1);
            mbar_init(full_a(s), UNPACK_WARPS);
            mbar_init(empty(s), 1 + EPI_WARPS);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(acc_full(b), 1);
            mbar_init(acc_empty(b), EPI_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == EPI_WARPS + UNPACK_WARPS + 1) {  // the MMA warp owns tensor memory
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_word)), "r"(NACC * BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_word;

    auto out_row_of = [&](int t) { return a.out_row ? a.out_row[t] : (t < a.m ? t : -1); };
    if (warp < EPI_WARPS) {
        // ------------------------------------------------------------ epilogue
        const int quad = warp & 3, chalf = warp >> 2;
        const int r = quad * 32 + lane;                // tile row = TMEM lane
        const bool row_ok = (KIND == FK_Q6_K ? (wrow0 + (r >> 1)) : (wrow0 + r)) < a.rows;
        const int orow = KIND == FK_Q6_K ? wrow0 + (r >> 1) : wrow0 + r;
        const bool writer = row_ok && (KIND != FK_Q6_K || !(r & 1));
        float acc[CW];                                 // CW token columns of one row
#pragma unroll
        for (int i = 0; i < CW; i++) acc[i] = 0.0f;
        const uint32_t taddr0 = tmem_base + ((uint32_t)(quad * 32) << 16) + chalf * CW;
        if (!a.n_tiles_dev) asm volatile("griddepcontrol.wait;" ::: "memory");
        // TMEM reads are double-buffered in chunks of 16 columns (two a run, or one): while one chunk is scaled the next is
        // already in flight, so a warp's chain per run is its arithmetic, not the accumulator hand-off latency.
        uint32_t va[16], vb[16];
        auto issue = [&](int kb, int c, uint32_t* dst) {   // kb counts from this CTA's first run
            if (c == 0 && kb % G == 0) {
                mbar_wait(acc_full((kb / G) & 1), (kb / NACC) & 1, a.err, 11);
                tc_fence_after();
                GTR(1, kb, warp == 0 && lane == 0);
            }
            tc_ld16(taddr0 + (kb % NACC) * BN + c * 16, dst);
        };
        issue(0, 0, va);
        tc_wait_ld();
        tc_ld_fence<16>(va);
        float dw = 0.0f, mw = 0.0f;
        // chunk c of run kb (= run j of the stage at sdx_s) out of cur, the chunk after it on its way into nxt
        auto step = [&](int kb, int j, int c, uint32_t sdx_s, uint32_t* cur, uint32_t* nxt) {
            const int kb_n = c == NCH - 1 ? kb + 1 : kb, c_n = c == NCH - 1 ? 0 : c + 1;
            if (c == 0) {
                const uint32_t sw = sdx_s + (uint32_t)(S::DW - S::DX) + (uint32_t)(j * BM + r) * 4u;
                dw = lds32f(sw);
                if (KIND == FK_Q4_K) mw = lds32f(sw + S::DW_BYTES);
            }
            if (kb_n < nkl) issue(kb_n, c_n, nxt);
            const uint32_t dxs = sdx_s + (uint32_t)(j * BN + chalf * CW + c * 16) * 4u;
            if (DUMP && row_ok) {
                // the exact integers of this run, before any scale touches them
                const int nruns = KIND == FK_Q6_K ? a.cols >> 4 : nkb, run = KIND == FK_Q6_K ? 2 * (kb_lo + kb) + (r & 1) : kb_lo + kb;
                for (int i = 0; i < 16; i++) {
                    const int dst = out_row_of(tok0 + chalf * CW + c * 16 + i);
                    if (dst >= 0) a.isums[((size_t)dst * a.rows + orow) * nruns + run] = (int32_t)cur[i];
                }
            }
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
                const float4 dx = lds128(dxs + 4u * i);
                const float dxa[4] = {dx.x, dx.y, dx.z, dx.w};
                float sxa[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if (KIND == FK_Q4_K) {
                    const float4 sx = lds128(dxs + 16u * BN + 4u * i);
                    sxa[0] = sx.x; sxa[1] = sx.y; sxa[2] = sx.z; sxa[3] = sx.w;
                }
                // two columns per instruction on the packed f32x2 path; int32 -> f32 (exact, |C| < 2^22) on the
                // conversion unit: one issue slot, where the magic-number add takes two on the integer and FP32 pipes
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                    const float2 f2 = make_float2((float)(int)cur[i + e], (float)(int)cur[i + e + 1]);
                    const float2 s2 = __fmul2_rn(make_float2(dw, dw), make_float2(dxa[e], dxa[e + 1]));
                    float2 t2 = __ffma2_rn(s2, f2, make_float2(acc[c * 16 + i + e], acc[c * 16 + i + e + 1]));
                    if (KIND == FK_Q4_K) t2 = __ffma2_rn(make_float2(-mw, -mw), make_float2(sxa[e], sxa[e + 1]), t2);
                    acc[c * 16 + i + e] = t2.x;
                    acc[c * 16 + i + e + 1] = t2.y;
                }
            }
            tc_wait_ld();
            tc_ld_fence<16>(nxt);
            if (kb_n < nkl && c_n == NCH - 1 && (kb_n % G == G - 1 || kb_n == nkl - 1)) {   // the group's last chunk is in registers: hand it back
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty((kb_n / G) & 1));
            }
        };
        for (int st = 0; st < nst; st++) {
            const int s = st % NSTAGE;
            mbar_wait(full_a(s), (st / NSTAGE) & 1, a.err, 9);    // the scale tiles of this stage: the weights' ...
            mbar_wait(full_b(s), (st / NSTAGE) & 1, a.err, 10);   // ... and the activations': dx [4][BN] then (Q4_K) sx [4][BN]
            const uint32_t sdx_s = sbase + s * S::STAGE + S::DX;
            // Rolled on purpose: the unrolled body falls out of the instruction cache.
#pragma unroll 1
            for (int q = 0; q < 4 * NCH; q += 2) {
                const int j = q / NCH, kb = 4 * st + j;
                if (kb >= nkl) break;
                step(kb, j, 0, sdx_s, va, vb);
                if (NCH == 1 && kb + 1 >= nkl) break;
                if (NCH == 1) step(kb + 1, j + 1, 0, sdx_s, vb, va);
                else step(kb, j, 1, sdx_s, vb, va);
            }
            // this warp is done with the stage's scale tiles
            __syncwarp();
            if (lane == 0) mbar_arrive(empty(s));
        }
        if (split == 1) {
            // ---- store: out[out_row[token]][weight row]
#pragma unroll
            for (int i = 0; i < CW; i++) {
                float v0 = acc[i];
                if (KIND == FK_Q6_K) v0 += __shfl_xor_sync(0xffffffffu, v0, 1);   // the two halves of a weight row sit in neighbouring lanes
                const int dst = out_row_of(tok0 + chalf * CW + i);
                if (writer && dst >= 0) a.out[(size_t)dst * a.rows + orow] = v0;
            }
        } else {
            // every epilogue warp is past its last read of the stages' scale tiles, and the last accumulator was read, so no
            // copy or MMA touches the stages any more: they hold this part's sums, [token column][tile row]
            asm volatile("bar.sync 1, %0;" ::"r"(EPI_WARPS * 32) : "memory");
            float* part = (float*)smem;
#pragma unroll
            for (int i = 0; i < CW; i++) part[(chalf * CW + i) * BM + r] = acc[i];
        }
    } else if (warp < EPI_WARPS + UNPACK_WARPS) {
        // ------------------------------------------------- weight unpack warps
        // A thread owns NR tile rows (Q8_0: their scales only); the loads of the next DEPTH stages are in flight while a stage
        // is written.  The slots are rotated by unrolling, not by copying: a register move out of a load that is still in
        // flight waits for it, and the prefetch with it (3072 x 3072 Q4_K in 32-token tiles: 62 us with moves, 46 without).
        constexpr int NR = BM / (32 * UNPACK_WARPS), DEPTH = BN == 64 ? 2 : 1, SLOTS = DEPTH + 1;
        const int t = (warp - EPI_WARPS) * 32 + lane;
        RawRow<KIND> raw[SLOTS][NR];
        RawScale<KIND> rsc[SLOTS][NR];
        auto load = [&](int p, int st) {
#pragma unroll
            for (int i = 0; i < NR; i++) {
                load_raw<KIND>(a, wb, wrow0, t + 32 * UNPACK_WARPS * i, st0 + st, st < nst, raw[p][i]);
                load_wscales<KIND>(a, wb, wrow0, t + 32 * UNPACK_WARPS * i, st0 + st, st < nst, rsc[p][i]);
            }
        };
#pragma unroll
        for (int p = 0; p < DEPTH; p++) load(p, p);
        for (int stu = 0; stu < nst; stu += SLOTS) {
#pragma unroll
            for (int u = 0; u < SLOTS; u++) {
                const int st = stu + u, s = st % NSTAGE;
                if (st >= nst) break;
                load((u + DEPTH) % SLOTS, st + DEPTH);
                if (st >= NSTAGE) mbar_wait(empty(s), ((st / NSTAGE) - 1) & 1, a.err, 20);
#pragma unroll
                for (int i = 0; i < NR; i++) {
                    const int r = t + 32 * UNPACK_WARPS * i;
                    if (KIND != FK_Q8_0) store_raw<KIND>(raw[u][i], r, smem + s * S::STAGE);
                    const StageScale sc = stage_scales<KIND>(rsc[u][i], 4 * (st0 + st));
                    float* sdw = (float*)(smem + s * S::STAGE + S::DW) + r;
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        float dw, mw;
                        run_scale<KIND>(sc, j, r, &dw, &mw);
                        sdw[j * BM] = dw;
                        if (KIND == FK_Q4_K) sdw[(4 + j) * BM] = mw;
                    }
                }
                fence_proxy_async();   // generic-proxy writes -> visible to the tensor core's reads
                __syncwarp();
                if (lane == 0) mbar_arrive(full_a(s));
                GTR(3, st, warp == EPI_WARPS && lane == 0);
            }
        }
    } else if (warp == EPI_WARPS + UNPACK_WARPS) {
        // --------------------------------------------------------- TMA producer
        if (!a.n_tiles_dev) asm volatile("griddepcontrol.wait;" ::: "memory");
        if (lane == 0) {
            constexpr uint32_t TX = S::B_BYTES + S::DX_BYTES + (KIND == FK_Q4_K ? S::DX_BYTES : 0) + (KIND == FK_Q8_0 ? S::A_BYTES : 0);
            for (int st = 0; st < nst; st++) {
                const int s = st % NSTAGE;
                if (st >= NSTAGE) mbar_wait(empty(s), ((st / NSTAGE) - 1) & 1, a.err, 30);
                const uint32_t sa = sbase + s * S::STAGE;
                mbar_expect_tx(full_b(s), TX);
                tma_load_2d(sa + S::A_BYTES, &map_q, (st0 + st) * KSTAGE, tok0, full_b(s));
                tma_load_2d(sa + S::DX, &map_dx, tok0, 4 * (st0 + st), full_b(s));
                if (KIND == FK_Q4_K) tma_load_2d(sa + S::DX + S::DX_BYTES, &map_sx, tok0, 4 * (st0 + st), full_b(s));
                if (KIND == FK_Q8_0) tma_load_3d(sa, &map_w, (st0 + st) * KSTAGE, wrow0, mat, full_b(s));   // [matrix][row][k]: rows past a matrix's end read as zeros
            }
        }
    } else {
        // ----------------------------------------------------------- MMA issuer
        if (lane == 0) {
            constexpr uint32_t IDESC = umma_idesc_i8(BM, BN);
            for (int st = 0; st < nst; st++) {
                const int s = st % NSTAGE;
                mbar_wait(full_b(s), (st / NSTAGE) & 1, a.err, 40);
                mbar_wait(full_a(s), (st / NSTAGE) & 1, a.err, 41);
                tc_fence_after();
                const uint32_t sa = sbase + s * S::STAGE;
                const uint64_t da = umma_desc(sa), db = umma_desc(sa + S::A_BYTES);
                for (int j = 0; j < 4; j++) {
                    const int kb = 4 * st + j;
                    if (kb >= nkl) break;
                    if (kb % G == 0) {
                        if (kb >= NACC) mbar_wait(acc_empty((kb / G) & 1), ((kb / NACC) - 1) & 1, a.err, 42);
                        tc_fence_after();
                    }
                    // K advances 32 bytes inside the 128-byte swizzle atom: +2 in the 16-byte address field
                    GTR(0, kb, true);
                    tc_mma_i8(tmem_base + (kb % NACC) * BN, da + 2 * j, db + 2 * j, IDESC);
                    if (kb % G == G - 1 || kb == nkl - 1) tc_commit(acc_full((kb / G) & 1));
                }
                tc_commit(empty(s));   // arrives once the MMAs that read this stage are done
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (split > 1) {
        // the parts of the tile meet through distributed shared memory: CTA `rank` adds up its share of the token columns,
        // in rank order (the same order whatever the timing), and writes it out
        cluster_sync_all();
        if (warp < EPI_WARPS) {
            const int cols_mine = BN / split;
            for (int i = threadIdx.x; i < cols_mine * BM; i += EPI_WARPS * 32) {
                const int r = i & (BM - 1), c = rank * cols_mine + i / BM;
                float pz[MAX_SPLIT];
#pragma unroll
                for (int z = 0; z < MAX_SPLIT; z++) pz[z] = z < split ? ld_cluster_f32(sbase + (uint32_t)(c * BM + r) * 4u, z) : 0.0f;
                float v0 = pz[0];
#pragma unroll
                for (int z = 1; z < MAX_SPLIT; z++) v0 += pz[z];
                if (KIND == FK_Q6_K) v0 += __shfl_xor_sync(0xffffffffu, v0, 1);
                const int orow = KIND == FK_Q6_K ? wrow0 + (r >> 1) : wrow0 + r;
                const int dst = out_row_of(tok0 + c);
                if (orow < a.rows && (KIND != FK_Q6_K || !(r & 1)) && dst >= 0) a.out[(size_t)dst * a.rows + orow] = v0;
            }
        }
        cluster_sync_all();     // no CTA leaves while another may still read its part
    }
    if (warp == EPI_WARPS + UNPACK_WARPS + 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(NACC * BN) : "memory");
    }
}

// ---------------------------------------------------------------------------
// Activation plan: q8_1 of every (padded) token row into an int8 plane [n_pad][cols] (row-major, K inner; MXFP4 keeps
// each run as (j, j+16) pairs) plus run-major scale planes dx[nkb][n_pad] and, for Q4_K, sx = dx * run sum.  A thread
// takes four values, eight lanes make a run.  Rows past the live tiles (`*n_tiles_dev * bn`, grouped form) are left
// alone: no tile reads them.  src_row == nullptr (dense): row t reads token t, rows from m on are padding.
template <bool PAIRS>
__global__ void quantize_acts4_kernel(const float* __restrict__ x, const int* __restrict__ src_row, int m, int n_pad, int cols, int8_t* __restrict__ q,
                                      float* __restrict__ dx, float* __restrict__ sx, const int* __restrict__ n_tiles_dev, int bn) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the GEMM may set itself up and fetch weights meanwhile
    const int nkb = cols >> 5;
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long run = gid >> 3;
    const int part = (int)(gid & 7);
    const int n_live = n_tiles_dev ? min(n_pad, *n_tiles_dev * bn) : n_pad;
    const bool ok = run < (long long)n_live * nkb;          // whole groups of eight lanes are in or out
    const int t = ok ? (int)(run / nkb) : 0, kb = ok ? (int)(run - (long long)t * nkb) : 0;
    const int src = !ok ? -1 : src_row ? src_row[t] : (t < m ? t : -1);
    float4 f = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (src >= 0) {
        // every row is whole runs of 128 bytes, so x alone decides whether float4 loads are aligned; the callers may pass a
        // view that starts at any float
        const float* p = x + (size_t)src * cols + kb * 32 + part * 4;
        if (((uintptr_t)x & 15) == 0) f = __ldg((const float4*)p);
        else f = make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
    }
    // the maximum over bit patterns, as fk_q8_1_lane takes it: a NaN is larger than every number there, so it becomes the run's
    // scale and reaches the output (fmaxf drops it, and the row came out finite)
    unsigned mb = max(max(__float_as_uint(fabsf(f.x)), __float_as_uint(fabsf(f.y))), max(__float_as_uint(fabsf(f.z)), __float_as_uint(fabsf(f.w))));
    mb = max(mb, __shfl_xor_sync(0xffffffffu, mb, 1));
    mb = max(mb, __shfl_xor_sync(0xffffffffu, mb, 2));
    mb = max(mb, __shfl_xor_sync(0xffffffffu, mb, 4));
    const float amax = __uint_as_float(mb);
    const float d = amax / 127.0f;
    int q0 = 0, q1 = 0, q2 = 0, q3 = 0;
    if (amax != 0.0f) {
        q0 = (int)roundf(f.x / d); q1 = (int)roundf(f.y / d); q2 = (int)roundf(f.z / d); q3 = (int)roundf(f.w / d);
    }
    int qsum = q0 + q1 + q2 + q3;
    qsum += __shfl_xor_sync(0xffffffffu, qsum, 1);
    qsum += __shfl_xor_sync(0xffffffffu, qsum, 2);
    qsum += __shfl_xor_sync(0xffffffffu, qsum, 4);
    const uint32_t mine = (uint32_t)(q0 & 0xFF) | ((uint32_t)(q1 & 0xFF) << 8) | ((uint32_t)(q2 & 0xFF) << 16) | ((uint32_t)(q3 & 0xFF) << 24);
    const uint32_t other = PAIRS ? __shfl_xor_sync(0xffffffffu, mine, 4) : 0u;      // elements 16 further on (lanes 0..3 of the run)
    if (!ok) return;
    if (!PAIRS)
        *(uint32_t*)(q + (size_t)t * cols + kb * 32 + part * 4) = mine;
    else if (part < 4)
        *(uint2*)(q + (size_t)t * cols + kb * 32 + part * 8) = make_uint2(__byte_perm(mine, other, 0x5140), __byte_perm(mine, other, 0x7362));
    if (part == 0) {
        const float dq = fk_h2f(fk_f2h(d));
        dx[(size_t)kb * n_pad + t] = dq;
        if (sx) sx[(size_t)kb * n_pad + t] = dq * (float)qsum;
    }
}

// Grouped plan (one block): every expert's rows padded up to whole tiles of BN.
// Permuted row p of expert e lands at pad_off[e] + (p - group_off[e]).  The offsets are a serial scan by one thread
// (a few hundred additions); everything else is spread over the block: a thread finds its row's expert by bisecting
// the group offsets in shared memory.
__global__ void grouped_plan_kernel(const int* __restrict__ group_off, const int* __restrict__ gather, int n_experts, int bn,
                                    int n_pad, int* src_row, int* out_row, int* tile_expert, int* n_tiles) {
    extern __shared__ int sm_plan[];  // pad_off [n_experts + 1] | group_off [n_experts + 1]
    int* pad_off = sm_plan;
    int* goff = sm_plan + n_experts + 1;
    for (int e = threadIdx.x; e <= n_experts; e += blockDim.x) goff[e] = group_off[e];
    __syncthreads();
    if (threadIdx.x == 0) {
        int acc = 0;
        for (int e = 0; e < n_experts; e++) {
            pad_off[e] = acc;
            acc += (goff[e + 1] - goff[e] + bn - 1) / bn * bn;
        }
        pad_off[n_experts] = acc;
        *n_tiles = acc / bn;
    }
    for (int t = threadIdx.x; t < n_pad; t += blockDim.x) {
        src_row[t] = -1;
        out_row[t] = -1;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x)
        for (int tl = pad_off[e] / bn; tl < pad_off[e + 1] / bn; tl++) tile_expert[tl] = e;
    const int pairs = goff[n_experts];
    for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
        int lo = 0, hi = n_experts;          // the expert e with goff[e] <= p < goff[e + 1] (empty experts are skipped by the bisection)
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (goff[mid] <= p) lo = mid; else hi = mid;
        }
        const int dst = pad_off[lo] + (p - goff[lo]);
        src_row[dst] = gather ? gather[p] : p;
        out_row[dst] = p;
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

// 2-D row-major tensor [outer][inner] of `esize`-byte elements, box [box_outer][box_inner].
int make_map(CUtensorMap* map, CUtensorMapDataType dt, int esize, void* base, uint64_t inner, uint64_t outer, uint32_t box_inner,
             uint32_t box_outer, CUtensorMapSwizzle sw) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fk_fail(FK_DRIVER_INIT, "gemm: the driver does not export cuTensorMapEncodeTiled");
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {inner * (uint64_t)esize};
    cuuint32_t box[2] = {box_inner, box_outer};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, dt, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fk_fail(FK_LAUNCH, "gemm: cuTensorMapEncodeTiled failed (%d) for a [%llu][%llu] tensor", (int)r,
                                          (unsigned long long)outer, (unsigned long long)inner);
    return FK_OK;
}

// The int8 plane of a stack of Q8_0 matrices as a [n_mats][rows][cols] tensor, box [1][BM][KSTAGE].
int make_map_q8_0(CUtensorMap* map, const fk_weight_s* w) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fk_fail(FK_DRIVER_INIT, "gemm: the driver does not export cuTensorMapEncodeTiled");
    cuuint64_t dims[3] = {(cuuint64_t)w->cols, (cuuint64_t)w->rows, (cuuint64_t)w->n_mats};
    cuuint64_t strides[2] = {(cuuint64_t)w->plane_stride[0], (cuuint64_t)w->mat_stride};
    cuuint32_t box[3] = {(cuuint32_t)KSTAGE, (cuuint32_t)BM, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, w->dev + w->plane_off[0], dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fk_fail(FK_LAUNCH, "gemm: cuTensorMapEncodeTiled failed (%d) for %d Q8_0 matrices of %d x %d", (int)r, w->n_mats, w->rows, w->cols);
    return FK_OK;
}

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

template <int KIND, int BN, bool DUMP = false>
int launch_gemm(fk_ctx* ctx, cudaStream_t st, const GemmArgs& a, const CUtensorMap& mq, const CUtensorMap& mdx, const CUtensorMap& msx,
                const CUtensorMap& mw, int n_token_tiles) {
    auto kern = gemm_kernel<KIND, BN, DUMP>;
    constexpr int SMEM = Smem<BN>::TOTAL;
    FK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM), FK_KERNEL);
    constexpr int WROWS = KIND == FK_Q6_K ? BM / 2 : BM;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((a.rows + WROWS - 1) / WROWS, n_token_tiles, a.split);
    cfg.blockDim = dim3(Tile<BN>::THREADS);
    cfg.dynamicSmemBytes = SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;    // set up and fetch weights while the quantizer runs
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = a.split;
    cfg.attrs = attr;
    cfg.numAttrs = a.split > 1 ? 2 : 1;
    FK_CUDA(cudaLaunchKernelEx(&cfg, kern, a, mq, mdx, msx, mw), FK_LAUNCH);
    ctx->launches++;
    return FK_OK;
}

template <int BN>
int launch_by_kind(fk_ctx* ctx, cudaStream_t st, const GemmArgs& a, int kind, const CUtensorMap& mq, const CUtensorMap& mdx, const CUtensorMap& msx,
                   const CUtensorMap& mw, int n_token_tiles) {
    if (a.isums) {
        switch (kind) {
            case FK_Q4_K: return launch_gemm<FK_Q4_K, BN, true>(ctx, st, a, mq, mdx, msx, mw, n_token_tiles);
            case FK_Q6_K: return launch_gemm<FK_Q6_K, BN, true>(ctx, st, a, mq, mdx, msx, mw, n_token_tiles);
            case FK_Q8_0: return launch_gemm<FK_Q8_0, BN, true>(ctx, st, a, mq, mdx, msx, mw, n_token_tiles);
            case FK_MXFP4: return launch_gemm<FK_MXFP4, BN, true>(ctx, st, a, mq, mdx, msx, mw, n_token_tiles);
        }
    }
    switch (kind) {
        case FK_Q4_K: return launch_gemm<FK_Q4_K, BN>(ctx, st, a, mq, mdx, msx, mw, n_token_tiles);
        case FK_Q6_K: return launch_gemm<FK_Q6_K, BN>(ctx, st, a, mq, mdx, msx, mw, n_token_tiles);
        case FK_Q8_0: return launch_gemm<FK_Q8_0, BN>(ctx, st, a, mq, mdx, msx, mw, n_token_tiles);
        case FK_MXFP4: return launch_gemm<FK_MXFP4, BN>(ctx, st, a, mq, mdx, msx, mw, n_token_tiles);
    }
    return fk_fail(FK_UNSUPPORTED, "gemm: kind %d has no kernel", kind);
}

// Which tile (token columns per CTA) and how many CTAs along K: the candidate with the smallest estimated time
//
//   waves * (runs / split * us_per_run(bn) + (split > 1) * exchange(bn)),   waves = CTAs / (SMs * CTAs per SM)
//
// The constants were measured on B200 (us; Q4_K, 3072 x 3072, cold L2; the other kinds are within 20 % below, but MXFP4 in
// 128-token tiles takes 0.80): a 128-token tile takes 0.68 a run of 32 K, a 64-token one 0.47, a 32-token one 0.42 alone on
// its SM and 0.56 beside another; the parts of a split tile take 6 to 8 to meet.  A tile's own time falls far less than its
// width -- its warps walk the same chain per run -- so what a short prompt needs is more CTAs, not only narrower ones
// (us, whole 128-token tiles in one part against the plan's): 3072 x 3072, M = 128 71 -> 32; 3072 x 8192 Q6_K, M = 77
// 146 -> 75; 512 x 3072, M = 16 71 -> 17; 8192 x 3072, M = 512 keeps whole 128-token tiles (138; 64-token tiles 177, 32-token
// ones 200).  Grouped: `tiles` expects half a tile of padding per expert, which is what 32-token tiles win by (128 experts, 8
// of them for each of 77 rows, 768 x 2048 Q4_K: 169 us against 230 with 64-token tiles and 345 with 128).
struct GemmPlan { int bn, split; };

GemmPlan gemm_plan(const fk_ctx* ctx, const fk_weight_s* w, int m, bool grouped) {
    const int wrows = w->kind == FK_Q6_K ? BM / 2 : BM, row_tiles = (w->rows + wrows - 1) / wrows;
    const int runs = w->cols / 32, stages = (runs + 3) / 4;
    GemmPlan best{128, 1};
    double best_us = 1e30;
    for (int bn : {128, 64, 32}) {
        const double tiles = grouped ? (double)m / bn + 0.5 * (m < w->n_mats ? m : w->n_mats) : (double)((m + bn - 1) / bn);
        for (int split = 1; split <= MAX_SPLIT && split <= stages; split *= 2) {
            const double ctas = tiles * row_tiles * split;
            const double sms = split == 8 ? 0.9 * ctx->sm_count : ctx->sm_count;       // clusters of eight do not tile every GPC
            const bool two = bn == 32 && ctas > sms;
            double us = bn == 128 ? (w->kind == FK_MXFP4 ? 0.80 : 0.68) : bn == 64 ? 0.47 : two ? 0.56 : 0.42;
            us = us * (4 * ((stages + split - 1) / split)) + (split > 1 ? (bn == 128 ? 8.0 : bn == 64 ? 7.0 : 6.0) : 0.0);
            const double waves = ctas / (two ? 2.0 * sms : sms);
            us *= waves > 4.0 ? waves + 0.25 : ceil(waves);
            if (us < best_us) { best_us = us; best = {bn, split}; }
        }
    }
    return best;
}

// The scratch of one call: q plane | dx | sx | row tables of the grouped form.
struct GemmScratch {
    size_t dx, sx, src, out, te, nt, total;
    GemmScratch(int n_pad, int cols, int n_tiles, bool grouped) {
        const int nkb = cols / 32;
        dx = align_up((size_t)n_pad * cols, 1024);
        sx = align_up(dx + (size_t)nkb * n_pad * 4, 1024);
        src = align_up(sx + (size_t)nkb * n_pad * 4, 1024);
        out = src + (grouped ? (size_t)n_pad * 4 : 0);
        te = out + (grouped ? (size_t)n_pad * 4 : 0);
        nt = te + (grouped ? (size_t)n_tiles * 4 : 0);
        total = nt + 16;
    }
};

// Quantizer and GEMM of one call on a prepared scratch block (fk_gemm, fk_gemm_grouped after its plan, fk_gemm_static).
int gemm_run(fk_ctx* ctx, cudaStream_t st, fk_weight w, int mat, const float* x, int m, float* out, int32_t* isums, const GemmPlan& plan,
             uint8_t* sc, const GemmScratch& L, int n_pad, bool grouped) {
    const int bn = plan.bn, nkb = w->cols / 32;
    int8_t* q = (int8_t*)sc;
    float *dx = (float*)(sc + L.dx), *sx = (float*)(sc + L.sx);
    const int* src_row = grouped ? (const int*)(sc + L.src) : nullptr;
    const int* n_tiles = grouped ? (const int*)(sc + L.nt) : nullptr;
    const unsigned qgrid = (unsigned)(((long long)n_pad * nkb + 31) / 32);
    float* sxq = w->kind == FK_Q4_K ? sx : nullptr;
    if (w->kind == FK_MXFP4) quantize_acts4_kernel<true><<<qgrid, 256, 0, st>>>(x, src_row, m, n_pad, w->cols, q, dx, sxq, n_tiles, bn);
    else quantize_acts4_kernel<false><<<qgrid, 256, 0, st>>>(x, src_row, m, n_pad, w->cols, q, dx, sxq, n_tiles, bn);
    FK_CUDA(cudaGetLastError(), FK_LAUNCH);
    ctx->launches++;

    int rc;
    CUtensorMap mq, mdx, msx, mw;
    if ((rc = make_map(&mq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, q, w->cols, n_pad, KSTAGE, bn, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
    if ((rc = make_map(&mdx, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, dx, n_pad, nkb, bn, 4, CU_TENSOR_MAP_SWIZZLE_NONE))) return rc;
    if ((rc = make_map(&msx, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, sx, n_pad, nkb, bn, 4, CU_TENSOR_MAP_SWIZZLE_NONE))) return rc;
    mw = mq;
    if (w->kind == FK_Q8_0 && (rc = make_map_q8_0(&mw, w))) return rc;
    GemmArgs a;
    a.w = w->dev;
    a.mat_stride = w->mat_stride;
    for (int i = 0; i < 4; i++) { a.plane_off[i] = w->plane_off[i]; a.plane_stride[i] = w->plane_stride[i]; }
    a.rows = w->rows;
    a.cols = w->cols;
    a.mat = mat;
    a.tile_expert = grouped ? (const int*)(sc + L.te) : nullptr;
    a.n_tiles_dev = n_tiles;
    a.out_row = grouped ? (const int*)(sc + L.out) : nullptr;
    a.m = m;
    a.split = plan.split;
    a.out = out;
    a.isums = isums;
    a.err = ctx->err_flag;
    const int tiles = n_pad / bn;
    return bn == 128  ? launch_by_kind<128>(ctx, st, a, w->kind, mq, mdx, msx, mw, tiles)
           : bn == 64 ? launch_by_kind<64>(ctx, st, a, w->kind, mq, mdx, msx, mw, tiles)
                      : launch_by_kind<32>(ctx, st, a, w->kind, mq, mdx, msx, mw, tiles);
}

// Shared body of fk_gemm (group_off == nullptr) and fk_gemm_grouped; `given` takes the place of the plan (test hook).
int gemm_common(fk_ctx* ctx, cudaStream_t st, fk_weight w, int mat, const int* group_off, const int* gather, const float* x,
                int n_tokens, float* out, int32_t* isums = nullptr, const GemmPlan* given = nullptr) {
    const bool grouped = group_off != nullptr;
    if (w->kind == FK_Q5_K || w->kind == FK_BF16)   // before anything is enqueued: the caller takes batches of 8 through the matvec
        return fk_fail(FK_UNSUPPORTED, "gemm: kind %d has the plain matvec only", w->kind);
    const GemmPlan plan = given ? *given : gemm_plan(ctx, w, n_tokens, grouped);
    const int n_tiles_max = (n_tokens + plan.bn - 1) / plan.bn + (grouped ? w->n_mats : 0), n_pad = n_tiles_max * plan.bn;
    const GemmScratch L(n_pad, w->cols, n_tiles_max, grouped);
    int rc = fk_ensure_scratch(ctx, st, L.total);
    if (rc) return rc;
    uint8_t* sc = ctx->scratch;
    if (grouped) {
        grouped_plan_kernel<<<1, 1024, 2 * (w->n_mats + 1) * sizeof(int), st>>>(group_off, gather, w->n_mats, plan.bn, n_pad, (int*)(sc + L.src),
                                                                             (int*)(sc + L.out), (int*)(sc + L.te), (int*)(sc + L.nt));
        FK_CUDA(cudaGetLastError(), FK_LAUNCH);
        ctx->launches++;
    }
    return gemm_run(ctx, st, w, mat, x, n_tokens, out, isums, plan, sc, L, n_pad, grouped);
}

}  // namespace

#ifdef FK_TRACE
extern "C" __attribute__((visibility("default"))) int fk_gemm_trace_read(void* host, size_t bytes) {
    return cudaMemcpyFromSymbol(host, fk_gemm_trace, bytes) == cudaSuccess ? 0 : 1;
}
#endif

// General 2-D map for the other kernel files: dtype 0 = uint8, 1 = uint16, 2 = uint32, 3 = float32;
// swizzle 0 = none, 1 = 32 B, 2 = 64 B, 3 = 128 B.
int fk_make_map_2d(void* map, int dtype, void* base, uint64_t inner, uint64_t outer, uint32_t box_inner, uint32_t box_outer, int swizzle) {
    static const CUtensorMapDataType dt[4] = {CU_TENSOR_MAP_DATA_TYPE_UINT8, CU_TENSOR_MAP_DATA_TYPE_UINT16, CU_TENSOR_MAP_DATA_TYPE_UINT32,
                                              CU_TENSOR_MAP_DATA_TYPE_FLOAT32};
    static const int es[4] = {1, 2, 4, 4};
    static const CUtensorMapSwizzle sw[4] = {CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_SWIZZLE_128B};
    return make_map((CUtensorMap*)map, dt[dtype], es[dtype], base, inner, outer, box_inner, box_outer, sw[swizzle]);
}

// Bytes as a [n2][n1][inner] tensor whose n1 rows lie stride1 bytes apart and whose n2 pieces of a row follow one another
// (inner bytes apart); box [b2][b1][b0], swizzle as above.
int fk_make_map_3d(void* map, void* base, uint32_t inner, uint64_t n1, uint64_t stride1, uint64_t n2, uint32_t b0, uint32_t b1, uint32_t b2, int swizzle) {
    static const CUtensorMapSwizzle sw[4] = {CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_SWIZZLE_128B};
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fk_fail(FK_DRIVER_INIT, "the driver does not export cuTensorMapEncodeTiled");
    cuuint64_t dims[3] = {inner, n1, n2};
    cuuint64_t strides[2] = {stride1, inner};
    cuuint32_t box[3] = {b0, b1, b2};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn((CUtensorMap*)map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw[swizzle],
                    CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fk_fail(FK_LAUNCH, "cuTensorMapEncodeTiled failed (%d) for a [%llu][%llu][%u] tensor", (int)r, (unsigned long long)n2,
                                          (unsigned long long)n1, inner);
    return FK_OK;
}

// A [outer][inner] tensor of 32-bit words, unswizzled, for the other kernel files.
int fk_make_map_u32(void* map, void* base, uint64_t inner_words, uint64_t outer, uint32_t box_inner, uint32_t box_outer) {
    return make_map((CUtensorMap*)map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, base, inner_words, outer, box_inner, box_outer, CU_TENSOR_MAP_SWIZZLE_NONE);
}

FK_EXPORT int fk_gemm(fk_ctx* ctx, void* stream, fk_weight w, int mat, const float* x_dev, int m, float* out_dev) {
    if (!ctx || !w || !x_dev || !out_dev) return fk_fail(FK_INVALID, "gemm: null argument");
    if (m < 1) return fk_fail(FK_INVALID, "gemm: m=%d", m);
    if (mat < 0 || mat >= w->n_mats) return fk_fail(FK_INVALID, "gemm: matrix %d of %d", mat, w->n_mats);
    FkDeviceGuard g(ctx->device);
    return gemm_common(ctx, (cudaStream_t)stream, w, mat, nullptr, nullptr, x_dev, m, out_dev);
}

FK_EXPORT int fk_gemm_isums(fk_ctx* ctx, void* stream, fk_weight w, int mat, const float* x_dev, int m, float* out_dev, int32_t* isums_dev) {
    if (!ctx || !w || !x_dev || !out_dev || !isums_dev) return fk_fail(FK_INVALID, "gemm_isums: null argument");
    if (m < 1) return fk_fail(FK_INVALID, "gemm_isums: m=%d", m);
    if (mat < 0 || mat >= w->n_mats) return fk_fail(FK_INVALID, "gemm_isums: matrix %d of %d", mat, w->n_mats);
    FkDeviceGuard g(ctx->device);
    return gemm_common(ctx, (cudaStream_t)stream, w, mat, nullptr, nullptr, x_dev, m, out_dev, isums_dev);
}

FK_EXPORT int fk_gemm_plan(fk_ctx* ctx, fk_weight w, int m, int grouped, int* tile, int* split) {
    if (!ctx || !w || !tile || !split) return fk_fail(FK_INVALID, "gemm_plan: null argument");
    if (m < 1) return fk_fail(FK_INVALID, "gemm_plan: m=%d", m);
    const GemmPlan plan = gemm_plan(ctx, w, m, grouped != 0);
    *tile = plan.bn;
    *split = plan.split;
    return FK_OK;
}

FK_EXPORT int fk_gemm_tiled(fk_ctx* ctx, void* stream, fk_weight w, int mat, const int* group_off_dev, const int* gather_dev, const float* x_dev, int m,
                            float* out_dev, int32_t* isums_dev, int tile, int split) {
    if (!ctx || !w || !x_dev || !out_dev) return fk_fail(FK_INVALID, "gemm_tiled: null argument");
    if (m < 1) return fk_fail(FK_INVALID, "gemm_tiled: m=%d", m);
    if (mat < 0 || mat >= w->n_mats) return fk_fail(FK_INVALID, "gemm_tiled: matrix %d of %d", mat, w->n_mats);
    if (tile != 128 && tile != 64 && tile != 32) return fk_fail(FK_INVALID, "gemm_tiled: tile %d", tile);
    const int stages = (w->cols + KSTAGE - 1) / KSTAGE;
    if (split < 1 || split > MAX_SPLIT || (split & (split - 1)) || split > stages)
        return fk_fail(FK_INVALID, "gemm_tiled: %d parts of %d stages", split, stages);
    FkDeviceGuard g(ctx->device);
    const GemmPlan plan{tile, split};
    return gemm_common(ctx, (cudaStream_t)stream, w, mat, group_off_dev, gather_dev, x_dev, m, out_dev, isums_dev, &plan);
}

FK_EXPORT int fk_gemm_grouped(fk_ctx* ctx, void* stream, fk_weight w, const int* group_off_dev, const int* gather_dev,
                              const float* x_dev, int pairs, float* out_dev) {
    if (!ctx || !w || !group_off_dev || !x_dev || !out_dev) return fk_fail(FK_INVALID, "gemm_grouped: null argument");
    if (pairs < 1) return fk_fail(FK_INVALID, "gemm_grouped: pairs=%d", pairs);
    FkDeviceGuard g(ctx->device);
    return gemm_common(ctx, (cudaStream_t)stream, w, 0, group_off_dev, gather_dev, x_dev, pairs, out_dev);
}

// ---------------------------------------------------------------------------
// fk_gemm without any allocation.
//
// Some callers cannot allocate device memory at the moment they need a GEMM: a
// host thread that is inside a CUDA stream capture (cudaMalloc is not allowed
// there), a serving loop that must not hit the implicit device-wide
// synchronisation of cudaMalloc/cudaFree, or a process whose memory budget was
// handed out up front.  fk_gemm grows the context's scratch block on demand,
// so it is not for them.  This variant keeps its scratch (the int8 activation
// plane, the two scale planes and the row tables) in the fixed array below,
// which every GPU that loads this library holds from load to exit.
constexpr size_t FK_GEMM_STATIC_BYTES = 6u << 20;   // 6 MiB: e.g. 512 tokens x 8192 columns
static __device__ __align__(256) uint8_t fk_gemm_static_scratch[FK_GEMM_STATIC_BYTES];

namespace {
// In host code the array's name is only a handle; the device address comes from
// cudaGetSymbolAddress, asked once per device with that device current.
std::mutex g_static_mu;
uint8_t* g_static_ptr[64] = {nullptr};

int static_scratch(fk_ctx* ctx, uint8_t** out) {
    std::lock_guard<std::mutex> lk(g_static_mu);
    if (ctx->device < 0 || ctx->device >= 64) return fk_fail(FK_INVALID, "gemm_static: device %d", ctx->device);
    if (!g_static_ptr[ctx->device]) {
        void* p = nullptr;
        FK_CUDA(cudaGetSymbolAddress(&p, fk_gemm_static_scratch), FK_DRIVER_INIT);
        g_static_ptr[ctx->device] = (uint8_t*)p;
    }
    *out = g_static_ptr[ctx->device];
    return FK_OK;
}
}  // namespace

FK_EXPORT int fk_gemm_static(fk_ctx* ctx, void* stream, fk_weight w, int mat, const float* x_dev, int m, float* out_dev) {
    if (!ctx || !w || !x_dev || !out_dev) return fk_fail(FK_INVALID, "gemm_static: null argument");
    if (m < 1) return fk_fail(FK_INVALID, "gemm_static: m=%d", m);
    if (mat < 0 || mat >= w->n_mats) return fk_fail(FK_INVALID, "gemm_static: matrix %d of %d", mat, w->n_mats);
    FkDeviceGuard g(ctx->device);
    cudaStream_t st = (cudaStream_t)stream;
    if (w->kind == FK_Q5_K || w->kind == FK_BF16) return fk_fail(FK_UNSUPPORTED, "gemm: kind %d has no kernel", w->kind);
    // Sized for tiles of 128 tokens whatever tile the plan picks (narrower ones pad less), and with two words a padded row as
    // the row tables of the grouped form take: which shapes fit is part of the interface and does not follow the plan.
    const int n_most = (m + 127) / 128 * 128;
    const size_t most = GemmScratch(n_most, w->cols, 0, false).src + 8 * (size_t)n_most;
    if (most > FK_GEMM_STATIC_BYTES)
        return fk_fail(FK_INVALID, "gemm_static: %d tokens x %d columns needs %zu bytes of scratch, the fixed block holds %zu (use fk_gemm)",
                       m, w->cols, most, (size_t)FK_GEMM_STATIC_BYTES);
    uint8_t* sc = nullptr;
    int rc = static_scratch(ctx, &sc);
    if (rc) return rc;
    // Nothing in the block has to start at zero: the quantizer writes every word the GEMM reads (padding rows included)
    // before it reads them.
    const GemmPlan plan = gemm_plan(ctx, w, m, false);
    const int n_pad = (m + plan.bn - 1) / plan.bn * plan.bn;
    return gemm_run(ctx, st, w, mat, x_dev, m, out_dev, nullptr, plan, sc, GemmScratch(n_pad, w->cols, 0, false), n_pad, false);
}

// The error word kernels raise when a bounded wait gives up: 0 = none.
FK_EXPORT int fk_device_error(fk_ctx* ctx, int* code, int reset) {
    if (!ctx || !code) return fk_fail(FK_INVALID, "device_error: null argument");
    FkDeviceGuard g(ctx->device);
    FK_CUDA(cudaMemcpy(code, ctx->err_flag, sizeof(int), cudaMemcpyDeviceToHost), FK_LAUNCH);
    if (reset && *code) {
        FK_CUDA(cudaMemset(ctx->err_flag, 0, sizeof(int)), FK_LAUNCH);
        *ctx->err_pin = 0;
    }
    return FK_OK;
}
