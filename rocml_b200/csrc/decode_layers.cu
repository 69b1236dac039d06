// All layers of a decode step of a plain dense decoder in ONE persistent kernel (bfloat16, up to eight tokens, one of each
// sequence): norm, q | k | v, attention over the paged cache, output projection, norm, gate | up with SiLU, down.
//
// A step of a few tokens is bound by reading the weights once.  As five kernels a layer, each of which first waits for the one
// before, a hand-over costs the memory system 3 to 5 us of silence: the successor can hold little of its weight in shared
// memory while its predecessor still runs.  Here one block a multiprocessor stays for the whole step, and what a
// block will read is known in advance: a thread of its own (the producer) walks through ALL the block's share of weights and
// cached keys and values, layer after layer, and keeps a ring of 24 stages of 8 KB full, whatever the warps that compute are waiting
// for.  While the blocks meet between two phases 29 MB of the next phases' weights arrive, which is 4 us of the memory's time.
//
// Products: a unit is 16 rows of the weight (of gate | up 8 gate rows and the 8 up rows of the same outputs) over all of K, so a
// block finishes what it begins and no sums cross blocks; unit u of the step belongs to block u mod grid, counted on through
// all phases and layers, so that the blocks' shares even out over the phases.  A stage is a unit's 256 values of k, one TMA box; a warp
// takes one or two stages of every unit, always the same values of k, so its share of the activations stays in registers (up to 4,096
// values of k a pass).  (All eight warps at every stage: 340 cycles a stage, of which the memory needs 350 to bring it.)  The
// arithmetic is mma.sync m16n8k16 with the weight's rows as the 16 and the tokens as the 8: a tcgen05 tile would be 128 rows,
// and the products are bound by their bytes either way.
//
// Attention: an item is (sequence, key/value head, part of the pages); the ring brings 16 keys and values a stage, and the warps take
// the stages in turn.  Only keys of EARLIER steps come through the ring; the new token's
// key and value, made by the item with the sequence's last pages, are one more partial result in the merge and are written to the cache.
// More parts than one (long contexts) leave partial results in global memory, and the last to arrive merges them in order.
//
// Norms are deferred as in the kernels that this one stands for: a product that adds into the 32-bit residual stream also
// writes residual * weight in bfloat16 and the units' sums of squares; 1/RMS is applied to the next product's sums.
//
// What it costs: a meeting of the blocks is a release, a poll and the next operands, a round trip to the L2 cache each (0.5 us), and the chain of
// a unit's sums, 4 us in all; under it the weights' stream goes on.  A step, with the layers' own kernels and so, microseconds: 28 layers of 1,024
// (31 MB) with one token 758 -> 667, 28 of 2,048 with one 1,131 -> 937, 36 of 2,560 with four 2,114 -> 1,947, 36 of 4,096 (386 MB, 6.0 TB/s in gate | up) with one 2,961 ->
// 2,761, with eight 3,096 -> 3,058.
//
// Every wait is bounded.  A warp that gives up raises the block's flag and records RB_ERR_TIMEOUT; from then on no wait of
// the block waits, and everything else runs on as always (garbage, at addresses that do not depend on data), so that no barrier is ever
// short of a warp and no block of a partner.  The launch is cooperative: all blocks are resident or none is.
//
// Semantics of a layer: rocml/src/forward/mod.rs:281-340 (attention.rs:56-244, ffn.rs:57-107).
#include "common.cuh"
#include "mma_tiles.cuh"
#include "per_device.h"
#include "sm100.cuh"

using namespace rb;
using mma_tiles::ldmatrix_x4;
using mma_tiles::ldmatrix_x4_trans;
using mma_tiles::movmatrix_trans;
using mma_tiles::pack_bf16;
using mma_tiles::tile_addr;

namespace {
constexpr int CW = 8;                         // warps that compute
constexpr int CTHREADS = CW * 32;
constexpr int THREADS = CTHREADS + 128;       // and the producer's warpgroup, of which one thread works
constexpr int UR = 16;                        // weight rows of a unit
constexpr int KC = 256;                       // values of k of a stage
constexpr int KB = 64;                        // values of k of a row of 128 bytes, the swizzle's width
constexpr int STAGE = UR * KC * 2;            // [KC / 64][16 rows][128 bytes], swizzled
constexpr int STAGES = 24;                    // a multiple of CW, see Compute::attention
constexpr int GROUP = 6;                      // units whose sums are kept from pass to pass
constexpr int HD = 128;
constexpr int SK = 16;                        // keys of a stage
constexpr int MAX_G = 8;                      // query heads a key/value head
constexpr int MERGE_HEADS = 4;                // heads whose partial results are merged at a time
constexpr int TOK = 20;                       // floats between two tokens' 16 sums: free of bank conflicts
constexpr int MAX_LAYERS = 38;                // of a launch: what its parameters hold
constexpr float NEG_BIG = -1e30f;
constexpr float LOG2E = 1.4426950408889634f;
static_assert(STAGE == 2 * SK * HD * 2 && STAGES % CW == 0, "a stage holds 16 keys and 16 values");
constexpr int TT = 8;                         // tokens of the MMA's tile
constexpr int CPW = 2;                        // stages a warp takes of a unit: what it holds activations for (64 registers)

struct LayerPtrs {
    const void *ff_norm, *next_norm;                     // the norm behind the mixer, and the next layer's first (null: none)
    const void *q_norm, *k_norm;                         // [128] or null
    __nv_bfloat16 *k, *v;                                // [pages][heads][64][128]: where the new rows go
    float ff_eps, in_eps;                                // of ff_norm, and of the norm whose rows this layer's first product reads
};

// A layer's phases in order.  One loop runs through them, and every product is the same code (54 KB in all, 131 with a copy for each phase).
enum { QKV, ATTENTION, OUT, GATED, DOWN, PHASES };

// A phase's shape, worked out by the host.  Its units go to the blocks in turn: `each` to every one and one
// more to `rest` of them.  A unit's sum over k is taken in `passes` of at most `per` stages, as few as the warps' registers allow; in a
// pass `warps` warps share a unit, and `units` units are in work at a time (one where there are several passes).
struct Plan {
    int each, rest;                           // (attention: its items stay with the same blocks in every layer, see Item)
    int K, stages, passes, per, warps, units;
};

// A step as the kernel's code reads it: a copy in each block's shared memory.  (A read of the launch's parameters through the caches
// is a read of the L2 cache after every meeting of the blocks, whose acquire empties the L1 cache.)
struct Step {
    Plan plan[PHASES];
    int T, H, I, nq, nkv, layers, splits, max_pages;
    int norm_f32, head_norm_f32;
    float head_eps, scale, inv_T, inv_nkv, inv_H;
    const float2* cos_sin;          // [T][64] or null
    const int* seq_slot;
    const int* kv_len;
    const int* block_table;         // [slots][max_pages]
    const void* first_norm;         // the first layer's first norm (null: xhat and sumsq are there already)
    float* resid;                   // [T][H]
    __nv_bfloat16* xhat;            // [T][H] residual * weight, in the products' order of k (see `ordered`), as are attn and h
    float* sumsq;                   // [T][H / 16]
    float* qkv;                     // [T][(nq + 2 nkv) * 128]
    __nv_bfloat16* attn;            // [T][nq * 128]
    __nv_bfloat16* h;               // [T][I]
    float* part_o;                  // [T][nq][splits][128]
    float* part_ml;                 // [T][nq][splits][2]
    unsigned* counters;             // [1 + T * nkv], zero at launch: blocks that arrived, parts of a (sequence, head) that arrived
    int* status;
    unsigned wait_limit;            // clock cycles
    LayerPtrs layer[MAX_LAYERS];
};
struct Params {
    CUtensorMap map[MAX_LAYERS][6];                      // q | k | v, keys, output, gate | up, down (as the phases), values; see weight_map, rows_map
    Step step;
};
static_assert(sizeof(Params) <= 32764, "what a launch's parameters may hold");

__device__ __forceinline__ void load_unit(uint32_t dst, const CUtensorMap* map, int row, int kb, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %3, %5}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(0), "r"(row), "r"(kb) : "memory");
}
__device__ __forceinline__ void load_rows(uint32_t dst, const CUtensorMap* map, int row, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %3}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(0), "r"(row) : "memory");
}
// (Neither these nor what goes between them clobbers memory: the step's facts, which lie in shared memory, are then read once and not
// again for every load.  They are volatile, as the barriers are, and stay between them.)
__device__ __forceinline__ void load_if(bool yes, uint4& v, const void* p) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t@p ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
                 : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w) : "l"(p), "r"((int)yes));
}
__device__ __forceinline__ void load_if(bool yes, float& v, const void* p) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p ld.global.cg.f32 %0, [%1];\n\t}" : "+f"(v) : "l"(p), "r"((int)yes));
}
// Where value k of a row of activations lies.  A product's lane (gq, tq) needs words tq (two values) of the eight 16-byte chunks of 64 values
// as the B operands of four MMAs (the A operands come from ldmatrix, in the weight's own order); stored together, they are two loads.
__device__ __forceinline__ int ordered(int k) { return (k & ~63) | (k >> 1 & 3) << 4 | (k >> 3 & 7) << 1 | (k & 1); }
__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, %0;" ::"n"(CTHREADS) : "memory"); }
__device__ __forceinline__ unsigned load_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// (release at the device's scope: it covers what the block's other threads wrote before the barrier ahead of it)
__device__ __forceinline__ void add_release(unsigned* p) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}
// Element i of either type's vector: its bits as they are, and what they say (apart, so that the load need not be waited for in between)
__device__ __forceinline__ uint32_t bits_any(const void* p, int f32, int i) {
    return f32 ? static_cast<const uint32_t*>(p)[i] : static_cast<const uint16_t*>(p)[i];
}
__device__ __forceinline__ float value_any(uint32_t bits, int f32) { return __uint_as_float(f32 ? bits : bits << 16); }

struct Smem {
    uint8_t ring[STAGES][STAGE];
    union {
        float part[2][CW][TT][TOK];           // the warps' sums of the units in work, two rounds in turn
        float o[CW][MERGE_HEADS][HD];         // the warps' partial attention results
    };
    float keep[GROUP][TT][UR];                // sums of earlier passes
    __nv_bfloat16 q[8][HD];                   // query heads, swizzled rows
    __nv_bfloat16 k_new[HD], v_new[HD];
    float m[CW + 1][MAX_G], l[CW + 1][MAX_G]; // the warps' and the new key's maxima and sums
    float rstd[TT];
    uint64_t full[STAGES], empty[STAGES];
    Step step;
    int slot[TT], old[TT], page[TT];          // of every sequence: its slot, the keys of earlier steps, the new key's page
    int abort, last;
};
constexpr int SMEM = (int)sizeof(Smem);
static_assert(SMEM <= 227 * 1024, "a block's shared memory");

// What every warp keeps while it walks through the ring: producer and computing warps make the same steps in the same order.
struct Walk {
    int stage = 0;
    uint32_t phase = 0;
    int unit = 0;                             // units of the phases so far, modulo the grid
    __device__ void skip(int n) {             // n < STAGES
        stage += n;
        if (stage >= STAGES) { stage -= STAGES; phase ^= 1; }
    }
    __device__ void skip_any(int n) {
        phase ^= (n / STAGES) & 1;
        skip(n % STAGES);
    }
    // this block's first of a phase's units, and how many it has; the walk goes on to the next phase
    __device__ int share(const Plan& plan, int& first) {
        const int G = (int)gridDim.x;
        first = (int)blockIdx.x - unit;
        if (first < 0) first += G;
        unit += plan.rest;
        if (unit >= G) unit -= G;
        return plan.each + (first < plan.rest ? 1 : 0);
    }
};

// Waits of one block: none waits any more once one of them has run out.
struct Waits {
    volatile int* abort;
    int* status;
    unsigned limit;
    __device__ bool gave_up() const { return *abort != 0; }
    // whether a wait that began at t0 is to end without success
    __device__ bool over(unsigned t0) const {
        if (gave_up()) return true;
        if ((unsigned)clock() - t0 <= limit) return false;
        *abort = 1;
        atomicExch(status, RB_ERR_TIMEOUT);
        return true;
    }
    __device__ bool barrier(uint64_t* bar, uint32_t parity) const {
        if (sm100::mbar_try_wait(bar, parity)) return true;
        const unsigned t0 = (unsigned)clock();
        while (!sm100::mbar_try_wait(bar, parity))
            if (over(t0)) return false;
        return true;
    }
};

// The first row of unit u.  Gate | up alternate in blocks of 16 rows: its other eight rows lie 16 further down, in place of 8.
__device__ __forceinline__ int weight_row(int phase, int u) { return phase == GATED ? (u >> 1) * 32 + (u & 1) * 8 : u * UR; }

// An item of attention: block b has items b, b + grid, .. in every layer.  Sequence, key/value head and part (a whole number below 2^20
// over a small one: exact in 32-bit), the keys of earlier steps (below 0: nobody's place), and of those this item's: its pages and keys.
struct Item {
    int b, head, part, old, p0, p1, key1;
    template <class S>
    __device__ void find(const S& s, int item) {
        const Step& p = s.step;
        const int pair = (int)(((float)item + 0.5f) * p.inv_T);
        b = item - pair * p.T;
        part = p.splits == 1 ? 0 : (int)(((float)pair + 0.5f) * p.inv_nkv);
        head = pair - part * p.nkv;
        old = s.slot[b] < 0 ? -1 : s.old[b];
        const int pages = (max(old, 0) + RB_PAGE - 1) / RB_PAGE;
        p0 = 0; p1 = pages;
        if (p.splits > 1) { p0 = part * pages / p.splits; p1 = (part + 1) * pages / p.splits; }
        key1 = min(max(old, 0), p1 * RB_PAGE);
    }
};

// ---- the producer ------------------------------------------------------------------------------------------
// One thread walks, so that a stage costs a few instructions (a warp in step, with an arrival each: 340 to 460 cycles a stage, which set the
// pace of the whole step).
struct Producer {
    Smem& s;
    Walk w;
    Waits waits;
    int issued = 0;

    __device__ Producer(Smem& s, Waits waits) : s(s), waits(waits) {}

    // The next stage is free, and its barrier knows what will land in it; false: given up.  (Once a wait has run out no
    // stage is handed back, see Compute::taken, so that none is armed while a copy into it may be on its way, and the drain at the end
    // finds each copy's own phase.)
    __device__ bool room() {
        if (!waits.barrier(&s.empty[w.stage], w.phase ^ 1)) return false;
        sm100::mbar_arrive_expect_tx(&s.full[w.stage], STAGE);         // (beyond K and beyond the cache's rows zeros arrive)
        ++issued;
        return true;
    }
    // What nobody has read since the step before is asked into the L2 cache.
    __device__ static void prefetch(const void* p, int bytes) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const uint8_t*>(p) + bytes));
    }

    __device__ void product(const Step& p, const CUtensorMap* weight, const LayerPtrs& L, int phase) {
        int first;
        const Plan& ps = p.plan[phase];
        const int mine = w.share(ps, first);
        const void* norm = phase == OUT ? L.ff_norm : (phase == DOWN ? L.next_norm : nullptr);
        const int group = ps.passes == 1 ? mine : GROUP;
#pragma unroll 1
        for (int g0 = 0; g0 < mine; g0 += group)
#pragma unroll 1
            for (int pass = 0; pass < ps.passes; ++pass)
#pragma unroll 1
                for (int u = g0; u < min(mine, g0 + group); ++u) {
                    const int row = weight_row(phase, first + u * (int)gridDim.x);
                    if (norm != nullptr && pass == 0) prefetch(norm, row * (p.norm_f32 ? 4 : 2));
                    const int end = min(ps.stages, (pass + 1) * ps.per) * (KC / KB);
#pragma unroll 1
                    for (int kb = pass * ps.per * (KC / KB); kb < end; kb += KC / KB) {
                        if (!room()) return;
                        load_unit(sm100::smem_u32(s.ring[w.stage]), weight, row, kb, sm100::smem_u32(&s.full[w.stage]));
                        w.skip(1);
                    }
                }
    }

    __device__ void keys(const Step& p, const CUtensorMap* maps, const LayerPtrs& L, const Item& mine) {
        const int items = p.T * p.nkv * p.splits;
        if (L.q_norm != nullptr && (int)blockIdx.x < items) {
            const int half = p.head_norm_f32 ? 256 : 128;
            prefetch(L.q_norm, 0); prefetch(L.q_norm, half); prefetch(L.k_norm, 0); prefetch(L.k_norm, half);
        }
        Item it = mine;
#pragma unroll 1
        for (int item = blockIdx.x; item < items; item += gridDim.x) {
            if (item != (int)blockIdx.x) it.find(s, item);
            if (it.old <= 0) continue;
            const int* table = p.block_table + (size_t)s.slot[it.b] * p.max_pages;
            int next = it.p0 < it.p1 ? table[it.p0] : 0;
#pragma unroll 1
            for (int pg = it.p0; pg < it.p1; ++pg) {
                const int row = (max(next, 0) * p.nkv + it.head) * RB_PAGE;
                next = table[min(pg + 1, it.p1 - 1)];                    // (a page ahead of its use)
                const int rows = min(RB_PAGE, it.old - pg * RB_PAGE);
#pragma unroll 1
                for (int r = 0; r < rows; r += SK) {
                    if (!room()) return;
                    const uint32_t to = sm100::smem_u32(s.ring[w.stage]), bar = sm100::smem_u32(&s.full[w.stage]);
                    load_rows(to, maps + ATTENTION, row + r, bar);
                    load_rows(to + STAGE / 2, maps + PHASES, row + r, bar);
                    w.skip(1);
                }
            }
        }
    }

    __device__ void run(const Step& p, const Params& params) {
        Item first;
        first.find(s, blockIdx.x);
#pragma unroll 1
        for (int i = 0; i < p.layers * PHASES && !waits.gave_up(); ++i) {
            const LayerPtrs& L = p.layer[i / PHASES];
            const CUtensorMap* maps = params.map[i / PHASES];
            const int phase = i % PHASES;
            if (phase == ATTENTION) keys(p, maps, L, first);
            else product(p, maps + phase, L, phase);
        }
        // The last copies land before the block's memory goes, whatever the warps that compute have waited for (a limit of its own:
        // once a wait has run out the others no longer wait).
        for (int i = 0; i < min(issued, STAGES); ++i) {
            if (w.stage == 0) { w.stage = STAGES; w.phase ^= 1; }
            --w.stage;
            sm100::mbar_wait(&s.full[w.stage], w.phase, sm100::RB_WAIT_CYCLES);
        }
    }
};

// ---- the warps that compute -----------------------------------------------------------------------------------
struct Compute {
    Smem& s;
    Walk w;
    Waits waits;
    const Step& p;
    unsigned met = 0;                         // arrivals that complete the meeting before this one
    unsigned turn = 0;                        // rounds of units summed so far: which half of s.part
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;

    __device__ Compute(Smem& s, Waits waits) : s(s), waits(waits), p(s.step) {}

    // The stage's copy has landed (or a wait has run out); and whether the stage may be handed back when it has been read: not once a wait
    // has run out, since the copy may then still be on its way.  Two uses of a stage are the same warp's or have a barrier of the
    // warps between them, so a wait that a given-up stage's parity lets pass finds the flag raised.  (The producer, one thread at
    // the ring's pace, looking at the flag for every stage instead: 0.6 to 1.4 % slower at 0.6b sizes and 1.7b with eight sequences.)
    __device__ bool taken(const Walk& at) {
        waits.barrier(&s.full[at.stage], at.phase);
        return !waits.gave_up();
    }
    __device__ void give_back(const Walk& at, bool whole) {
        __syncwarp();
        if (lane == 0 && whole) sm100::mbar_arrive(&s.empty[at.stage]);
    }

    // Every block has come this far, and what it wrote is visible (read it past the L1 cache).  In two halves: what the next phase needs to
    // know of itself is worked out between them.
    __device__ void arrive() {
        compute_sync();
        met += gridDim.x;
        if (threadIdx.x == 0) add_release(p.counters);
    }
    __device__ void wait() {
        if (threadIdx.x == 0) {
            const unsigned t0 = (unsigned)clock();
            while ((int)(load_acquire(p.counters) - met) < 0 && !waits.over(t0)) {}
        }
        compute_sync();
    }

    // 1/RMS of every token's row, from the units' sums of squares: a warp a token.  The loads of the first 256 units
    // go out ahead of the first unit's products, the sums follow behind them.
    struct Squares { float v[8]; };
    __device__ void ask_squares(Squares& q) {
        const int n = p.H / UR, T = p.T;
        const float* from = p.sumsq + (warp * n + lane);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            q.v[j] = 0.f;
            load_if(warp < T && j * 32 + lane < n, q.v[j], from + j * 32);
        }
    }
    __device__ void row_scales(const Squares& q, float eps) {
        const int n = p.H / UR;
        if (warp < p.T) {
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 8; ++j) sum += q.v[j];
#pragma unroll 1
            for (int u = 256 + lane; u < n; u += 32) sum += __ldcg(p.sumsq + (warp * n + u));
            sum = warp_sum(sum);
            if (lane == 0) s.rstd[warp] = rsqrtf(sum * p.inv_H + eps);
        }
    }

    // What a unit's sums become: what the thread of row r and token t needs for that, looked up once a phase.
    struct Out {
        int phase, H;
        bool live, next;           // the token exists; a norm follows
        const void* norm;          // its weights
        float* f32;                // QKV: the token's row of the projections, otherwise of the stream
        __nv_bfloat16* bf16;       // GATED: the token's row of h, otherwise of xhat
        float* sumsq;
        float before;
        uint32_t weight;
    };
    __device__ Out output(int phase, const void* norm, int t) {
        Out o;
        o.phase = phase; o.H = p.H; o.live = t < p.T; o.next = norm != nullptr; o.norm = norm;
        o.f32 = phase == QKV ? p.qkv + t * ((p.nq + 2 * p.nkv) * HD) : p.resid + t * p.H;
        o.bf16 = phase == GATED ? p.h + t * p.I : p.xhat + t * p.H;
        o.sumsq = p.sumsq + t * (p.H / UR);
        o.before = 0.f; o.weight = 0u;
        return o;
    }
    // ahead of the unit's last stages
    __device__ void begin(Out& o, int u, int r) {
        if (o.phase != OUT && o.phase != DOWN) return;
        load_if(o.live, o.before, o.f32 + (u * UR + r));
        if (o.next) o.weight = bits_any(o.norm, p.norm_f32, u * UR + r);
    }
    // x: the stream's new value at column u * 16 + r: kept, and the next norm's rows and sums of squares
    __device__ void to_stream(const Out& o, int u, int r, float x, bool keep) {
        float sq = x * x;
#pragma unroll
        for (int d = 8; d > 0; d >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, d);
        if (o.live) {
            if (keep) o.f32[u * UR + r] = x;
            if (o.next) {
                o.bf16[ordered(u * UR + r)] = __float2bfloat16_rn(x * value_any(o.weight, p.norm_f32));
                if (r == 0) o.sumsq[u] = sq;
            }
        }
    }
    // the sum is there (whole warps: 16 rows of two tokens each)
    __device__ void finish(const Out& o, int u, int t, int r, float sum) {
        if (o.phase == OUT || o.phase == DOWN) {
            to_stream(o, u, r, o.before + sum, true);
            return;
        }
        const float v = sum * s.rstd[t];
        if (o.phase == QKV) {
            if (o.live) o.f32[u * UR + r] = v;
        } else {                              // SiLU(gate) * up: rows 0..7 and 8..15 of the unit
            const float up = __shfl_down_sync(0xffffffffu, v, 8, 16);
            if (r < 8 && o.live) o.bf16[ordered(u * 8 + r)] = __float2bfloat16_rn(silu(v) * up);
        }
    }
    // The first layer's first norm: the stream's rows times its weight, and their sums of squares
    __device__ void first_rows() {
        const int t = threadIdx.x >> 4, r = threadIdx.x & 15;
        Out o = output(DOWN, p.first_norm, t);
#pragma unroll 1
        for (int u = blockIdx.x; u < p.H / UR; u += gridDim.x) {
            begin(o, u, r);
            to_stream(o, u, r, o.before, false);
        }
    }

    // A product of the step's rows [T][K] with this block's units: which, and where this thread's share of everything is.  (The plan stays in
    // shared memory: a copy in registers made steps of 2,560 wide layers 4 % slower.)
    struct Job {
        int phase;
        int first, mine, group, my_unit, my_stage;      // (unit and stage of those in work)
        bool scaled;
        float eps;
        const __nv_bfloat16* row;
        Out out;
    };
    __device__ void prepare(Job& job, int i) {
        const LayerPtrs& L = p.layer[i / PHASES];
        const int phase = i % PHASES, T = p.T;
        const Plan& ps = p.plan[phase];
        job.phase = phase;
        job.mine = w.share(ps, job.first);
        job.group = ps.passes == 1 ? job.mine : GROUP;
        job.my_unit = warp / ps.warps;
        job.my_stage = (warp - job.my_unit * ps.warps) * CPW;
        job.scaled = phase == QKV || phase == GATED;
        job.eps = phase == QKV ? L.in_eps : L.ff_eps;
        const __nv_bfloat16* x = phase == OUT ? p.attn : (phase == DOWN ? p.h : p.xhat);
        job.row = x + (min(gq, T - 1) * ps.K + job.my_stage * KC + tq * 16);
        job.out = output(phase, phase == OUT ? L.ff_norm : L.next_norm, threadIdx.x / UR % TT);
    }

    __device__ void product(Job& job) {
        constexpr int C = CPW, OUTS = UR * TT, A = 4;
        const Plan& ps = p.plan[job.phase];
        const int first = job.first, mine = job.mine, group = job.group, my_unit = job.my_unit, my_stage = job.my_stage, K = ps.K;
        // the lane's row of the four 8 x 8 matrices of a 16 x 16 A operand: rows 0..7 and 8..15 of two neighbouring chunks
        const uint32_t lane_ring = sm100::smem_u32(s.ring[0]) + (lane & 15) * 128 + (((lane >> 4) ^ (lane & 7)) << 4);
        // who sums what: a thread row r of token t of one of the units in work, and (short sums) of the next but one
        const int r = threadIdx.x & 15, t = threadIdx.x / UR % TT;
        Out& out = job.out;
#pragma unroll 1
        for (int g0 = 0; g0 < mine; g0 += group)
#pragma unroll 1
            for (int pass = 0; pass < ps.passes; ++pass) {
                const int c0 = pass * ps.per, nc = min(ps.stages - c0, ps.per);
                // This warp's share of the activations, as the B operands of four MMAs a block of 64 values of k (see `ordered`).  Columns of
                // the tile beyond the last token repeat it and are dropped.
                const int blocks = (min(nc, my_stage + C) - my_stage) * (KC / KB);
                const int nb = min(blocks, K / KB - (c0 + my_stage) * (KC / KB));
                uint4 B[C * (KC / KB)][2];
                const __nv_bfloat16* row = job.row + c0 * KC;
#pragma unroll
                for (int j = 0; j < C * (KC / KB); ++j)
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        B[j][half] = make_uint4(0u, 0u, 0u, 0u);
                        load_if(j < nb, B[j][half], row + j * KB + half * 8);
                    }
                bool scales = job.scaled && g0 == 0 && pass == 0;
                Squares squares;
                if (scales) ask_squares(squares);
                const bool last = pass == ps.passes - 1;
                const int end = min(mine, g0 + group);
#pragma unroll 1
                for (int i = g0; i < end; i += ps.units) {
                    const int units = min(ps.units, end - i);
                    int unit = threadIdx.x / OUTS;
                    if (last && unit < units) begin(out, first + (i + unit) * (int)gridDim.x, r);
                    float acc[A][4];                          // A chains of MMAs, added at the end
#pragma unroll
                    for (int k = 0; k < A * 4; ++k) acc[k >> 2][k & 3] = 0.f;
                    if (my_unit < units) {
                        Walk at = w;
                        at.skip(my_unit * nc + my_stage);
#pragma unroll
                        for (int c = 0; c < C; ++c)
                            if (my_stage + c < nc) {
                                const bool whole = taken(at);
                                const uint32_t a = lane_ring + at.stage * STAGE;
                                // a block's four operands are loaded while the block before is multiplied
                                uint32_t m[2][4][4];
#pragma unroll
                                for (int j = 0; j <= KC / KB; ++j) {
                                    if (j < KC / KB && c * (KC / KB) + j < nb)
#pragma unroll
                                        for (int k = 0; k < 4; ++k)
                                            ldmatrix_x4((a ^ (k * 32)) + j * (UR * 128), m[j & 1][k][0], m[j & 1][k][1], m[j & 1][k][2], m[j & 1][k][3]);
                                    if (j > 0 && c * (KC / KB) + j - 1 < nb)
#pragma unroll
                                        for (int k = 0; k < 4; ++k) {
                                            const uint4 b = B[c * (KC / KB) + (j > 0 ? j - 1 : 0)][k >> 1];
                                            mma_tiles::mma_bf16(acc[k % A], m[(j & 1) ^ 1][k], k & 1 ? b.z : b.x, k & 1 ? b.w : b.y);
                                        }
                                }
                                give_back(at, whole);
                                at.skip(1);
                            }
                        // the warps' sums meet; the other half of s.part is free: its readers have passed this barrier's predecessor
                        float* to = &s.part[turn & 1][warp][tq * 2][gq];
#pragma unroll
                        for (int a = 2; a < A; ++a)
#pragma unroll
                            for (int k = 0; k < 4; ++k) acc[a & 1][k] += acc[a][k];
                        to[0] = acc[0][0] + acc[1][0];
                        to[TOK] = acc[0][1] + acc[1][1];
                        to[8] = acc[0][2] + acc[1][2];
                        to[TOK + 8] = acc[0][3] + acc[1][3];
                    }
                    if (scales) row_scales(squares, job.eps);
                    scales = false;
                    // (behind this barrier every warp has left the stages of the round, which are fewer than the ring's: what a warp waits
                    // for next is at most one use of a stage away, so that its parity says which)
                    w.skip(units * nc);
                    compute_sync();
#pragma unroll 1
                    for (; unit < units; unit += CTHREADS / OUTS) {
                        const float* from = &s.part[turn & 1][unit * ps.warps][t][r];
                        float sum = 0.f;
#pragma unroll
                        for (int k = 0; k < CW; ++k)
                            if (k < ps.warps) sum += from[k * (TT * TOK)];
                        if (ps.passes > 1) {
                            float* kept = &s.keep[i - g0][t][r];
                            if (pass > 0) sum += *kept;
                            if (!last) *kept = sum;
                        }
                        if (last) {
                            const int u = first + (i + unit) * (int)gridDim.x;
                            if (unit >= CTHREADS / OUTS) begin(out, u, r);
                            finish(out, u, t, r, sum);
                        }
                    }
                    ++turn;
                }
            }
    }

    // ---- attention ----
    // One head of 128 values by half a warp: lane i of 16 holds 4 i .. 4 i + 3 and 64 + 4 i .. of it.
    __device__ void head(const float* src, bool value, const void* weight, int t, float* v) {
        const int i = lane & 15;
        const float4 lo = __ldcg(reinterpret_cast<const float4*>(src + i * 4)), hi = __ldcg(reinterpret_cast<const float4*>(src + 64 + i * 4));
        float4 cs[2] = {make_float4(1.f, 0.f, 1.f, 0.f), make_float4(1.f, 0.f, 1.f, 0.f)};
        if (!value && p.cos_sin != nullptr) {
            const float4* c = reinterpret_cast<const float4*>(p.cos_sin + t * 64 + i * 4);
            cs[0] = c[0]; cs[1] = c[1];
        }
        float wj[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) wj[j] = 1.f;
        if (!value && weight != nullptr) {
            load4_any(weight, p.head_norm_f32, i * 4, wj);
            load4_any(weight, p.head_norm_f32, 64 + i * 4, wj + 4);
        }
        v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
        v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += v[j] * v[j];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (!value && weight != nullptr) {
            const float inv = rsqrtf(ss * (1.f / 128.f) + p.head_eps);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = v[j] * inv * wj[j];
        }
        if (!value && p.cos_sin != nullptr) {
            const float c[4] = {cs[0].x, cs[0].z, cs[1].x, cs[1].z}, sn[4] = {cs[0].y, cs[0].w, cs[1].y, cs[1].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float a = v[j], b = v[4 + j];
                v[j] = a * c[j] - b * sn[j];
                v[4 + j] = a * sn[j] + b * c[j];
            }
        }
    }

    __device__ static uint2 pack4(const float* v) { return make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3])); }

    __device__ void attention(const LayerPtrs& L, const Item& mine, int g) {
        const int items = p.T * p.nkv * p.splits, width = (p.nq + 2 * p.nkv) * HD;
        Item it = mine;
#pragma unroll 1
        for (int item = blockIdx.x; item < items; item += gridDim.x) {
            if (item != (int)blockIdx.x) it.find(s, item);
            const int b = it.b, kvh = it.head, part = it.part, old = it.old;
            if (old < 0) {
                // a place without a sequence: zeros, so that the products behind it stay finite
                if (part == 0)
#pragma unroll 1
                    for (int i = threadIdx.x; i < g * HD; i += CTHREADS) p.attn[(b * p.nq + kvh * g) * HD + i] = __float2bfloat16_rn(0.f);
                continue;
            }
            const int key0 = it.p0 * RB_PAGE, key1 = it.key1;
            const bool owner = part == p.splits - 1;                     // makes the new key and value
            compute_sync();                                             // the item before is done with s.q and s.o
            {
                const int task = warp * 2 + (lane >> 4), sub = lane & 15;
                const int kind = task < g ? 0 : task - g + 1;            // query, key, value; beyond: nothing
                const bool real = kind == 0 || (owner && kind <= 2);
                const int col = kind == 0 ? kvh * g + task : (kind == 1 ? p.nq + kvh : p.nq + p.nkv + kvh);
                float v[8];
                head(p.qkv + (b * width + (real ? col : 0) * HD), real && kind == 2, kind == 1 ? L.k_norm : L.q_norm, b, v);
                if (real) {
                    const uint2 lo = pack4(v), hi = pack4(v + 4);
                    if (kind == 0) {
                        uint8_t* row = reinterpret_cast<uint8_t*>(s.q[task]);
                        *reinterpret_cast<uint2*>(row + (((sub >> 1) ^ (task & 7)) << 4) + (sub & 1) * 8) = lo;
                        *reinterpret_cast<uint2*>(row + (((8 + (sub >> 1)) ^ (task & 7)) << 4) + (sub & 1) * 8) = hi;
                    } else {
                        __nv_bfloat16* to = kind == 1 ? s.k_new : s.v_new;
                        *reinterpret_cast<uint2*>(to + sub * 4) = lo;
                        *reinterpret_cast<uint2*>(to + 64 + sub * 4) = hi;
                        const int page = s.page[b];
                        if (page >= 0) {
                            __nv_bfloat16* out = (kind == 1 ? L.k : L.v) + (((size_t)page * p.nkv + kvh) * RB_PAGE + old % RB_PAGE) * HD;
                            *reinterpret_cast<uint2*>(out + sub * 4) = lo;
                            *reinterpret_cast<uint2*>(out + 64 + sub * 4) = hi;
                        }
                    }
                }
            }
            compute_sync();
            const float sl2 = p.scale * LOG2E;
            uint32_t qb[HD / 16][2];                                     // the query heads as the B operand
            const uint32_t q_base = sm100::smem_u32(s.q);
#pragma unroll
            for (int ks = 0; ks < HD / 16; ks += 2)
                ldmatrix_x4(tile_addr<HD>(q_base, lane & 7, ks * 2 + (lane >> 3)), qb[ks][0], qb[ks][1], qb[ks + 1][0], qb[ks + 1][1]);
            // transposed products: 16 keys as rows, heads as the 8 columns; O^T has the head size as rows
            float mx_w[2] = {NEG_BIG, NEG_BIG}, l_w[2] = {0.f, 0.f}, ot[HD / 16][4];
#pragma unroll
            for (int i = 0; i < HD / 16; ++i) { ot[i][0] = ot[i][1] = ot[i][2] = ot[i][3] = 0.f; }
            // Stage i of the item is warp i % 8's.  The ring's length is a multiple of 8, so that a stage that comes round again within the item
            // is the same warp's: a parity is never two uses away.
            // (keys, then values, each as two halves of the head, [16 rows][128 bytes], swizzled)
            const uint32_t k_lane = sm100::smem_u32(s.ring[0]) + (lane & 15) * 128 + (((lane >> 4) ^ (lane & 7)) << 4);
            const uint32_t v_lane = sm100::smem_u32(s.ring[0]) + STAGE / 2 + ((lane & 7) + (lane >> 4) * 8) * 128 + (((lane >> 3 & 1) ^ (lane & 7)) << 4);
            const int n_stages = (max(key1 - key0, 0) + SK - 1) / SK;
            Walk at = w;
            at.skip(warp);
            w.skip_any(n_stages);
#pragma unroll 1
            for (int i = warp; i < n_stages; i += CW) {
                const bool whole = taken(at);
                const int j0 = key0 + i * SK;
                const uint32_t kt = k_lane + at.stage * STAGE, vt = v_lane + at.stage * STAGE;
                const bool ragged = j0 + SK > key1;
                if (ragged) {
                    // the rows behind the last key: whatever the page held there must not meet a weight of zero
#pragma unroll 1
                    for (int x = lane; x < (j0 + SK - key1) * 16; x += 32)
                        *reinterpret_cast<uint4*>(s.ring[at.stage] + STAGE / 2 + (x & 1) * (STAGE / 4) + (key1 - j0 + (x >> 4)) * 128 + (x >> 1 & 7) * 16) =
                            make_uint4(0u, 0u, 0u, 0u);
                    __syncwarp();
                }
                float st[4] = {0.f, 0.f, 0.f, 0.f}, st2[4] = {0.f, 0.f, 0.f, 0.f};
                uint32_t va[HD / 16][4];
                {
                    uint32_t ka[HD / 16][4];
#pragma unroll
                    for (int k = 0; k < HD / 16; ++k)
                        ldmatrix_x4((kt ^ ((k & 3) * 32)) + (k >> 2) * (STAGE / 4), ka[k][0], ka[k][1], ka[k][2], ka[k][3]);
#pragma unroll
                    for (int k = 0; k < HD / 16; ++k)
                        ldmatrix_x4_trans((vt ^ ((k & 3) * 32)) + (k >> 2) * (STAGE / 4), va[k][0], va[k][1], va[k][2], va[k][3]);
#pragma unroll
                    for (int k = 0; k < HD / 16; ++k) mma_tiles::mma_bf16(k & 1 ? st2 : st, ka[k], qb[k][0], qb[k][1]);
                }
                const bool ok0 = j0 + gq < key1, ok1 = j0 + gq + 8 < key1;
                st[0] = ok0 ? (st[0] + st2[0]) * sl2 : -INFINITY;
                st[1] = ok0 ? (st[1] + st2[1]) * sl2 : -INFINITY;
                st[2] = ok1 ? (st[2] + st2[2]) * sl2 : -INFINITY;
                st[3] = ok1 ? (st[3] + st2[3]) * sl2 : -INFINITY;
                float alpha[2];
#pragma unroll
                for (int r = 0; r < 2; ++r) {                        // a head's keys lie along the lanes' groups
                    float mx = fmaxf(st[r], st[r + 2]);
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                    const float m_new = fmaxf(mx_w[r], mx);
                    alpha[r] = ex2(mx_w[r] - m_new);
                    mx_w[r] = m_new;
                    l_w[r] *= alpha[r];
                }
#pragma unroll
                for (int k = 0; k < HD / 16; ++k) {
                    ot[k][0] *= alpha[0]; ot[k][1] *= alpha[1];
                    ot[k][2] *= alpha[0]; ot[k][3] *= alpha[1];
                }
                const float e0 = ex2(st[0] - mx_w[0]), e1 = ex2(st[1] - mx_w[1]);
                const float e2 = ex2(st[2] - mx_w[0]), e3 = ex2(st[3] - mx_w[1]);
                l_w[0] += e0 + e2;
                l_w[1] += e1 + e3;
                const uint32_t pb0 = movmatrix_trans(pack_bf16(e0, e1)), pb1 = movmatrix_trans(pack_bf16(e2, e3));
#pragma unroll
                for (int k = 0; k < HD / 16; ++k) mma_tiles::mma_bf16(ot[k], va[k], pb0, pb1);
                if (ragged) sm100::fence_proxy_async();                  // (the copy engine writes there next)
                give_back(at, whole);
                at.skip(CW);
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                l_w[r] += __shfl_xor_sync(0xffffffffu, l_w[r], 4);
                l_w[r] += __shfl_xor_sync(0xffffffffu, l_w[r], 8);
                l_w[r] += __shfl_xor_sync(0xffffffffu, l_w[r], 16);
                if (gq == 0) { s.m[warp][tq * 2 + r] = mx_w[r]; s.l[warp][tq * 2 + r] = l_w[r]; }
            }
            if (warp < g) {                                              // the new key, a warp a head
                float m_new = NEG_BIG;
                if (owner) {
                    const uint2 a = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint8_t*>(s.q[warp]) +
                                                                    (((lane >> 1) ^ (warp & 7)) << 4) + (lane & 1) * 8);
                    float qv[4], kv[4];
                    load4(reinterpret_cast<const __nv_bfloat16*>(&a), qv);
                    load4(s.k_new + lane * 4, kv);
                    m_new = warp_sum(qv[0] * kv[0] + qv[1] * kv[1] + qv[2] * kv[2] + qv[3] * kv[3]) * sl2;
                }
                if (lane == 0) { s.m[CW][warp] = m_new; s.l[CW][warp] = owner ? 1.f : 0.f; }
            }
            const int row0 = b * p.nq + kvh * g;                         // this group's first query head, over all sequences
#pragma unroll 1
            for (int h0 = 0; h0 < g; h0 += MERGE_HEADS) {
                if (h0 > 0) compute_sync();
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int hh = tq * 2 + r - h0;
                    if (hh >= 0 && hh < MERGE_HEADS && hh + h0 < g)
#pragma unroll
                        for (int i = 0; i < HD / 16; ++i) {
                            s.o[warp][hh][i * 16 + gq] = ot[i][r];
                            s.o[warp][hh][i * 16 + gq + 8] = ot[i][r + 2];
                        }
                }
                compute_sync();
#pragma unroll 1
                for (int idx = threadIdx.x; idx < min(MERGE_HEADS, g - h0) * HD; idx += CTHREADS) {
                    const int r = idx / HD + h0, d = idx % HD;
                    float M = NEG_BIG;
#pragma unroll
                    for (int k = 0; k <= CW; ++k) M = fmaxf(M, s.m[k][r]);
                    float sum = 0.f, A = 0.f;
#pragma unroll
                    for (int k = 0; k <= CW; ++k) {
                        const float wt = ex2(s.m[k][r] - M);             // a warp that saw no key has l = 0 and o = 0
                        sum = fmaf(wt, s.l[k][r], sum);
                        A = fmaf(wt, k < CW ? s.o[k < CW ? k : 0][r - h0][d] : (owner ? __bfloat162float(s.v_new[d]) : 0.f), A);
                    }
                    if (p.splits == 1) {
                        p.attn[ordered((row0 + r) * HD + d)] = __float2bfloat16_rn(A / sum);
                    } else {
                        p.part_o[((row0 + r) * p.splits + part) * HD + d] = A;
                        if (d == 0) *reinterpret_cast<float2*>(p.part_ml + ((row0 + r) * p.splits + part) * 2) = make_float2(M, sum);
                    }
                }
            }
            if (p.splits > 1) {
                compute_sync();
                if (threadIdx.x == 0) {
                    unsigned before;
                    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(p.counters + 1 + b * p.nkv + kvh) : "memory");
                    s.last = (before + 1) % (unsigned)p.splits == 0;      // (every layer adds `splits`)
                }
                compute_sync();
                if (s.last)
#pragma unroll 1
                    for (int idx = threadIdx.x; idx < g * HD; idx += CTHREADS) {
                        const int r = idx / HD, d = idx % HD;
                        const float2* ml = reinterpret_cast<const float2*>(p.part_ml) + (row0 + r) * p.splits;
                        const float* o = p.part_o + (row0 + r) * p.splits * HD + d;
                        float M = NEG_BIG, sum = 0.f, A = 0.f;
#pragma unroll 1
                        for (int k0 = 0; k0 < p.splits; k0 += 8) {           // eight parts' loads in flight
                            float2 x[8];
                            float a[8];
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                x[k] = k0 + k < p.splits ? __ldcg(ml + k0 + k) : make_float2(NEG_BIG, 0.f);
                                a[k] = k0 + k < p.splits ? __ldcg(o + (k0 + k) * HD) : 0.f;
                            }
                            float top = M;
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                                if (x[k].y > 0.f) top = fmaxf(top, x[k].x);
                            const float old_wt = ex2(M - top);
                            sum *= old_wt; A *= old_wt; M = top;
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                const float wt = x[k].y > 0.f ? ex2(x[k].x - M) : 0.f;
                                sum = fmaf(wt, x[k].y, sum);
                                A = fmaf(wt, a[k], A);
                            }
                        }
                        p.attn[ordered((row0 + r) * HD + d)] = __float2bfloat16_rn(A / sum);
                    }
            }
        }
    }

    __device__ void run() {
        Item mine;
        mine.find(s, blockIdx.x);
        const int g = p.nq / p.nkv;
        Job job;
        if (p.first_norm != nullptr) {
            first_rows();
            arrive();
            prepare(job, 0);
            wait();
        } else {
            prepare(job, 0);
        }
        const int n = p.layers * PHASES;
#pragma unroll 1
        for (int i = 0; i < n; ++i) {
            if (i % PHASES == ATTENTION) attention(p.layer[i / PHASES], mine, g);
            else product(job);
            if (i + 1 < n) {
                arrive();
                if ((i + 1) % PHASES != ATTENTION) prepare(job, i + 1);
                wait();
            }
        }
    }
};

__global__ void __launch_bounds__(THREADS, 1) decode_layers_kernel(const __grid_constant__ Params params) {
    extern __shared__ __align__(1024) uint8_t raw[];
    Smem& s = *reinterpret_cast<Smem*>(raw);
    if ((sm100::smem_u32(raw) & 1023) != 0) {              // the swizzle's atoms (a block's shared memory has always begun on one)
        if (threadIdx.x == 0) atomicExch(params.step.status, RB_ERR_BAD_ALIGN);
        return;
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) {
            sm100::mbar_init(&s.full[i], 1);             // the producer
            sm100::mbar_init(&s.empty[i], 1);            // the warp that took it
        }
        s.abort = 0;
        sm100::fence_barrier_init();
    }
    for (int i = threadIdx.x; i < (int)sizeof(Step) / 4; i += THREADS)
        reinterpret_cast<uint32_t*>(&s.step)[i] = reinterpret_cast<const uint32_t*>(&params.step)[i];
    if ((int)threadIdx.x < params.step.T) {
        const Step& p = params.step;
        const int t = threadIdx.x, slot = p.seq_slot[t], old = p.kv_len[t] - 1;
        s.slot[t] = slot;
        s.old[t] = old;
        s.page[t] = slot >= 0 && old >= 0 ? p.block_table[(size_t)slot * p.max_pages + old / RB_PAGE] : -1;
    }
    for (int i = threadIdx.x; i < (int)sizeof(s.q) / 16; i += THREADS) reinterpret_cast<uint4*>(s.q)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    const Waits waits{&s.abort, s.step.status, s.step.wait_limit};
    // Registers move to the warps that compute: 12 warps of 168 at launch, 4 of 40 and 8 of 232 from here on.
    if (threadIdx.x >= CTHREADS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (threadIdx.x == CTHREADS) {
            Producer producer(s, waits);
            producer.run(s.step, params);
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
        Compute compute(s, waits);
        compute.run();
    }
}

struct Ready { int sms = 0; };
PerDevice<Ready> g_ready;

int encode(const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box, CUtensorMap* out) {
    const sm100::EncodeTiledFn fn = sm100::encode_fn();
    if (fn == nullptr) return RB_ERR_NO_DRIVER_FN;
    const cuuint32_t one[4] = {1, 1, 1, 1};
    const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? RB_OK : RB_ERR_BAD_ALIGN;
}
// A weight [rows][K] as (64 values of k, row, eight rows further down, block of 64 values): a box is a stage, 16 rows of 256 values.
// `step`: rows between the two eights.
int weight_map(const void* w, int rows, int K, int step, CUtensorMap* out) {
    const cuuint64_t row = (cuuint64_t)K * 2, dims[4] = {KB, (cuuint64_t)rows, 2, (cuuint64_t)(K / KB)}, strides[3] = {row, row * step, KB * 2};
    const cuuint32_t box[4] = {KB, 8, 2, KC / KB};
    return encode(w, 4, dims, strides, box, out);
}
// Rows of 128 values of keys or values as (64 values, row, half): a box is 16 rows.
int rows_map(const void* rows, unsigned long long n, CUtensorMap* out) {
    const cuuint64_t dims[3] = {KB, n, HD / KB}, strides[2] = {HD * 2, KB * 2};
    const cuuint32_t box[3] = {KB, SK, HD / KB};
    return encode(rows, 3, dims, strides, box, out);
}
}  // namespace

// What the caller gives: a layer's pointers and a step's (see Step; `wait_limit` 0 stands for the default).
struct rb_DecodeLayer {
    const void *qkv, *o, *gate_up, *down, *ff_norm, *next_norm, *q_norm, *k_norm;
    void *k, *v;
    float ff_eps, in_eps;
};
struct rb_DecodeStep {
    int T, H, I, nq, nkv, layers, splits, max_pages, norm_f32, head_norm_f32, n_pages;
    float head_eps, scale;
    const float* cos_sin;
    const int *seq_slot, *kv_len, *block_table;
    const void* first_norm;
    float* resid;
    void* xhat;
    float *sumsq, *qkv;
    void *attn, *h;
    float *part_o, *part_ml;
    unsigned* counters;
    int* status;
    long long wait_limit;
    const rb_DecodeLayer* layer;
};

// The step's layers, as many launches as their number asks for (38 a launch).  RB_ERR_BAD_SIZE or RB_ERR_BAD_ALIGN: the kernel does
// not take these sizes or pointers and nothing was launched.
extern "C" int rb_decode_layers(const void* step, void* stream) {
    const rb_DecodeStep& q = *static_cast<const rb_DecodeStep*>(step);
    if (q.T < 1 || q.T > TT || q.layers < 1 || q.splits < 1 || q.n_pages < 1 || q.H % 64 || q.I % 64 || q.H <= 0 || q.I <= 0 || q.nkv < 1 ||
        q.nq % q.nkv || q.nq / q.nkv > MAX_G)
        return RB_ERR_BAD_SIZE;
    // (indices are 32-bit)
    if ((long long)q.T * q.nkv * q.splits >= 1 << 20 || 16ll * q.splits * (q.nq + 2ll * q.nkv) * HD >= 1ll << 31 || 32ll * q.I >= 1ll << 31 ||
        16ll * q.H >= 1ll << 31 || (long long)q.n_pages * q.nkv * RB_PAGE >= 1ll << 31)
        return RB_ERR_BAD_SIZE;
    auto off16 = [](const void* a) { return ((uintptr_t)a & 15) != 0; };
    if (off16(q.resid) || off16(q.xhat) || off16(q.qkv) || off16(q.attn) || off16(q.h) || off16(q.part_ml) || off16(q.cos_sin)) return RB_ERR_BAD_ALIGN;
    for (int i = 0; i < q.layers; ++i) {
        const rb_DecodeLayer& L = q.layer[i];
        if (off16(L.qkv) || off16(L.o) || off16(L.gate_up) || off16(L.down) || off16(L.k) || off16(L.v) || off16(L.q_norm) || off16(L.k_norm))
            return RB_ERR_BAD_ALIGN;
    }
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return (int)e;
    const Ready* ready = nullptr;
    int rc = g_ready.get(device, &ready, [&](Ready& r) {
        cudaError_t a = cudaFuncSetAttribute(decode_layers_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (a == cudaSuccess) a = cudaDeviceGetAttribute(&r.sms, cudaDevAttrMultiProcessorCount, device);
        return (int)a;
    });
    if (rc != RB_OK) return rc;
    Params params = {};
    Step& p = params.step;
    p.T = q.T; p.H = q.H; p.I = q.I; p.nq = q.nq; p.nkv = q.nkv; p.splits = q.splits; p.max_pages = q.max_pages;
    p.norm_f32 = q.norm_f32; p.head_norm_f32 = q.head_norm_f32; p.head_eps = q.head_eps; p.scale = q.scale;
    p.inv_T = 1.f / (float)q.T; p.inv_nkv = 1.f / (float)q.nkv; p.inv_H = 1.f / (float)q.H;
    p.cos_sin = reinterpret_cast<const float2*>(q.cos_sin);
    p.seq_slot = q.seq_slot; p.kv_len = q.kv_len; p.block_table = q.block_table;
    p.resid = q.resid; p.xhat = static_cast<__nv_bfloat16*>(q.xhat); p.sumsq = q.sumsq; p.qkv = q.qkv;
    p.attn = static_cast<__nv_bfloat16*>(q.attn); p.h = static_cast<__nv_bfloat16*>(q.h);
    p.part_o = q.part_o; p.part_ml = q.part_ml; p.counters = q.counters; p.status = q.status;
    p.wait_limit = (unsigned)(q.wait_limit > 0 && q.wait_limit < sm100::RB_WAIT_CYCLES ? q.wait_limit : sm100::RB_WAIT_CYCLES);
    const int work[PHASES] = {(q.nq + 2 * q.nkv) * HD / UR, 0, q.H / UR, 2 * q.I / UR, q.H / UR};
    const int inputs[PHASES] = {q.H, KC, q.nq * HD, q.H, q.I};
    for (int i = 0; i < PHASES; ++i) {
        Plan& a = p.plan[i];
        a.each = work[i] / ready->sms; a.rest = work[i] % ready->sms;
        a.K = inputs[i]; a.stages = (a.K + KC - 1) / KC;
        a.passes = (a.stages + CW * CPW - 1) / (CW * CPW);
        a.per = (a.stages + a.passes - 1) / a.passes;
        a.warps = (a.per + CPW - 1) / CPW;
        a.units = a.warps > 4 ? 1 : (a.warps > 2 ? 2 : 4);
    }
    const unsigned long long cached = (unsigned long long)q.n_pages * q.nkv * RB_PAGE;
    for (int i0 = 0; i0 < q.layers; i0 += MAX_LAYERS) {
        p.layers = q.layers - i0 < MAX_LAYERS ? q.layers - i0 : MAX_LAYERS;
        p.first_norm = i0 > 0 ? nullptr : q.first_norm;
        for (int i = 0; i < p.layers; ++i) {
            const rb_DecodeLayer& L = q.layer[i0 + i];
            LayerPtrs& to = p.layer[i];
            CUtensorMap* map = params.map[i];
            if ((rc = weight_map(L.qkv, (q.nq + 2 * q.nkv) * HD, q.H, 8, map + QKV)) != RB_OK || (rc = weight_map(L.o, q.H, q.nq * HD, 8, map + OUT)) != RB_OK ||
                (rc = weight_map(L.gate_up, 2 * q.I, q.H, 16, map + GATED)) != RB_OK || (rc = weight_map(L.down, q.H, q.I, 8, map + DOWN)) != RB_OK ||
                (rc = rows_map(L.k, cached, map + ATTENTION)) != RB_OK || (rc = rows_map(L.v, cached, map + PHASES)) != RB_OK)
                return rc;
            to.ff_norm = L.ff_norm; to.next_norm = L.next_norm; to.q_norm = L.q_norm; to.k_norm = L.k_norm;
            to.k = static_cast<__nv_bfloat16*>(L.k); to.v = static_cast<__nv_bfloat16*>(L.v);
            to.ff_eps = L.ff_eps; to.in_eps = L.in_eps;
        }
        e = cudaMemsetAsync(p.counters, 0, (1 + (size_t)p.T * p.nkv) * sizeof(unsigned), (cudaStream_t)stream);
        if (e != cudaSuccess) return (int)e;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(ready->sms);
        cfg.blockDim = dim3(THREADS);
        cfg.dynamicSmemBytes = SMEM;
        cfg.stream = (cudaStream_t)stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, decode_layers_kernel, params);
        if (e != cudaSuccess) return (int)e;
    }
    return RB_OK;
}
