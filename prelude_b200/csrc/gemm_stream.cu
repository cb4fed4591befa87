// y[M, N] = x[M, K] * W[N, K]^T (+ bias) for the few rows of a decode step
// (M <= 16), bfloat16 in, float32 accumulation, bfloat16 or float32 out.
//
// With so few rows the product is a stream over the weight matrix: every byte
// of W is read once and the time is W's bytes over the memory bandwidth, plus
// whatever the kernel adds before the first byte and after the last.  The
// kernel is built to add little:
//  * Every block owns a contiguous run of output features (N / blocks of them,
//    give or take one) and the whole of K for them: no block waits for another,
//    and nothing is summed across blocks afterwards.
//  * Four loader warps stream the block's rows of W through a ring of
//    shared-memory stages (8 rows x one chunk of K per stage, one bulk copy per
//    row, full and empty barriers); the compute warps take the stages two at a
//    time.  Issuing a bulk copy costs a warp about 60 cycles whatever its size,
//    and as much goes into a stage's wait and its announcement; warps issue side
//    by side, so they share a stage only as far as its copies are waited for
//    (GsPlan) and take the stages in turn, and the chunks are as long as leaves
//    four stages.
//    How K is cut into chunks changes no sum: a step is dealt to its warp and
//    chain by its place in K, or in a part of K that the rows' number sets.
//    Weights are written by no kernel, so the
//    loaders fill the ring before they wait for the kernel before this one on
//    the stream: the stream is already flowing when x becomes available.
//  * x (a few KB per row) is copied whole into shared memory by the compute warps
//    the moment that kernel is done.
//  * Eight compute warps share the 16-element steps of every pair of stages; W is
//    the row operand of mma.m16n8k16 (16 features: ldmatrix takes its 16 row
//    addresses from the two stages), x the column operand (8 batch rows per
//    instruction), both fetched from rows padded by 16 bytes; every warp keeps
//    four independent chains of sums.  When a 16-feature tile has seen all of K
//    the warps' sums are added through shared memory and stored.
//  * Where K is long and the output narrow (the down projection), x would crowd
//    the ring out of shared memory and every block would fetch all of it.  K can
//    then be cut into a few parts: the grid gets a second dimension, every part
//    works on its columns of W and x only and writes float32 partial sums of
//    its own, and whoever reads the output adds the parts (the residual add
//    does).  Nothing waits for anything.
//  * The gated form serves a feed-forward's merged gate and up projection: W
//    holds the N gate rows, then the N up rows; a tile is 8 features, its first
//    stage their gate rows and its second their up rows, so the two halves of
//    the tensor-core tile are gate and up of the same features and the
//    epilogue writes silu(gate) * up (float32 sums, one rounding) - the
//    activation costs no kernel and the 2N-wide intermediate never exists.
//  * Waits on barriers are bounded in time; a warp that gives up raises the
//    status word and the block goes on to its end.
// The reference leaves these shapes to its GEMM libraries
// (crates/prelude-cuda/src/ops/gemm.rs:35-137; DeepGEMM's small-M path).
// Needs K % 16 == 0, 16-byte aligned rows of W and x, and x to fit in shared
// memory beside the ring (pb_gemm_stream_supported says whether a shape is taken).
#include "attention_common.cuh"

PB_TIMELINE_UNIT(gemm_stream)

#define GS_WARPS 8                              // compute warps
#define GS_LOADERS 4                            // loader warps
#define GS_THREADS ((GS_WARPS + GS_LOADERS) * 32)
#define GS_ROWS 8                               // features per stage; a tile of the product is two stages
#define GS_MAX_STAGES 16
#define GS_CHAINS 4                             // independent accumulators per warp
#define GS_SMEM_LIMIT (227 * 1024 - 2048)

struct GsParams {
    const __nv_bfloat16* W;
    const __nv_bfloat16* X;
    void* out;
    const float* bias;
    long long ldw, ldx, ldo;
    int M, N, K;
    int ks;                 // elements of K per stage
    int part;               // elements of K whose steps are dealt to the warps' chains from the first on; stages do not go across parts
    int stages;
    int share;              // loader warps that bring a stage together
    int sets;               // of the warps' sums in shared memory: two, or one where a second does not fit
    int out_f32;
    long long split_stride; // elements between the partial outputs of the splits of K (gridDim.y of them)
    int gated;              // W holds N gate rows, then N up rows; the output is silu(gate) * up, N wide
    int act;                // PbAct: what the epilogue does with the sums (gated or plain forms)
    float limit, alpha;
    // plain form with the residual add and the squashing behind it in the epilogue (res not null): res[m, n] += sum,
    // out[m, n] = tanh(slope * res[m, n]) * gain[n] + shift[n]; res float32 [M, N] dense
    float* res;
    const float* gain;
    const float* shift;
    float slope;
    int* status;
};

__device__ __forceinline__ void gs_mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void gs_bar_compute() { asm volatile("bar.sync 1, %0;\n" ::"n"(GS_WARPS * 32) : "memory"); }
__device__ __forceinline__ void ldmatrix_x4_a(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

__device__ __forceinline__ void ldmatrix_x2(unsigned& r0, unsigned& r1, unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(r0), "=r"(r1) : "r"(addr));
}

// MT: 8-row tiles of x (M <= 8 * MT).  RES: the plain form with the residual add and the squashing in its epilogue.
template <int MT, bool RES>
__global__ void __launch_bounds__(GS_THREADS, 1) gemm_stream_kernel(GsParams p) {
    pb_grid_dep_launch();
    PB_TL(PB_TL_GEMM_STREAM, PB_TL_ENTRY);
    if (gridDim.y > 1) {
        // K is cut into gridDim.y equal parts (p.K is the length of one); part s multiplies its columns of W with
        // its columns of x and writes a partial output of its own, which the reader adds up
        const int s = blockIdx.y;
        p.W += (size_t)s * p.K;
        p.X += (size_t)s * p.K;
        p.out = reinterpret_cast<float*>(p.out) + (size_t)s * p.split_stride;
        if (s > 0) p.bias = nullptr;
    }
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t full_bar[GS_MAX_STAGES], empty_bar[GS_MAX_STAGES], x_bar;
    __shared__ int s_dead;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int x_stride = p.K * 2 + 16;                         // bytes between rows of x in shared memory
    const int w_stride = p.ks * 2 + 16;                        // bytes between rows of a stage
    const int stage_bytes = GS_ROWS * w_stride;
    unsigned char* sX = smem;                                  // [M] rows
    unsigned char* ring = sX + (size_t)p.M * x_stride;
    // sets of [GS_WARPS][8 MT batch rows][16 features], which tiles take in turn: of two, one is written again behind the next tile's barrier only
    float* sums = reinterpret_cast<float*>(ring + (size_t)p.stages * stage_bytes);

    // This block's features, in tiles of 16 = two stages of 8 (the last tile may have one).  Loader and compute
    // warps walk the stages in the same order: tile, chunk of K, half.
    const int r0 = (int)((long long)blockIdx.x * p.N / gridDim.x), r1 = (int)((long long)(blockIdx.x + 1) * p.N / gridDim.x);
    const int span = p.gated ? GS_ROWS : 16;                   // features per tile
    const int n_tiles = (r1 - r0 + span - 1) / span;

    // a thread a stage: all 33 barriers by one thread make a product of 2.5 us 0.15 longer
    if (threadIdx.x < 32) {
        if (lane == 0) {
            s_dead = 0;
            mbar_init(&x_bar, GS_LOADERS);
        }
        if (lane < p.stages) { mbar_init(&full_bar[lane], p.share); mbar_init(&empty_bar[lane], GS_WARPS); }
        mbar_fence_init();
    }
    __syncthreads();

    if (warp >= GS_WARPS) {
        // ---------------- loaders: `share` warps at a time take the stages in turn, a lane copies a row ----------------
        // No more turns than stages: a warp that waits for a stage's tenant of one lap ago then knows that the one of two laps ago has left (it
        // has waited for that or a later one), and a parity tells only two laps apart
        const int lw = (warp - GS_WARPS) / p.share, n_loaders = min(GS_LOADERS / p.share, p.stages);
        const int per = GS_ROWS / p.share, row = (warp - GS_WARPS) % p.share * per + lane;   // this lane's, of the first `per` lanes
        bool ok = true;
        int stage = 0, phase = 0, i = 0, turn = 0;
#pragma unroll 1
        for (int tile = 0; tile < n_tiles && ok; ++tile) {
            const int halves = (p.gated || r1 - (r0 + tile * span) > GS_ROWS) ? 2 : 1;
#pragma unroll 1
            for (int k0 = 0, end = 0, len; k0 < p.K && ok; k0 += len) {
                if (k0 == end) end = min(end + p.part, p.K);
                len = min(p.ks, end - k0);
                for (int h = 0; h < halves; ++h, ++i) {
                    if (turn == lw) {
                        if (i >= p.stages) {                   // the first ring-full finds every stage free
                            ok = mbar_wait_bounded(&empty_bar[stage], phase ^ 1);
                            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                        }
                        const int feat0 = r0 + tile * span + (p.gated ? 0 : h * GS_ROWS);   // first feature of the stage
                        const int row0 = feat0 + (p.gated ? h * p.N : 0);             // its row of W: up rows follow the gate rows
                        const int n_rows = min(GS_ROWS, r1 - feat0);
                        // the copies may land before the expected bytes are posted: the phase cannot end before this arrival
                        if (lane == 0) mbar_arrive_expect_tx(&full_bar[stage], (unsigned)min(per, max(0, n_rows - row)) * len * 2);
                        if (lane < per && row < n_rows)
                            bulk_copy_g2s(ring + (size_t)stage * stage_bytes + (size_t)row * w_stride, p.W + (size_t)(row0 + row) * p.ldw + k0,
                                          (unsigned)len * 2, &full_bar[stage]);
                    }
                    if (++turn == n_loaders) turn = 0;
                    if (++stage == p.stages) { stage = 0; phase ^= 1; }
                }
            }
        }
        if (!ok && lane == 0 && p.status) atomicExch(p.status, 11);
        return;
    }

    // ---------------- compute warps ----------------
    pb_grid_dep_wait();                                        // the output may still be in use by the kernel before
    PB_TL(PB_TL_GEMM_STREAM, PB_TL_AFTER_WAIT);
    const int g = lane >> 2, t4 = lane & 3;
    if (warp < GS_LOADERS) {
        // x is this kernel's only input that another kernel writes: the first four compute warps fetch it the
        // moment that kernel is done (warp j brings rows j, j + 4, ...), whatever the loaders are busy with
        const int mine = (p.M - warp + GS_LOADERS - 1) / GS_LOADERS;
        if (lane == 0) mbar_arrive_expect_tx(&x_bar, (unsigned)max(mine, 0) * p.K * 2);
        const int m = warp + lane * GS_LOADERS;
        if (m < p.M) bulk_copy_g2s(sX + (size_t)m * x_stride, p.X + (size_t)m * p.ldx, (unsigned)p.K * 2, &x_bar);
    }
    // A warp that gives up waiting says so in s_dead; the compute warps meet at their barrier all the same
    // and leave together, so none is left waiting for one that has gone.
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&x_bar, 0))) {
        if (lane == 0) { *(volatile int*)&s_dead = 1; if (p.status) atomicExch(p.status, 12); }
    }
    gs_bar_compute();
    if (*(volatile int*)&s_dead) return;
    PB_TL(PB_TL_GEMM_STREAM, PB_TL_INPUT);
    const unsigned sX_a = smem_u32(sX), ring_a = smem_u32(ring);
    // ldmatrix lanes.  W (row operand, 16 features x 16 k): lane -> feature lane & 15 (the first eight in one
    // stage, the others in the next), k half lane >> 4.  x (column operand): 8 batch rows x 16 k (x2), or
    // 16 batch rows (x4); rows that do not exist read the last row that does, and their sums are never stored.
    const unsigned a_off = (lane & 7) * w_stride + (lane >> 4) * 16;
    const bool upper = (lane & 8) != 0;                        // this lane addresses a row of the second stage
    const int x_row = (MT == 1) ? (lane & 7) : ((lane & 7) + (lane >> 4) * 8);
    const unsigned b_off = min(x_row, p.M - 1) * x_stride + ((lane >> 3) & 1) * 16;
    int stage = 0, phase = 0;
#pragma unroll 1
    for (int tile = 0; tile < n_tiles; ++tile) {
        const int halves = (p.gated || r1 - (r0 + tile * span) > GS_ROWS) ? 2 : 1;
        // GS_CHAINS independent chains of sums, so that a product does not wait for the one before it
        float acc[GS_CHAINS][MT][4];
        // the residual form's addend of this thread's output (at most one a tile: M * 16 <= 256), fetched ahead
        float r_pre = 0.f, gain_pre = 0.f, shift_pre = 0.f;
        if (RES) {
            const int m = threadIdx.x >> 4, n = r0 + tile * 16 + (threadIdx.x & 15);
            if (m < p.M && n < r1) { r_pre = p.res[(size_t)m * p.N + n]; gain_pre = p.gain[n]; shift_pre = p.shift[n]; }
        }
#pragma unroll
        for (int c = 0; c < GS_CHAINS; ++c)
#pragma unroll
            for (int j = 0; j < MT; ++j) acc[c][j][0] = acc[c][j][1] = acc[c][j][2] = acc[c][j][3] = 0.f;
#pragma unroll 1
        for (int k0 = 0, end = 0, first = 0, len; k0 < p.K; k0 += len) {
            if (k0 == end) { first = end; end = min(end + p.part, p.K); }
            len = min(p.ks, end - k0);
            const int stage2 = (stage + 1 == p.stages) ? 0 : stage + 1, phase2 = (stage + 1 == p.stages) ? phase ^ 1 : phase;
            bool landed = mbar_wait_bounded(&full_bar[stage], phase);
            if (halves == 2) landed = landed && mbar_wait_bounded(&full_bar[stage2], phase2);
            if (!__all_sync(0xffffffffu, landed)) {
                if (lane == 0) { *(volatile int*)&s_dead = 1; if (p.status) atomicExch(p.status, 12); }
                break;
            }
            // the stage's steps go on where the part's last stage stopped: step i of a part is warp i % 8's, chain i / 8 % 4, however it is cut
            const int steps = len >> 4, at = ((k0 - first) >> 4) & (GS_WARPS * GS_CHAINS - 1);
            // with one stage only, the upper eight rows read the lower ones again (their sums are not stored)
            const unsigned a_base = ring_a + ((upper && halves == 2) ? stage2 : stage) * stage_bytes + a_off;
            const unsigned b_base = sX_a + b_off + k0 * 2;
#pragma unroll 1
            for (int s0 = warp - at; s0 < steps; s0 += GS_WARPS * GS_CHAINS) {
                unsigned a[GS_CHAINS][4], b[GS_CHAINS][4];
#pragma unroll
                for (int c = 0; c < GS_CHAINS; ++c) {
                    const int s = s0 + c * GS_WARPS;
                    if ((unsigned)s < (unsigned)steps) {
                        ldmatrix_x4_a(a[c], a_base + s * 32);
                        if (MT == 1) ldmatrix_x2(b[c][0], b[c][1], b_base + s * 32);
                        else ldmatrix_x4_a(b[c], b_base + s * 32);
                    }
                }
#pragma unroll
                for (int c = 0; c < GS_CHAINS; ++c) {
                    if ((unsigned)(s0 + c * GS_WARPS) < (unsigned)steps) {
                        mma_bf16_free(acc[c][0], a[c], b[c][0], b[c][1]);
                        if (MT == 2) mma_bf16_free(acc[c][MT - 1], a[c], b[c][2], b[c][3]);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) {                                   // this warp is done with the stages
                gs_mbar_arrive(&empty_bar[stage]);
                if (halves == 2) gs_mbar_arrive(&empty_bar[stage2]);
            }
            for (int h = 0; h < halves; ++h)
                if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
        // add the eight warps' sums: acc[.][j][e] is feature g (+8 for e >= 2), batch row 8 j + 2 t4 + (e & 1)
        float* red = sums + (p.sets == 2 ? tile & 1 : 0) * (GS_WARPS * 16 * 8 * MT);
        float* mine = red + (size_t)warp * 16 * 8 * MT;
#pragma unroll
        for (int j = 0; j < MT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float v = acc[0][j][e];
#pragma unroll
                for (int c = 1; c < GS_CHAINS; ++c) v += acc[c][j][e];
                mine[(8 * j + 2 * t4 + (e & 1)) * 16 + g + 8 * (e >> 1)] = v;
            }
        gs_bar_compute();
        if (*(volatile int*)&s_dead) return;
        if (p.gated) {
            // rows 0..7 of the tile are the gate sums of 8 features, rows 8..15 the up sums of the same features
            for (int idx = threadIdx.x; idx < p.M * GS_ROWS; idx += GS_WARPS * 32) {
                const int m = idx >> 3, rr = idx & 7;
                const int n = r0 + tile * GS_ROWS + rr;
                if (n < r1) {
                    float gsum = 0.f, usum = 0.f;
#pragma unroll
                    for (int w = 0; w < GS_WARPS; ++w) {
                        gsum += red[(size_t)w * 16 * 8 * MT + m * 16 + rr];
                        usum += red[(size_t)w * 16 * 8 * MT + m * 16 + rr + 8];
                    }
                    float v;
                    if (p.act == PB_ACT_CLAMPED) {
                        const float a = fminf(gsum, p.limit), b = fminf(fmaxf(usum, -p.limit), p.limit);
                        v = a / (1.0f + expf(-p.alpha * a)) * (b + 1.0f);
                    } else if (p.act == PB_ACT_GELU_TANH) {
                        v = pb_gelu_tanh(gsum) * usum;
                    } else if (p.act == PB_ACT_RELU) {
                        v = fmaxf(gsum, 0.f) * usum;
                    } else {
                        v = gsum / (1.0f + expf(-gsum)) * usum;
                    }
                    if (p.out_f32) reinterpret_cast<float*>(p.out)[(size_t)m * p.ldo + n] = v;
                    else reinterpret_cast<__nv_bfloat16*>(p.out)[(size_t)m * p.ldo + n] = __float2bfloat16_rn(v);
                }
            }
        } else {
            for (int idx = threadIdx.x; idx < p.M * 16; idx += GS_WARPS * 32) {
                const int m = idx >> 4, rr = idx & 15;
                const int n = r0 + tile * 16 + rr;
                if (n < r1) {
                    float v = 0.f;
#pragma unroll
                    for (int w = 0; w < GS_WARPS; ++w) v += red[(size_t)w * 16 * 8 * MT + idx];
                    if (p.bias) v += p.bias[n];
                    if (p.act == PB_ACT_RELU2) v = pb_relu2(v);
                    if (RES) {
                        v += r_pre;
                        p.res[(size_t)m * p.N + n] = v;
                        v = pb_squash(v, p.slope, gain_pre, shift_pre);
                    }
                    if (p.out_f32) reinterpret_cast<float*>(p.out)[(size_t)m * p.ldo + n] = v;
                    else reinterpret_cast<__nv_bfloat16*>(p.out)[(size_t)m * p.ldo + n] = __float2bfloat16_rn(v);
                }
            }
        }
        if (p.sets == 1) gs_bar_compute();                     // the sums are read before the next tile overwrites them
    }
    PB_TL(PB_TL_GEMM_STREAM, PB_TL_DONE);
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
static int g_gs_sms = 0;
static int gs_sms() {
    if (g_gs_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_gs_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_gs_sms <= 0) g_gs_sms = 148;
    }
    return g_gs_sms;
}

// How a product's rows of W pass through shared memory.
// Parts: they decide the order of the sums and nothing else does: the fewest equal ones, in steps of 16, of which three fit beside the rows of x and one
// set of sums, or two.
// Pieces of a part: all of it where the block's rows then lie in the ring at once, as copies are few and nothing waits; else the longest equal cut of which
// four stages fit (a tile takes its stages two by two: with three, one is on its way while it waits); else, and for blocks of eight rows, which
// take single stages and wait for each, the longest of which two do.
// Stages: all that fit; where all rows do, no more than eight, so that short rows leave the next kernel's blocks room (512 x 2,112, 1 row: with sixteen
// 2.55, with eight 2.1), but no fewer: a block that leaves room where the kernel before it ran one to a multiprocessor meets a second of its own
// there while others have none (2,048 x 2,048, 8 rows, behind a linear-attention step: with the two stages that its rows fill 0.9 us more).
// Two sets of the warps' sums unless the second costs a pair of stages.
// Warps a stage: two; all four where there are three stages, which the tiles wait for whatever is done, and for blocks of eight rows; one where
// pieces are short, as what a warp spends on a stage besides its copies then counts.
// us, piece x stages, 64 MB of weights: K = 2,560, 12 rows 2,560 x 3 16.1, 1,280 x 7 14.6; 4,096, 2 rows 4,096 x 3 13.8, 2,048 x 6 13.2; 16 MB: 2,560, 12
// rows 2,560 x 3 6.2, 1,280 x 7 6.7; 4,096, 2 rows 4.8 and 5.1.  One, two and four warps a stage: 67 MB, 4,096, 16 rows, 1,376 x 4 13.5, 13.2, 13.5 (134 MB
// 27.3, 26.6, 27.8); 67 to 80 MB, 6,912, 10 rows, 864 x 6 14.4, 14.1, 15.6; 9,728, 8 rows, 608 x 6 21.0, 21.7, 27.0; 8,192, 11 rows, 832 x 3 30.4, 29.7, 28.5;
// 8,192, 12 rows, 768 x 2 34.6, 32.8, 36.8 (512 x 3 40.4, 39.0, 37.7).
struct GsPlan {
    int part, ks, stages, sets, share;      // as in GsParams
    size_t smem;
};

// `rows`: of W, of one block (0: any number).  False: not even two stages fit.
static bool gs_plan(int M, int K, int rows, GsPlan* p) {
    const size_t x_bytes = (size_t)M * ((size_t)K * 2 + 16), set_bytes = (size_t)GS_WARPS * 16 * (M <= 8 ? 8 : 16) * 4, least = 8192;
    auto taken = [&](int sets) { return x_bytes + (sets * set_bytes < least ? least : sets * set_bytes); };
    auto stage_of = [](int k) { return (size_t)GS_ROWS * ((size_t)k * 2 + 16); };
    auto fit = [&](int k, int sets) { return taken(sets) < GS_SMEM_LIMIT ? (int)((GS_SMEM_LIMIT - taken(sets)) / stage_of(k)) : 0; };
    p->part = 0;
    for (int want = 3; want >= 2 && p->part == 0; --want)
        for (int n = 1; n <= K / 16; ++n) {
            const int k_per = ((K + n - 1) / n + 15) / 16 * 16;
            if (k_per < 512 && n > 1) break;
            if (fit(k_per, 1) >= want) { p->part = k_per; break; }
        }
    if (p->part == 0) return false;
    if (p->part % (16 * GS_WARPS * GS_CHAINS) == 0) p->part = K;          // whole turns over the chains: dealt as K in one part is
    const int unit = p->part == K ? 16 * GS_WARPS : 16, all = (rows + GS_ROWS - 1) / GS_ROWS * ((K + p->part - 1) / p->part);
    const int whole = fit(p->part, 1);
    const bool few = rows > 0 && rows <= GS_ROWS;
    for (int rule = all > 0 && all <= GS_MAX_STAGES && whole >= all && whole >= 2 ? 0 : few ? 2 : 1; rule < 3; ++rule)
        for (int n = 1; n <= p->part / 16; ++n) {
            const int want = rule == 0 && all > 2 ? all : rule == 1 ? 4 : 2, ks = n == 1 ? p->part : ((p->part + n - 1) / n + unit - 1) / unit * unit;
            if (ks < 512 && n > 1) break;                                   // copies this short are not worth having
            const int one = fit(ks, 1), two = fit(ks, 2);
            if (one < want) continue;
            p->sets = rule == 0 ? (two >= want ? 2 : 1) : two == one || two >= 6 || (two >= 4 && two / 2 == one / 2) ? 2 : 1;
            const int fits = p->sets == 2 ? two : one, stages = rule == 0 && fits > 8 ? (want > 8 ? want : 8) : fits;
            p->ks = ks;
            p->stages = stages > GS_MAX_STAGES ? GS_MAX_STAGES : stages;
            p->share = few || p->stages == 3 ? 4 : ks <= 704 && p->stages > 3 ? 1 : 2;
            p->smem = taken(p->sets) + p->stages * stage_of(ks);
            return true;
        }
    return false;
}

// Whether the kernel takes the shape (else the caller uses another product).
PB_API int pb_gemm_stream_supported(int M, int N, int K, long long ldw, long long ldx) {
    if (M < 1 || M > 16 || N < 1 || K < 16 || K % 16 || ldw % 8 || ldx % 8) return 0;
    GsPlan plan;
    return gs_plan(M, K, 0, &plan) ? 1 : 0;
}

// gated: W is [2 N, K], N gate rows then N up rows, and out [M, N] = silu(x Wg^T) * (x Wu^T); no bias, no splits.
// splits > 1 cuts K into that many equal parts (K %% (16 * splits) == 0): out is then float32
// [splits][M][ldo-strided N] with split_stride elements between the parts, and the caller adds them.
struct GsResidual {
    float* res;
    const float* gain;
    const float* shift;
    float slope;
};
static int gs_run(const void* X, const void* W, const float* bias, void* out, int M, int N, int K, long long ldx, long long ldw,
                  long long ldo, int out_f32, int splits, long long split_stride, int gated, int act, float limit, float alpha,
                  int* status, cudaStream_t stream, GsResidual residual = GsResidual{}) {
    PB_REQUIRE(!gated || (splits == 1 && bias == nullptr), "gemm_stream: the gated form takes no bias and no cut of K");
    PB_REQUIRE(splits >= 1 && splits <= 16 && (splits == 1 || K % (16 * splits) == 0), "gemm_stream: K=%d cannot be cut into %d parts of whole 16-element steps", K, splits);
    PB_REQUIRE(splits == 1 || (out_f32 && split_stride >= (long long)(M - 1) * ldo + N), "gemm_stream: partial sums are float32, %d apart at least", M * N);
    const int k_part = K / splits;
    PB_REQUIRE(pb_gemm_stream_supported(M, N, k_part, ldw, ldx),
               "gemm_stream: M=%d N=%d K=%d not taken (M <= 16, K %% 16 == 0, 16-byte aligned rows, x must fit in shared memory)", M, N, k_part);
    PB_REQUIRE(X && W && out && pb_aligned(X, 16) && pb_aligned(W, 16), "gemm_stream: null or unaligned pointer");
    GsParams p{};
    p.W = (const __nv_bfloat16*)W; p.X = (const __nv_bfloat16*)X; p.out = out; p.bias = bias;
    p.ldw = ldw; p.ldx = ldx; p.ldo = ldo; p.M = M; p.N = N; p.K = k_part; p.out_f32 = out_f32; p.status = status;
    p.split_stride = split_stride;
    p.gated = gated ? 1 : 0;
    p.act = act; p.limit = limit; p.alpha = alpha;
    p.res = residual.res; p.gain = residual.gain; p.shift = residual.shift; p.slope = residual.slope;
    int blocks = gs_sms() / splits;
    if (blocks < 1) blocks = 1;
    if (blocks > (N + 7) / 8) blocks = (N + 7) / 8;           // at least 8 features per block
    const int features = (N + blocks - 1) / blocks;
    GsPlan plan;
    gs_plan(M, k_part, gated ? (features + GS_ROWS - 1) / GS_ROWS * 2 * GS_ROWS : features, &plan);
    p.part = plan.part; p.ks = plan.ks; p.stages = plan.stages; p.sets = plan.sets; p.share = plan.share;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_stream_kernel<1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, GS_SMEM_LIMIT);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_stream_kernel<2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, GS_SMEM_LIMIT);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_stream_kernel<1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, GS_SMEM_LIMIT);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_stream_kernel<2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, GS_SMEM_LIMIT);
        if (e != cudaSuccess) return pb_fail("gemm_stream: cannot get %d bytes of shared memory: %s", GS_SMEM_LIMIT, cudaGetErrorString(e));
        configured = true;
    }
    if (p.res) {
        if (M <= 8) pb_launch(gemm_stream_kernel<1, true>, dim3(blocks, splits), dim3(GS_THREADS), plan.smem, stream, p);
        else pb_launch(gemm_stream_kernel<2, true>, dim3(blocks, splits), dim3(GS_THREADS), plan.smem, stream, p);
    } else {
        if (M <= 8) pb_launch(gemm_stream_kernel<1, false>, dim3(blocks, splits), dim3(GS_THREADS), plan.smem, stream, p);
        else pb_launch(gemm_stream_kernel<2, false>, dim3(blocks, splits), dim3(GS_THREADS), plan.smem, stream, p);
    }
    PB_CHECK_LAUNCH("gemm_stream");
    return 0;
}

PB_API int pb_gemm_stream_bf16(const void* X, const void* W, const float* bias, void* out, int M, int N, int K,
                               long long ldx, long long ldw, long long ldo, int out_f32, int splits, long long split_stride,
                               int gated, int* status, cudaStream_t stream) {
    return gs_run(X, W, bias, out, M, N, K, ldx, ldw, ldo, out_f32, splits, split_stride, gated, 0, 0.f, 0.f, status, stream);
}

// The gated form with the tanh form of GELU in its epilogue: out [M, N] = gelu(x Wg^T) * (x Wu^T); W is [2 N, K], N gate
// rows then N up rows.
PB_API int pb_gemm_stream_gelu_glu_bf16(const void* X, const void* W, void* out, int M, int N, int K, long long ldx, long long ldw,
                                        long long ldo, int out_f32, int* status, cudaStream_t stream) {
    return gs_run(X, W, nullptr, out, M, N, K, ldx, ldw, ldo, out_f32, 1, 0, 1, PB_ACT_GELU_TANH, 0.f, 0.f, status, stream);
}

// The gated form with the clamped unit in its epilogue: out [M, N] = a * sigmoid(alpha a) * (b + 1) with
// a = min(x Wg^T, limit) and b = clamp(x Wu^T, -limit, limit); W is [2 N, K], N gate rows then N up rows.
PB_API int pb_gemm_stream_clamped_glu_bf16(const void* X, const void* W, void* out, int M, int N, int K, long long ldx,
                                           long long ldw, long long ldo, int out_f32, float limit, float alpha, int* status,
                                           cudaStream_t stream) {
    PB_REQUIRE(limit > 0.f, "gemm_stream: the clamped unit needs a positive limit");
    return gs_run(X, W, nullptr, out, M, N, K, ldx, ldw, ldo, out_f32, 1, 0, 1, PB_ACT_CLAMPED, limit, alpha, status, stream);
}

// An activation without constants in the epilogue: gated (W [2 N, K], N gate rows then N up rows) relu(x Wg^T) * (x Wu^T) for
// PB_ACT_RELU; plain (W [N, K]) relu(x W^T)^2 for PB_ACT_RELU2.
PB_API int pb_gemm_stream_act_bf16(const void* X, const void* W, void* out, int M, int N, int K, long long ldx, long long ldw, long long ldo,
                                   int out_f32, int gated, int act, int* status, cudaStream_t stream) {
    PB_REQUIRE(gated ? (act == PB_ACT_RELU || act == PB_ACT_SILU || act == PB_ACT_GELU_TANH) : (act == PB_ACT_RELU2 || act == PB_ACT_NONE),
               "gemm_stream: activation %d in the %s form", act, gated ? "gated" : "plain");
    return gs_run(X, W, nullptr, out, M, N, K, ldx, ldw, ldo, out_f32, 1, 0, gated, act, 0.f, 0.f, status, stream);
}

// The product that a sublayer ends with, the residual add and the squashing that follows, in one kernel: res [M, N] float32
// (dense) += x W^T, out [M, N] bfloat16 = tanh(slope * res) * gain + shift with gain, shift float32 [N].
PB_API int pb_gemm_stream_add_tanh_bf16(const void* X, const void* W, float* res, float slope, const float* gain, const float* shift, void* out,
                                        int M, int N, int K, long long ldx, long long ldw, int* status, cudaStream_t stream) {
    PB_REQUIRE(res && gain && shift, "gemm_stream: null pointer");
    return gs_run(X, W, nullptr, out, M, N, K, ldx, ldw, N, 0, 1, 0, 0, PB_ACT_NONE, 0.f, 0.f, status, stream, GsResidual{res, gain, shift, slope});
}
