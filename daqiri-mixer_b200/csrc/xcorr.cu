// xcorr.cu -- lower-triangle complex Hermitian GEMM V = X X^H per channel on
// tcgen05 int8 tensor cores (sm_100a).
//
// Replaces cgemm_blk_t<ACC> (reference src/cgemm.cuh:28-69).  The reference
// issues four wmma 16x16x16 products per tile from global memory, negates the
// A_im fragment (src/cgemm.cuh:52, wraps for -128) and computes the full
// square.  Here, per channel c and 128 x 128 tile (i, j) with j <= i, the B
// operand is the 256-row stack [Xr_j ; Xi_j] (the two plane tiles sit next to
// each other in shared memory), so two M=128, N=256 MMAs per 32-sample step
// produce all four real products:
//
//   D1 = Xr_i [Xr_j ; Xi_j]^T = [ R1 | P2 ]      (TMEM columns   0..255)
//   D2 = Xi_i [Xr_j ; Xi_j]^T = [ P1 | R2 ]      (TMEM columns 256..511)
//   Re V = R1 + R2,  Im V = P1 - P2              (epilogue)
//
// No operand is ever negated, so every int8 input, -128 included, is exact.
// Diagonal tiles (i == j) use the A tiles [Xr_i ; Xi_i] as B and load half
// the bytes.  When N is not a multiple of 128 the last block holds r < 128
// antennas; its tiles put that block on the N side with r16 = r rounded up to
// 16 rows per plane (N = 2 r16): tile (nb-1, j < nb-1) is computed as its
// conjugate transpose, A = block j and B = [Xr_nb-1 ; Xi_nb-1] (r16 rows
// each, one TMA box over both planes), and written back transposed; tile
// (nb-1, nb-1) has its own block on both sides (own_rows).  Operands come from the corner-turned
// planes [2][C][N][kt] through 4-D TMA tensor loads (128-byte swizzle,
// 128 x 128-byte boxes)
// into a 3-deep shared-memory ring.  One elected thread issues all
// tcgen05.mma; the int32 accumulators stay in TMEM for the whole K range of
// the launch; eight epilogue warps read them back with tcgen05.ld into
// registers, release TMEM and add them into the tile-packed int32 or int64
// cube in HBM while the next tile's MMAs run.
//
// What bounds it: the int8 tensor rate at the clock the 1000 W cap leaves for
// long K, the cube's read-modify-write in HBM for short K.  One tile's four
// products fill TMEM, so the next tile waits for the drain alone (850 clocks;
// 1000 from its last MMA to the next tile's first) instead of for the adds: 128 result registers a
// thread, which the register split below pays for.  One B200, against adds straight from TMEM: 4096
// elements x 64 channels, K 2048 with its corner-turn 5.81 -> 5.49 ms; 1024 x
// 64, K 2048 int64 328 -> 301 us, K 8192 802 -> 782 us; 200 x 128, K 1536
// int32 and flush 121 -> 117 us; 48 small arrays in one launch 573 -> 557 us;
// 1024 elements, K 1024 and K 32 768: the same within 0.4 %.  D1 is drained
// first, and the next tile's first D1 MMAs run while D2 is read: 4096 x 64, K
// 2048 step another 2 %, int32 at K 1024 3-4 %.
//
// Warp roles (384 threads, one CTA per SM, persistent over work items):
//   warp 0      TMA producer; picks the CTA's next item and passes its index
//               to the other roles through a shared-memory ring
//   warp 1      TMEM allocator + MMA issuer
//   warps 2, 3  idle (they complete the first warpgroup, whose registers go
//               to the epilogue)
//   warps 4..11 epilogue (TMEM lane quadrant = warp % 4, every other
//               16-column chunk)
// The grid is one CTA per item, of which one per SM runs at a time; the
// running CTAs take over the waiting ones' items in list order (cluster launch
// control), so they stay on neighbouring items, which share operand blocks in
// L2, whatever each item costs.  Launches with few items per SM, and those
// with a CTA limit, hand CTA b the items b, b + grid, ... (launch_grid).
#include "common.cuh"
#include "xcorr.cuh"
#include <cstdlib>
#include <cstring>

namespace mixer {

namespace {

// Pipeline geometry (build-time options): samples per stage (128 with the
// 128-byte swizzle or 64 with the 64-byte swizzle) and stage count.
#ifndef MIXER_XCORR_KC
#define MIXER_XCORR_KC 128
#endif
#ifndef MIXER_XCORR_STAGES
#define MIXER_XCORR_STAGES 3
#endif
constexpr int kTile = 128;                       // tile rows = cols
constexpr int kWorkChunk = 128;                  // samples per work-list K unit
constexpr int kKc = MIXER_XCORR_KC;              // samples (bytes) per pipeline stage
constexpr int kSubPerChunk = kWorkChunk / kKc;
constexpr int kStages = MIXER_XCORR_STAGES;
constexpr int kTileBytes = kTile * kKc;
constexpr int kStageBytes = 4 * kTileBytes;      // Ar, Ai, Br, Bi
static_assert(kKc == 64 || kKc == 128, "stage of 64 or 128 samples");
constexpr int kEpiGroups = 2;                    // epilogue warps per TMEM lane quadrant
constexpr int kEpiWarps = 4 * kEpiGroups;
constexpr int kEpiCols = kTile / kEpiGroups;     // 64 columns per warp
constexpr int kEpiChunks = kEpiCols / 16;        // 16-column chunks per warp
constexpr int kEpiWarp0 = 4;                     // first epilogue warp
constexpr int kThreads = 32 * (kEpiWarp0 + kEpiWarps);
constexpr int kPairThreads = 64 + 32 * kEpiWarps;
constexpr int kBarBytes = 512;
// Item ring: the producer publishes each item index to the MMA and epilogue
// warps through kItemSlots slots after the pipeline barriers.
constexpr int kItemSlots = 8;
constexpr int kItemBar0 = 24;                    // first ring barrier (uint64 index)
static_assert(2 * MIXER_XCORR_STAGES + 6 <= kItemBar0, "barrier area");
constexpr int kClcSlot = (kItemBar0 + 3 * kItemSlots) * 8;   // 16-byte launch-control answer
static_assert(kClcSlot % 16 == 0 && kClcSlot + 16 <= kBarBytes, "barrier area");
// Transpose area of the ragged tiles: per epilogue warp 32 rows of 16 words,
// padded to 17 (row writes and the two-rows-per-read pattern are conflict-free).
constexpr int kXposeStride = 17;
constexpr int kXposeBytes = kEpiWarps * 32 * kXposeStride * 4;
constexpr int kSmemBase = kStages * kStageBytes + 1024 + kBarBytes;
constexpr int kSmemBytes = kSmemBase + kXposeBytes;   // the most a launch asks for
static_assert(kSmemBytes <= 232448, "shared memory");
constexpr uint32_t kTmemCols = 512;              // D1 (256) + D2 (256)
constexpr uint32_t kIdesc = idesc_i8(128, 256);

struct XcorrArgs {
    int32_t nant, ntiles;   // ntiles: tiles of a channel
    int32_t kbeg, nkc;   // first sample, number of 128-sample chunks
    int32_t mode;
    int32_t dynamic;     // 1: one CTA per item, taken over by the running ones; 0: CTA b
                         // takes items b, b + grid, ...
    // Single array: the first nwhole tiles are one item each, the last nsplit
    // several, `kpart` chunks of the range each.
    int32_t nsplit, kpart;
    int64_t nwhole;
    int64_t nwork;       // items
    void* vis;
    int32_t* err;
    // Batched mode (work != nullptr): per-array tensor maps, problems, work list.
    // Two maps per array: [2p] the 128-row operand boxes, [2p + 1] the ragged
    // last block's box over both planes.
    const CUtensorMap* tmaps;
    const XcorrProblem* probs;
    const XcorrWork* work;
};

__device__ __forceinline__ void decode_tile(int t, int& i, int& j) {
    int ii = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while ((ii + 1) * (ii + 2) / 2 <= t) ++ii;
    while (ii * (ii + 1) / 2 > t) --ii;
    i = ii;
    j = t - ii * (ii + 1) / 2;
}

__device__ __forceinline__ uint64_t sdesc(uint32_t saddr) {
    return kKc == 128 ? sdesc_sw128(saddr) : sdesc_sw64(saddr);
}

struct Item {
    const CUtensorMap* map;
    const CUtensorMap* map_tail;
    void* vis;
    int c, t, i, j, kbeg, kc0, nkc, mode, ntiles;
    int tail;   // rows per plane of the ragged last block on the N side (0: full tile)
    int rows;   // rows of the MMA's M side that hold antennas
};

// A ragged block's diagonal tile has its block for both operands.  Where it pays
// (own_rows) no 128-row A is loaded: the MMAs read A from B's rows, Xr from
// the first on and Xi from row it.tail on (the M rows past it.tail are whatever
// lies there, and not added; stores want zeros there and keep the 128-row A),
// and a stage holds several K steps.  Arrays of one block: 32 elements x 256
// channels, K 512 8.9 -> 8.0 us, K 4096 35.5 -> 28.1; 27 x 85, K 5952 26.2 ->
// 20.4; 64 x 592, K 1024 31.4 -> 28.4.  Behind other blocks only long ranges
// gain: 200 x 128, K 4096 76.0 -> 72.6, but 300 x 85, K 1024 48.7 -> 50.6.
constexpr int kOwnChunks = 12;
__device__ __forceinline__ bool own_rows(const Item& it) {
    return it.tail && it.i == it.j && (it.i == 0 || it.nkc >= kOwnChunks) &&
           it.mode != MIXER_VIS_STORE_I32;
}
// K steps of such a tile in a stage: all, if they fit, else what fits, at most 8
// and a third of them (40 x 128, K 1024 with five and three 9.6 us, in twos 9.0).
__device__ __forceinline__ int own_steps(int r16, int steps) {
    const int fit = r16 <= 32 ? 8 : r16 <= 48 ? 5 : r16 <= 64 ? 4 : r16 <= 80 ? 3 : 2;
    return steps <= fit ? steps : max(1, min(fit, steps / 3));
}
static_assert(8 * 2 * 32 * kKc <= kStageBytes && 5 * 2 * 48 * kKc <= kStageBytes &&
                  4 * 2 * 64 * kKc <= kStageBytes && 3 * 2 * 80 * kKc <= kStageBytes &&
                  2 * 2 * 112 * kKc <= kStageBytes,
              "K steps of a ragged diagonal tile in a stage");
// The M rows past the block reach furthest beyond a stage with 32 rows (8 K
// steps fill it): behind the last stage they read the barriers and the
// transpose area, which every launch with a ragged array has.
static_assert((7 * 2 * 32 + 32 + kTile) * kKc - kStageBytes <= kBarBytes + kXposeBytes,
              "rows past a ragged block stay inside the launch's shared memory");

// Rows per plane of the last 128-row block rounded up to 16 (128 when full).
__host__ __device__ __forceinline__ int tail_rows(int nant) {
    const int r = nant - ((nant - 1) / kTile) * kTile;
    return (r + 15) & ~15;
}

__device__ __forceinline__ Item get_item(const XcorrArgs& a, const CUtensorMap* pmap,
                                         const CUtensorMap* pmap_tail, int64_t w) {
    Item it;
    int nant;
    if (a.work == nullptr) {
        it.kc0 = 0;
        it.nkc = a.nkc;
        if (w >= a.nwhole) {          // K ranges of the last tiles, one range after the other
            const int part = (int)(w - a.nwhole) / a.nsplit;
            w -= (int64_t)part * a.nsplit;
            it.kc0 = part * a.kpart;
            it.nkc = min(a.kpart, a.nkc - it.kc0);
        }
        it.c = (int)(w / a.ntiles);
        it.t = (int)(w - (int64_t)it.c * a.ntiles);
        it.map = pmap;
        it.map_tail = pmap_tail;
        nant = a.nant;
        it.vis = a.vis;
        it.kbeg = a.kbeg;
        it.mode = a.mode;
        it.ntiles = a.ntiles;
    } else {
        const XcorrWork wk = a.work[w];
        const XcorrProblem& pr = a.probs[wk.prob];
        it.c = (int)wk.chan;
        it.t = (int)wk.tile;
        it.map = a.tmaps + 2 * wk.prob;
        it.map_tail = it.map + 1;
        nant = pr.nant;
        it.vis = pr.vis;
        it.kbeg = pr.kbeg;
        it.kc0 = (int)wk.kc0;
        it.nkc = (int)wk.nkc;
        it.mode = pr.mode;
        it.ntiles = pr.ntiles;
    }
    decode_tile(it.t, it.i, it.j);
    const int r16 = tail_rows(nant);
    it.tail = (r16 < kTile && it.i == (nant - 1) / kTile) ? r16 : 0;
    it.rows = it.i == it.j ? min(nant - it.i * kTile, kTile) : kTile;
    return it;
}

// Chunks of item w (of a K range, at most).
__device__ __forceinline__ int item_chunks(const XcorrArgs& a, int64_t w) {
    if (a.work) return (int)a.work[w].nkc;
    return w < a.nwhole ? a.nkc : a.kpart;
}

// Four 32x32b.x16 TMEM loads (16 columns each) and the wait, in one asm
// statement so no use of the results can be scheduled before the wait.
__device__ __forceinline__ void tmem_ld4_x16(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t (&r)[4][16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%64];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%65];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47}, [%66];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%67];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0][0]), "=r"(r[0][1]), "=r"(r[0][2]), "=r"(r[0][3]), "=r"(r[0][4]),
          "=r"(r[0][5]), "=r"(r[0][6]), "=r"(r[0][7]), "=r"(r[0][8]), "=r"(r[0][9]),
          "=r"(r[0][10]), "=r"(r[0][11]), "=r"(r[0][12]), "=r"(r[0][13]), "=r"(r[0][14]),
          "=r"(r[0][15]), "=r"(r[1][0]), "=r"(r[1][1]), "=r"(r[1][2]), "=r"(r[1][3]),
          "=r"(r[1][4]), "=r"(r[1][5]), "=r"(r[1][6]), "=r"(r[1][7]), "=r"(r[1][8]),
          "=r"(r[1][9]), "=r"(r[1][10]), "=r"(r[1][11]), "=r"(r[1][12]), "=r"(r[1][13]),
          "=r"(r[1][14]), "=r"(r[1][15]), "=r"(r[2][0]), "=r"(r[2][1]), "=r"(r[2][2]),
          "=r"(r[2][3]), "=r"(r[2][4]), "=r"(r[2][5]), "=r"(r[2][6]), "=r"(r[2][7]),
          "=r"(r[2][8]), "=r"(r[2][9]), "=r"(r[2][10]), "=r"(r[2][11]), "=r"(r[2][12]),
          "=r"(r[2][13]), "=r"(r[2][14]), "=r"(r[2][15]), "=r"(r[3][0]), "=r"(r[3][1]),
          "=r"(r[3][2]), "=r"(r[3][3]), "=r"(r[3][4]), "=r"(r[3][5]), "=r"(r[3][6]),
          "=r"(r[3][7]), "=r"(r[3][8]), "=r"(r[3][9]), "=r"(r[3][10]), "=r"(r[3][11]),
          "=r"(r[3][12]), "=r"(r[3][13]), "=r"(r[3][14]), "=r"(r[3][15])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3)
        : "memory");
}

// Eight loads of 16 columns (four of D1's first half 32 columns apart, four of
// its second half) and the wait, likewise in one statement.
__device__ __forceinline__ void tmem_ld8_x16(uint32_t a, uint32_t b, uint32_t (&p)[64],
                                             uint32_t (&q)[64]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%128];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%129];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47}, [%130];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%131];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%64,%65,%66,%67,%68,%69,%70,%71,%72,%73,%74,%75,%76,%77,%78,%79}, [%132];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%80,%81,%82,%83,%84,%85,%86,%87,%88,%89,%90,%91,%92,%93,%94,%95}, [%133];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%96,%97,%98,%99,%100,%101,%102,%103,%104,%105,%106,%107,%108,%109,%110,%111}, [%134];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%112,%113,%114,%115,%116,%117,%118,%119,%120,%121,%122,%123,%124,%125,%126,%127}, [%135];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(p[0]), "=r"(p[1]), "=r"(p[2]), "=r"(p[3]), "=r"(p[4]), "=r"(p[5]), "=r"(p[6]),
          "=r"(p[7]), "=r"(p[8]), "=r"(p[9]), "=r"(p[10]), "=r"(p[11]), "=r"(p[12]),
          "=r"(p[13]), "=r"(p[14]), "=r"(p[15]), "=r"(p[16]), "=r"(p[17]), "=r"(p[18]),
          "=r"(p[19]), "=r"(p[20]), "=r"(p[21]), "=r"(p[22]), "=r"(p[23]), "=r"(p[24]),
          "=r"(p[25]), "=r"(p[26]), "=r"(p[27]), "=r"(p[28]), "=r"(p[29]), "=r"(p[30]),
          "=r"(p[31]), "=r"(p[32]), "=r"(p[33]), "=r"(p[34]), "=r"(p[35]), "=r"(p[36]),
          "=r"(p[37]), "=r"(p[38]), "=r"(p[39]), "=r"(p[40]), "=r"(p[41]), "=r"(p[42]),
          "=r"(p[43]), "=r"(p[44]), "=r"(p[45]), "=r"(p[46]), "=r"(p[47]), "=r"(p[48]),
          "=r"(p[49]), "=r"(p[50]), "=r"(p[51]), "=r"(p[52]), "=r"(p[53]), "=r"(p[54]),
          "=r"(p[55]), "=r"(p[56]), "=r"(p[57]), "=r"(p[58]), "=r"(p[59]), "=r"(p[60]),
          "=r"(p[61]), "=r"(p[62]), "=r"(p[63]), "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]),
          "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7]), "=r"(q[8]), "=r"(q[9]), "=r"(q[10]),
          "=r"(q[11]), "=r"(q[12]), "=r"(q[13]), "=r"(q[14]), "=r"(q[15]), "=r"(q[16]),
          "=r"(q[17]), "=r"(q[18]), "=r"(q[19]), "=r"(q[20]), "=r"(q[21]), "=r"(q[22]),
          "=r"(q[23]), "=r"(q[24]), "=r"(q[25]), "=r"(q[26]), "=r"(q[27]), "=r"(q[28]),
          "=r"(q[29]), "=r"(q[30]), "=r"(q[31]), "=r"(q[32]), "=r"(q[33]), "=r"(q[34]),
          "=r"(q[35]), "=r"(q[36]), "=r"(q[37]), "=r"(q[38]), "=r"(q[39]), "=r"(q[40]),
          "=r"(q[41]), "=r"(q[42]), "=r"(q[43]), "=r"(q[44]), "=r"(q[45]), "=r"(q[46]),
          "=r"(q[47]), "=r"(q[48]), "=r"(q[49]), "=r"(q[50]), "=r"(q[51]), "=r"(q[52]),
          "=r"(q[53]), "=r"(q[54]), "=r"(q[55]), "=r"(q[56]), "=r"(q[57]), "=r"(q[58]),
          "=r"(q[59]), "=r"(q[60]), "=r"(q[61]), "=r"(q[62]), "=r"(q[63])
        : "r"(a), "r"(a + 32), "r"(a + 64), "r"(a + 96), "r"(b), "r"(b + 32), "r"(b + 64),
          "r"(b + 96)
        : "memory");
}

// Register split: the launch gives 384 threads 168 registers each; the four
// control warps keep kCtrlRegs and the eight epilogue warps take kEpiRegs,
// which hold a warp's whole share of a tile (128 values a thread) and 64 more
// on their way from TMEM.
constexpr int kCtrlRegs = 72, kEpiRegs = 216;
static_assert(4 * kCtrlRegs + 8 * kEpiRegs <= 12 * 168, "register split");
template <int R>
__device__ __forceinline__ void reg_inc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R));
}
template <int R>
__device__ __forceinline__ void reg_dec() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R));
}

// Adds into the cube.  The cube's address comes out of a table, so atomicAdd
// would test it for shared memory at every call: 138 KB of code where these
// make 80 KB, and an epilogue that any change to its code could slow by 2-100 %.
// 48 small arrays in one launch 517 -> 493 us; 200 x 128, K 1024 69 -> 50 us.
__device__ __forceinline__ void red_add(unsigned long long* p, int32_t x) {
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)),
                 "l"((long long)x)
                 : "memory");
}
__device__ __forceinline__ void red_add(int* p, int32_t x) {
    asm volatile("red.relaxed.gpu.global.add.s32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)),
                 "r"(x)
                 : "memory");
}

// Spreads a tile's adds over the next tile's MMAs: after every kPaceCols columns
// the warp sleeps until its share of the time has passed.  The MMAs at full
// rate take all that one SM can read from L2 (64 bytes a clock), so operands
// that come late are not made up for, and while the adds leave in one burst
// the operand loads get about a third of that: 16 chunks of MMAs took 28 000
// clocks beside the int64 adds, against 16 400 alone; paced they take 25 600
// (int32: 18 500).  One B200, without -> with: int64, 4096 x 8, K 2048 531 -> 488 us, K
// 3072 685 -> 607, K 8192 1553 -> 1441; 1024 x 64, K 2048 298 -> 279; 640 x 48,
// K 8192 257 -> 247; int32, 4096 x 8, K 1024 263 -> 254, K 2048 413 -> 370.
// Shorter tiles are bound by the cube's traffic itself and are not paced.  The
// time spread over is the MMA time (1024 clocks a chunk) of the tile or of the
// next one, whichever is shorter: adds that outlast the next tile's MMAs hold
// up the tile after it (K ranges behind whole rounds, 128 x 760, K 8192 333 ->
// 322 us against the tile's own time).  1.2 times that for int64 (1.0: 0-7 %
// slower, 0.9: 3-8 %), at most 64 x kPaceMax clocks.
constexpr int kPaceCols = 4;
constexpr int kPaceChunks64 = 16, kPaceChunks32 = 8;   // shortest tile paced
constexpr int kPaceMax64 = 600, kPaceMax32 = 400;      // clocks per column

struct Pace {
    uint32_t t0, dt, due;   // start, clocks per step, clocks after t0 at which the next is due
    __device__ __forceinline__ void begin(int mode, int nkc) {
        const int col = mode == MIXER_VIS_ACC_I64 ? min(nkc * 19, kPaceMax64)
                                                  : min(nkc * 16, kPaceMax32);
        dt = (uint32_t)(col * kPaceCols);
        due = 0;
        t0 = now();
    }
    __device__ __forceinline__ void step() {
        due += dt;
        const int32_t ahead = (int32_t)(due - (now() - t0));
        // a quarter of the clocks left in ns: shorter than they are at any clock rate
        if (ahead > 48) asm volatile("nanosleep.u32 %0;" ::"r"(ahead / 4) : "memory");
    }
    static __device__ __forceinline__ uint32_t now() {
        uint32_t c;
        asm volatile("mov.u32 %0, %%clock;" : "=r"(c)::"memory");
        return c;
    }
};

// Adds (or stores) 16 elements of one row of TMEM into the cube: columns e of
// the re plane, kTile apart, and of the im plane kTile * kTile further on.
template <bool kPaced>
__device__ __forceinline__ void store16(const Item& it, size_t e0, const uint32_t* re,
                                        const uint32_t* im, Pace& pace) {
    if (it.mode == MIXER_VIS_ACC_I64) {
        unsigned long long* v = reinterpret_cast<unsigned long long*>(it.vis) + e0;
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            red_add(v + e * kTile, (int32_t)re[e]);
            red_add(v + e * kTile + kTile * kTile, (int32_t)im[e]);
            if (kPaced && e % kPaceCols == kPaceCols - 1) pace.step();
        }
    } else if (it.mode == MIXER_VIS_ACC_I32) {
        int* v = reinterpret_cast<int*>(it.vis) + e0;
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            red_add(v + e * kTile, (int32_t)re[e]);
            red_add(v + e * kTile + kTile * kTile, (int32_t)im[e]);
            if (kPaced && e % kPaceCols == kPaceCols - 1) pace.step();
        }
    } else {
        int* v = reinterpret_cast<int*>(it.vis) + e0;
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            v[e * kTile] = (int)re[e];
            v[e * kTile + kTile * kTile] = (int)im[e];
            if (kPaced && e % kPaceCols == kPaceCols - 1) pace.step();
        }
    }
}

// Adds (or stores) one element of the cube, in the item's mode.
__device__ __forceinline__ void store1(const Item& it, size_t e, int32_t x) {
    if (it.mode == MIXER_VIS_ACC_I64) {
        red_add(reinterpret_cast<unsigned long long*>(it.vis) + e, x);
    } else if (it.mode == MIXER_VIS_ACC_I32) {
        red_add(reinterpret_cast<int*>(it.vis) + e, x);
    } else {
        reinterpret_cast<int*>(it.vis)[e] = x;
    }
}

__global__ void __launch_bounds__(kThreads, 1)
    k_xcorr_tri(const __grid_constant__ CUtensorMap tmap,
                const __grid_constant__ CUtensorMap tmap_tail, const XcorrArgs args) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;           // 1 KiB aligned (swizzle atoms)
    uint8_t* gbase = smem_raw + (base - raw);
    uint64_t* bars = reinterpret_cast<uint64_t*>(gbase + kStages * kStageBytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int32_t* xchg = reinterpret_cast<int32_t*>(gbase + kStages * kStageBytes + kBarBytes);
    volatile int64_t* witems = reinterpret_cast<volatile int64_t*>(bars + kItemBar0 + 2 * kItemSlots);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int FULL = 0, EMPTY = kStages, ACCF = 2 * kStages, ACCE = 2 * kStages + 1,
              DRAIN = 2 * kStages + 2, CLC = 2 * kStages + 3, ACCE2 = 2 * kStages + 5,
              IFULL = kItemBar0, IEMPTY = kItemBar0 + kItemSlots;
    auto bar = [&](int k) { return smem_u32(&bars[k]); };

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(bar(FULL + s), 1);
            mbar_init(bar(EMPTY + s), 1);
        }
        mbar_init(bar(ACCF), 1);
        mbar_init(bar(ACCE), 32 * kEpiWarps);
        mbar_init(bar(ACCE2), 32 * kEpiWarps);
        mbar_init(bar(DRAIN), 1);
        mbar_init(bar(CLC), 1);
        for (int s = 0; s < kItemSlots; ++s) {
            mbar_init(bar(IFULL + s), 1);
            mbar_init(bar(IEMPTY + s), 1 + kEpiWarps);   // the MMA thread, one per epilogue warp
        }
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 0 && lane == 0 && args.work == nullptr) {
        prefetch_tmap(&tmap);
        prefetch_tmap(&tmap_tail);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();   // the planes, the cube and the work list are other kernels' until here

    if (warp < kEpiWarp0) reg_dec<kCtrlRegs>();
    if (warp == 0) {
        // ------------------------------------------------------------ producer
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            int64_t issued = 0;
            bool ok = true;
            int islot = 0;
            uint32_t iphase = 0;
            int64_t w = blockIdx.x;
            uint32_t clc_phase = 0;
            bool asked = false;   // a request for the next item is under way
            const uint32_t clc_slot = smem_u32(gbase + kStages * kStageBytes + kClcSlot);
            while (ok) {
                // publish the item (or the end mark -1) to the MMA and epilogue warps
                if (w >= args.nwork) w = -1;
                if (!mbar_wait(bar(IEMPTY + islot), iphase ^ 1u, abort_flag)) {
                    ok = false;
                    break;
                }
                witems[islot] = w;
                mbar_arrive(bar(IFULL + islot));
                if (++islot == kItemSlots) {
                    islot = 0;
                    iphase ^= 1u;
                }
                if (w < 0) break;
                if (args.dynamic) {
                    // ask for the next item now: the answer comes during this one
                    mbar_expect_tx(bar(CLC), 16);
                    clc_request(clc_slot, bar(CLC));
                    asked = true;
                }
                const Item it = get_item(args, &tmap, &tmap_tail, w);
                const bool diag = (it.i == it.j);
                const uint32_t bytes = it.tail ? 2 * kTileBytes + 2 * it.tail * kKc
                                               : (diag ? 2 * kTileBytes : 4 * kTileBytes);
                // A block: block j for a transposed ragged tile, else block i
                const int ia = (it.tail && !diag) ? it.j : it.i;
                const bool own = own_rows(it);
                if (own) {
                    const int steps = it.nkc * kSubPerChunk, per = own_steps(it.tail, steps);
                    const uint32_t each = 2 * it.tail * kKc;
                    for (int kc = 0; kc < steps; kc += per) {
                        if (!mbar_wait(bar(EMPTY + stage), phase ^ 1u, abort_flag)) {
                            ok = false;
                            break;
                        }
                        const int n = min(per, steps - kc);
                        const uint32_t fb = bar(FULL + stage);
                        mbar_expect_tx(fb, n * each);
                        for (int u = 0; u < n; ++u)
                            tma_load_4d(base + stage * kStageBytes + u * each, it.map_tail, fb,
                                        it.kbeg + it.kc0 * kWorkChunk + (kc + u) * kKc,
                                        it.i * kTile, it.c, 0);
                        ++issued;
                        if (++stage == kStages) {
                            stage = 0;
                            phase ^= 1u;
                        }
                    }
                }
                for (int kc = 0; !own && kc < it.nkc * kSubPerChunk; ++kc) {
                    if (!mbar_wait(bar(EMPTY + stage), phase ^ 1u, abort_flag)) {
                        ok = false;
                        break;
                    }
                    const uint32_t sb = base + stage * kStageBytes;
                    const uint32_t fb = bar(FULL + stage);
                    mbar_expect_tx(fb, bytes);
                    const int k = it.kbeg + it.kc0 * kWorkChunk + kc * kKc;
                    tma_load_4d(sb + 0 * kTileBytes, it.map, fb, k, ia * kTile, it.c, 0);
                    tma_load_4d(sb + 1 * kTileBytes, it.map, fb, k, ia * kTile, it.c, 1);
                    if (it.tail) {
                        // [Xr ; Xi] of the ragged block, it.tail rows each, one box
                        tma_load_4d(sb + 2 * kTileBytes, it.map_tail, fb, k, it.i * kTile, it.c, 0);
                    } else if (!diag) {
                        tma_load_4d(sb + 2 * kTileBytes, it.map, fb, k, it.j * kTile, it.c, 0);
                        tma_load_4d(sb + 3 * kTileBytes, it.map, fb, k, it.j * kTile, it.c, 1);
                    }
                    ++issued;
                    if (++stage == kStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                if (!args.dynamic) {
                    w += gridDim.x;
                } else if (ok && mbar_wait(bar(CLC), clc_phase, abort_flag)) {
                    clc_phase ^= 1u;
                    asked = false;
                    w = clc_answer(clc_slot);
                } else {
                    ok = false;
                }
            }
            if (!ok) {
                if (args.err) atomicOr(args.err, 1);
                *abort_flag = 1;
                // Let the copies already issued land before the CTA exits.
                for (int64_t q = issued - 1; q >= 0 && q >= issued - kStages; --q)
                    mbar_wait(bar(FULL + (int)(q % kStages)), (uint32_t)((q / kStages) & 1));
                // Take over the CTAs that have not started, so that the launch
                // ends here instead of giving each of them its own time-out.
                while (args.dynamic && w >= 0) {
                    if (!asked) {
                        mbar_expect_tx(bar(CLC), 16);
                        clc_request(clc_slot, bar(CLC));
                    }
                    asked = false;
                    if (!mbar_wait(bar(CLC), clc_phase)) break;
                    clc_phase ^= 1u;
                    w = clc_answer(clc_slot);
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            const uint32_t t_d1 = tmem, t_d2 = tmem + 256;
            int islot = 0;
            uint32_t iphase = 0;
            while (true) {
                if (!mbar_wait(bar(IFULL + islot), iphase, abort_flag)) {
                    ok = false;
                    break;
                }
                const int64_t w = witems[islot];
                mbar_arrive(bar(IEMPTY + islot));
                if (++islot == kItemSlots) {
                    islot = 0;
                    iphase ^= 1u;
                }
                if (w < 0) break;
                const Item it = get_item(args, &tmap, &tmap_tail, w);
                const bool diag = (it.i == it.j);
                const uint32_t id1 = it.tail ? idesc_i8(128, 2 * it.tail) : kIdesc;
                if (!mbar_wait(bar(ACCE), acc_phase ^ 1u, abort_flag)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const bool own = own_rows(it);
                if (own) {
                    const int steps = it.nkc * kSubPerChunk, per = own_steps(it.tail, steps);
                    const uint64_t each = (uint64_t)((2 * it.tail * kKc) >> 4);
                    if (!mbar_wait(bar(ACCE2), acc_phase ^ 1u, abort_flag)) ok = false;
                    tc_fence_after();
                    for (int kc = 0; ok && kc < steps; kc += per) {
                        if (!mbar_wait(bar(FULL + stage), phase, abort_flag)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        uint64_t b = sdesc(base + stage * kStageBytes);
                        const uint64_t im = (uint64_t)((it.tail * kKc) >> 4);
                        const int n = min(per, steps - kc);
#pragma unroll 1
                        for (int u = 0; u < n; ++u, b += each) {
                            const uint32_t acc = kc + u > 0 ? 1u : 0u;
#pragma unroll
                            for (int kk = 0; kk < kKc / 32; ++kk) {
                                mma_i8(t_d1, b + (kk * 2), b + (kk * 2), id1, kk > 0 ? 1u : acc);
                                mma_i8(t_d2, b + im + (kk * 2), b + (kk * 2), id1,
                                       kk > 0 ? 1u : acc);
                            }
                        }
                        tc_commit(bar(EMPTY + stage));
                        if (++stage == kStages) {
                            stage = 0;
                            phase ^= 1u;
                        }
                    }
                }
                for (int kc = 0; !own && kc < it.nkc * kSubPerChunk; ++kc) {
                    if (!mbar_wait(bar(FULL + stage), phase, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sb = base + stage * kStageBytes;
                    const uint64_t ar = sdesc(sb);
                    const uint64_t ai = sdesc(sb + kTileBytes);
                    // 256-row B operand [Xr_j ; Xi_j]: two adjacent tiles (2 it.tail
                    // rows for a ragged block)
                    const uint64_t b = (diag && !it.tail) ? ar : sdesc(sb + 2 * kTileBytes);
                    if (kc == 0) {
                        // the first stage's D1 products while the epilogue reads D2
#pragma unroll
                        for (int kk = 0; kk < kKc / 32; ++kk)
                            mma_i8(t_d1, ar + (kk * 2), b + (kk * 2), id1, kk > 0 ? 1u : 0u);
                        if (!mbar_wait(bar(ACCE2), acc_phase ^ 1u, abort_flag)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
#pragma unroll
                        for (int kk = 0; kk < kKc / 32; ++kk)
                            mma_i8(t_d2, ai + (kk * 2), b + (kk * 2), id1, kk > 0 ? 1u : 0u);
                    } else {
#pragma unroll
                        for (int kk = 0; kk < kKc / 32; ++kk) {
                            const uint64_t o = (uint64_t)((kk * 32) >> 4);   // 32-byte K step
                            mma_i8(t_d1, ar + o, b + o, id1, 1u);
                            mma_i8(t_d2, ai + o, b + o, id1, 1u);
                        }
                    }
                    tc_commit(bar(EMPTY + stage));   // stage free once these MMAs finish
                    if (++stage == kStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                if (!ok) break;
                tc_commit(bar(ACCF));                // accumulators complete
                acc_phase ^= 1u;
            }
            if (!ok) {
                if (args.err) atomicOr(args.err, 2);
                *abort_flag = 1;
            }
            // No MMA may still be writing TMEM when it is released.
            tc_commit(bar(DRAIN));
            mbar_wait(bar(DRAIN), 0);
        }
    } else if (warp >= kEpiWarp0) {
        // ------------------------------------------------------------ epilogue
        // Eight warps: TMEM lane quadrant warp % 4, every other 16-column chunk.
        // Each warp reads its (up to 64) columns of the four products into 128
        // registers, releases TMEM to the next tile's MMAs and then adds.
        reg_inc<kEpiRegs>();
        const int q = warp & 3;
        const int g = (warp - kEpiWarp0) >> 2;
        const int m = q * 32 + lane;
        const uint32_t tq = tmem + ((uint32_t)(q * 32) << 16);
        uint32_t acc_phase = 0;
        int islot = 0;
        uint32_t iphase = 0;
        while (true) {
            if (!mbar_wait(bar(IFULL + islot), iphase, abort_flag)) {
                if (args.err) atomicOr(args.err, 4);
                *abort_flag = 1;
                break;
            }
            const int64_t w = witems[islot];
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(IEMPTY + islot));
            if (++islot == kItemSlots) {
                islot = 0;
                iphase ^= 1u;
            }
            if (w < 0) break;
            const Item it = get_item(args, &tmap, &tmap_tail, w);
            if (!mbar_wait(bar(ACCF), acc_phase, abort_flag)) {
                if (args.err) atomicOr(args.err, 4);
                *abort_flag = 1;
                break;
            }
            tc_fence_after();
            const size_t tb = ((size_t)it.c * it.ntiles + it.t) * (size_t)(2 * kTile * kTile);
            // Columns n < nt of each product: R1 | P2 at 0 | nt, P1 | R2 at
            // 256 | 256 + nt; nt = 128 or, for the ragged last block on the N
            // side, its rows.  Transposed tile (ragged, i != j): TMEM row m is
            // column m of tile (i, j) and column n its row n, so Re = R1 + R2,
            // Im = P2 - P1.  Columns past nt are zeros (store mode writes them).
            const bool tr = it.tail && it.i != it.j;
            const int nt = it.tail ? it.tail : kTile;
            // Chunk k holds the 16 columns from 16 * (2 k + g).
            const auto n0_of = [&](int k) { return 16 * (kEpiGroups * k + g); };
            uint32_t re[kEpiCols], im[kEpiCols];
            if (!it.tail) {
                // D1 first, so that the next tile's first D1 MMAs run while D2 is read
                const uint32_t tc = tq + 16 * g;
                tmem_ld8_x16(tc, tc + 128, re, im);           // R1, P2
                tc_fence_before();
                mbar_arrive(bar(ACCE));
#pragma unroll
                for (int k = 0; k < kEpiChunks; k += 2) {
                    uint32_t r[4][16];                        // P1, R2 of two chunks
                    tmem_ld4_x16(tc + 256 + 32 * k, tc + 384 + 32 * k, tc + 288 + 32 * k,
                                 tc + 416 + 32 * k, r);
#pragma unroll
                    for (int e = 0; e < 32; ++e) {
                        re[16 * k + e] += r[2 * (e >> 4) + 1][e & 15];
                        im[16 * k + e] = r[2 * (e >> 4)][e & 15] - im[16 * k + e];
                    }
                }
            } else {
#pragma unroll
                for (int k = 0; k < kEpiChunks; ++k) {
                    const int n0 = n0_of(k);
                    uint32_t r[4][16];                        // R1, P2, P1, R2
                    if (n0 < nt) {
                        tmem_ld4_x16(tq + n0, tq + nt + n0, tq + 256 + n0, tq + 256 + nt + n0, r);
                    } else {
#pragma unroll
                        for (int e = 0; e < 16; ++e) r[0][e] = r[1][e] = r[2][e] = r[3][e] = 0;
                    }
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        re[16 * k + e] = r[0][e] + r[3][e];
                        im[16 * k + e] = tr ? r[1][e] - r[2][e] : r[2][e] - r[1][e];
                    }
                }
                tc_fence_before();
                mbar_arrive(bar(ACCE));
            }
            tc_fence_before();
            mbar_arrive(bar(ACCE2));                 // TMEM is free for the next tile
            const int ncols = it.mode == MIXER_VIS_STORE_I32 ? kTile : nt;
            const int pace_min = it.mode == MIXER_VIS_ACC_I64 ? kPaceChunks64 : kPaceChunks32;
            Pace pace;
            // Not in short launches, nor for the CTA's last tile, which no MMAs follow.
            const bool many = args.dynamic || args.nwork > 4 * (int64_t)gridDim.x;
            int beside = 0;   // chunks to spread the adds over
            if (many && it.nkc >= pace_min && !it.tail &&
                __all_sync(0xffffffffu, mbar_test(bar(IFULL + islot), iphase)) &&
                witems[islot] >= 0)
                beside = min(it.nkc, item_chunks(args, witems[islot]));
            if (beside >= pace_min) {
                pace.begin(it.mode, beside);
#pragma unroll
                for (int k = 0; k < kEpiChunks; ++k)
                    store16<true>(it, tb + (size_t)n0_of(k) * kTile + m, &re[16 * k], &im[16 * k],
                                  pace);
                acc_phase ^= 1u;
                continue;
            }
#pragma unroll
            for (int k = 0; k < kEpiChunks; ++k) {
                const int n0 = n0_of(k);
                if (n0 >= ncols) break;
                if (!tr) {
                    // rows past the last antenna would add zeros (half of a 64-element
                    // array's adds: 64 x 64, K 256 8.6 -> 7.3 us); stores write them
                    if (m < it.rows || it.mode == MIXER_VIS_STORE_I32)
                        store16<false>(it, tb + (size_t)n0 * kTile + m, &re[16 * k], &im[16 * k],
                                       pace);
                } else if (it.mode == MIXER_VIS_STORE_I32 &&
                           (reinterpret_cast<uintptr_t>(it.vis) & 15) == 0) {
                    // stores: a thread's 16 elements are contiguous, 4 x 16 bytes
                    int4* vr = reinterpret_cast<int4*>(reinterpret_cast<int*>(it.vis) + tb +
                                                       (size_t)m * kTile + n0);
                    int4* vi = vr + kTile * kTile / 4;
#pragma unroll
                    for (int e = 0; e < 16; e += 4) {
                        const uint32_t *vre = &re[16 * k + e], *vim = &im[16 * k + e];
                        vr[e / 4] = make_int4(vre[0], vre[1], vre[2], vre[3]);
                        vi[e / 4] = make_int4(vim[0], vim[1], vim[2], vim[3]);
                    }
                } else {
                    // row `lane` of the warp's 32 x 16 block -> pairs of rows,
                    // 16 consecutive elements each, per instruction
                    int32_t* xs = xchg + (warp - kEpiWarp0) * 32 * kXposeStride;
                    const int rr = lane >> 4, cc = lane & 15;
#pragma unroll
                    for (int pl = 0; pl < 2; ++pl) {
#pragma unroll
                        for (int e = 0; e < 16; ++e)
                            xs[lane * kXposeStride + e] = pl ? im[16 * k + e] : re[16 * k + e];
                        __syncwarp();
                        const size_t pb = tb + (size_t)pl * kTile * kTile + n0 + cc;
#pragma unroll 4
                        for (int s2 = 0; s2 < 16; ++s2) {
                            const int row = 2 * s2 + rr;
                            store1(it, pb + (size_t)(q * 32 + row) * kTile,
                                   xs[row * kXposeStride + cc]);
                        }
                        __syncwarp();
                    }
                }
            }
            acc_phase ^= 1u;
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

// =============================================================================
// Pair kernel: one work item per cluster of two CTAs on two SMs.
//
// tcgen05 cta_group::2.  The pair's leader (cluster rank 0) issues M 256 x
// N 256 MMAs: A's 256 rows are 128 from each CTA's shared memory, and the
// 256-row B operand [Xr_j ; Xi_j] is split with Xr_j in the leader and Xi_j
// in the peer (same offsets).  Each CTA's TMEM then holds the four products
// of its own 128-row block against column block j,
//   D1 = Xr_a [Xr_j ; Xi_j]^T = [R1 | P2],  D2 = Xi_a [Xr_j ; Xi_j]^T = [P1 | R2],
// so one item computes two tiles (a0, j), (a1, j) that share column block j.
// Per SM and 32-sample step the tensor cores read 16 KB of shared memory
// instead of 24 KB and TMA writes 12 KB instead of 16 KB: 112 instead of 160
// bytes per clock at the full MMA rate.  Stages are 48 KB, four of them.
//
// Pairing.  Column block j holds tiles (i, j), i = j .. nb-1.  Consecutive
// rows pair up; a column with an odd count leaves its last tile (nb-1, j).
// Those leftovers share ROW block nb-1, so they pair as the products
// X_j X_{nb-1}^H against B = block nb-1, and the epilogue writes tile element
// (m, n) = conj(D[n][m]) (for the diagonal tile this is D itself).  Per
// channel: f(nb) = floor(nb^2/4) regular pairs, column j's first at
// f(nb) - f(nb - j), then ceil(ceil(nb/2)/2) leftover pairs; when ceil(nb/2)
// is odd the last leftover pair has no second tile and its peer half is
// computed and discarded.
// =============================================================================
constexpr int kPairStages = 4;
constexpr int kPairStageBytes = 3 * kTileBytes;   // A_re, A_im, this CTA's half of B
constexpr int kPairSmemBytes = kPairStages * kPairStageBytes + 1024 + kBarBytes;
constexpr uint32_t kIdescPair = idesc_i8(256, 256);
static_assert(kPairSmemBytes <= 232448, "shared memory");

struct PairArgs {
    int32_t nant, nch, nblk, ntiles;
    int32_t kbeg, nkc;   // first sample, number of 128-sample chunks
    int32_t mode;
    int32_t nreg;        // regular pairs per channel
    int32_t npairs;      // pairs per channel
    int32_t pad_;
    int64_t nwork;       // nch * npairs
    void* vis;
    int32_t* err;
};

// This CTA's half of pair item w.
struct PairHalf {
    int c, a, j, t;      // channel, A row block, B column block, stored tile
    bool valid, transposed;
};

__device__ __forceinline__ int quarter_sq(int n) { return (n * n) >> 2; }

__device__ __forceinline__ PairHalf pair_half(const PairArgs& g, int64_t w, int rank) {
    PairHalf h;
    h.c = (int)(w / g.npairs);
    const int p = (int)(w - (int64_t)h.c * g.npairs);
    const int nb = g.nblk;
    if (p < g.nreg) {
        // column j = nb - n with n the smallest count whose f(n) >= q
        const int q = g.nreg - p;
        int n = (int)(2.0f * sqrtf((float)q));
        if (n < 2) n = 2;
        while (quarter_sq(n) < q) ++n;
        while (n > 2 && quarter_sq(n - 1) >= q) --n;
        h.j = nb - n;
        h.a = h.j + 2 * (quarter_sq(n) - q) + rank;
        h.t = h.a * (h.a + 1) / 2 + h.j;
        h.valid = true;
        h.transposed = false;
    } else {
        const int s = 2 * (p - g.nreg) + rank;          // leftover of column nb-1-2s
        h.j = nb - 1;
        h.valid = s < ((nb + 1) >> 1);
        h.a = h.valid ? nb - 1 - 2 * s : nb - 1;
        h.t = (nb - 1) * nb / 2 + h.a;                  // tile (nb-1, a)
        h.transposed = true;
    }
    return h;
}

__global__ void __launch_bounds__(kPairThreads, 1)
    k_xcorr_pair(const __grid_constant__ CUtensorMap tmap, const PairArgs args) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;            // same offset in both CTAs
    uint8_t* gbase = smem_raw + (base - raw);
    uint64_t* bars = reinterpret_cast<uint64_t*>(gbase + kPairStages * kPairStageBytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kPairStages + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const bool leader = (rank == 0);
    const int64_t cid = blockIdx.x >> 1, ncl = gridDim.x >> 1;
    const int FULL = 0, EMPTY = kPairStages, ACCF = 2 * kPairStages, ACCE = 2 * kPairStages + 1,
              DRAIN = 2 * kPairStages + 2;
    auto bar = [&](int k) { return smem_u32(&bars[k]); };
    // A wait that gives up stops both CTAs of the pair.
    auto raise_abort = [&]() {
        *abort_flag = 1;
        st_cluster_u32(mapa_shared(smem_u32((const void*)abort_flag), rank ^ 1u), 1u);
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < kPairStages; ++s) {
            mbar_init(bar(FULL + s), 1);      // leader: its expect_tx + both CTAs' bytes
            mbar_init(bar(EMPTY + s), 1);     // the leader's multicast commit
        }
        mbar_init(bar(ACCF), 1);
        mbar_init(bar(ACCE), 2 * 32 * kEpiWarps);   // leader: every epilogue thread of both
        mbar_init(bar(DRAIN), 1);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 0 && lane == 0) prefetch_tmap(&tmap);
    if (warp == 1) {
        tmem_alloc_pair(smem_u32(tmem_slot), kTmemCols);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    cluster_sync_all();                       // barriers and TMEM ready in both CTAs
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------------------ producer (both)
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int64_t w = cid; w < args.nwork && ok; w += ncl) {
                const PairHalf h = pair_half(args, w, (int)rank);
                for (int kc = 0; kc < args.nkc; ++kc) {
                    if (!mbar_wait(bar(EMPTY + stage), phase ^ 1u, abort_flag)) {
                        ok = false;
                        break;
                    }
                    const uint32_t sb = base + stage * kPairStageBytes;
                    const uint32_t fb = mapa_shared(bar(FULL + stage), 0);
                    if (leader) mbar_expect_tx(bar(FULL + stage), 2 * kPairStageBytes);
                    const int k = args.kbeg + kc * kKc;
                    tma_load_4d_pair(sb, &tmap, fb, k, h.a * kTile, h.c, 0);
                    tma_load_4d_pair(sb + kTileBytes, &tmap, fb, k, h.a * kTile, h.c, 1);
                    tma_load_4d_pair(sb + 2 * kTileBytes, &tmap, fb, k, h.j * kTile, h.c, (int)rank);
                    if (++stage == kPairStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
            if (!ok) {
                if (args.err) atomicOr(args.err, 1);
                raise_abort();
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (leader)
        if (lane == 0 && leader) {
            int stage = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            int64_t consumed = 0;
            const uint32_t t_d1 = tmem, t_d2 = tmem + 256;
            for (int64_t w = cid; w < args.nwork; w += ncl) {
                if (!mbar_wait(bar(ACCE), acc_phase ^ 1u, abort_flag)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                for (int kc = 0; kc < args.nkc; ++kc) {
                    if (!mbar_wait(bar(FULL + stage), phase, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sb = base + stage * kPairStageBytes;
                    const uint64_t ar = sdesc(sb);
                    const uint64_t ai = sdesc(sb + kTileBytes);
                    const uint64_t b = sdesc(sb + 2 * kTileBytes);
#pragma unroll
                    for (int kk = 0; kk < kKc / 32; ++kk) {
                        const uint64_t o = (uint64_t)((kk * 32) >> 4);   // 32-byte K step
                        const uint32_t acc = (kc > 0 || kk > 0) ? 1u : 0u;
                        mma_i8_pair(t_d1, ar + o, b + o, kIdescPair, acc);
                        mma_i8_pair(t_d2, ai + o, b + o, kIdescPair, acc);
                    }
                    tc_commit_pair(bar(EMPTY + stage), 0x3);   // stage free in both CTAs
                    ++consumed;
                    if (++stage == kPairStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                if (!ok) break;
                tc_commit_pair(bar(ACCF), 0x3);               // both CTAs' accumulators
                acc_phase ^= 1u;
            }
            if (!ok) {
                if (args.err) atomicOr(args.err, 2);
                raise_abort();
                // Let loads already counted on this CTA's barriers land.
                for (int64_t q = consumed; q < consumed + kPairStages; ++q)
                    mbar_wait(bar(FULL + (int)(q % kPairStages)), (uint32_t)((q / kPairStages) & 1));
            }
            // No MMA may still be writing either CTA's TMEM when it is released:
            // the peer deallocates only after the closing cluster barrier,
            // which this thread reaches after the wait.
            tc_commit_pair(bar(DRAIN), 0x1);
            mbar_wait(bar(DRAIN), 0);
        }
    } else {
        // ------------------------------------------------------------ epilogue (both)
        const int q = warp & 3;
        const int col0 = kEpiCols * ((warp - 2) >> 2);
        const int m = q * 32 + lane;
        const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)col0;
        const uint32_t acce = mapa_shared(bar(ACCE), 0);
        uint32_t acc_phase = 0;
        for (int64_t w = cid; w < args.nwork; w += ncl) {
            const PairHalf h = pair_half(args, w, (int)rank);
            if (!mbar_wait(bar(ACCF), acc_phase, abort_flag)) {
                if (args.err) atomicOr(args.err, 4);
                raise_abort();
                break;
            }
            tc_fence_after();
            const size_t tb = ((size_t)h.c * args.ntiles + h.t) * (size_t)(2 * kTile * kTile);
#pragma unroll 1
            for (int n0 = 0; n0 < kEpiCols; n0 += 16) {
                uint32_t r[4][16];   // R1, P2, P1, R2
                tmem_ld4_x16(trow + n0, trow + 128 + n0, trow + 256 + n0, trow + 384 + n0, r);
                if (n0 == kEpiCols - 16) {           // this warp's TMEM reads are done
                    tc_fence_before();
                    mbar_arrive_cluster(acce);
                }
                if (!h.valid) continue;
                // plain tile: element (m, n) at n * 128 + m; conjugate transpose:
                // D[m][n] goes to element (n, m), at m * 128 + n, with Im negated
                const size_t e0 = h.transposed ? tb + (size_t)m * kTile + (col0 + n0)
                                               : tb + (size_t)(col0 + n0) * kTile + m;
                const int es = h.transposed ? 1 : kTile;
                const int sg = h.transposed ? -1 : 1;
                if (args.mode == MIXER_VIS_ACC_I64) {
                    unsigned long long* v = reinterpret_cast<unsigned long long*>(args.vis) + e0;
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        red_add(v + e * es, (int32_t)(r[0][e] + r[3][e]));
                        red_add(v + e * es + kTile * kTile, sg * (int32_t)(r[2][e] - r[1][e]));
                    }
                } else if (args.mode == MIXER_VIS_ACC_I32) {
                    int* v = reinterpret_cast<int*>(args.vis) + e0;
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        red_add(v + e * es, (int32_t)(r[0][e] + r[3][e]));
                        red_add(v + e * es + kTile * kTile, sg * (int32_t)(r[2][e] - r[1][e]));
                    }
                } else {
                    int* v = reinterpret_cast<int*>(args.vis) + e0;
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        v[e * es] = (int)(r[0][e] + r[3][e]);
                        v[e * es + kTile * kTile] = sg * (int)(r[2][e] - r[1][e]);
                    }
                }
            }
            acc_phase ^= 1u;
        }
    }

    // Neither CTA leaves while the pair may still use its shared memory or TMEM.
    tc_fence_before();
    cluster_sync_all();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem, kTmemCols);
    }
}


// Dense int8 tensor-core rate with the GEMM's own instruction stream: one CTA
// per SM issues `iters` times the k_xcorr_tri K-step (two M 128 x N 256 x K 32
// kind::i8 MMAs per 32 samples, four steps per 128-byte stage) from one
// resident shared-memory stage, with no loads, into the same 512 TMEM columns.
// The operand bytes are pseudo-random so the tensor cores draw realistic power.
__global__ void __launch_bounds__(128, 1) k_mma_peak(int64_t iters, int32_t* err) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (base - raw);
    uint64_t* bar = reinterpret_cast<uint64_t*>(gbase + kStageBytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 1);
    const int warp = threadIdx.x >> 5;
    for (int q = threadIdx.x; q < kStageBytes / 4; q += blockDim.x)
        reinterpret_cast<uint32_t*>(gbase)[q] = (uint32_t)q * 2654435761u ^ 0x9e3779b9u;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(bar), 1);
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (threadIdx.x == 0) {
        const uint64_t ar = sdesc(base), ai = sdesc(base + kTileBytes), b = sdesc(base + 2 * kTileBytes);
        for (int64_t it = 0; it < iters; ++it) {
#pragma unroll
            for (int kk = 0; kk < kKc / 32; ++kk) {
                const uint64_t o = (uint64_t)((kk * 32) >> 4);
                const uint32_t acc = (it > 0 || kk > 0) ? 1u : 0u;
                mma_i8(tmem, ar + o, b + o, kIdesc, acc);
                mma_i8(tmem + 256, ai + o, b + o, kIdesc, acc);
            }
        }
        tc_commit(smem_u32(bar));
        if (!mbar_wait(smem_u32(bar), 0) && err) atomicOr(err, 2);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                              const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn get_encode() {
    static EncodeFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeFn>(p);
    }
    return fn;
}

int sm_count() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
    return n > 0 ? n : 148;
}

}  // namespace

int xcorr_encode_map(CUtensorMap* map, const int8_t* planes, int32_t nant, int32_t nch, int64_t kt,
                     int64_t kend) {
    EncodeFn enc = get_encode();
    if (!enc) return MIXER_ECUDA;
    // dim 0 ends at kend so the last chunk of a range reads zeros past it.
    const cuuint64_t dims[4] = {(cuuint64_t)kend, (cuuint64_t)nant, (cuuint64_t)nch, 2};
    const cuuint64_t strides[3] = {(cuuint64_t)kt, (cuuint64_t)kt * nant,
                                   (cuuint64_t)kt * nant * nch};
    const cuuint32_t box[4] = {kKc, kTile, 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<int8_t*>(planes), dims,
                     strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     kKc == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? MIXER_OK : MIXER_EINVAL;
}

int xcorr_encode_maps(CUtensorMap* maps, const int8_t* planes, int32_t nant, int32_t nch, int64_t kt,
                      int64_t kend) {
    int rc = xcorr_encode_map(&maps[0], planes, nant, nch, kt, kend);
    if (rc != MIXER_OK) return rc;
    EncodeFn enc = get_encode();
    if (!enc) return MIXER_ECUDA;
    // The ragged last block: tail_rows(nant) rows of both planes in one box,
    // landing as [Xr rows ; Xi rows] (the 2 r16-row B operand).  Encoded for
    // every array; unused when N is a multiple of 128.
    const cuuint64_t dims[4] = {(cuuint64_t)kend, (cuuint64_t)nant, (cuuint64_t)nch, 2};
    const cuuint64_t strides[3] = {(cuuint64_t)kt, (cuuint64_t)kt * nant,
                                   (cuuint64_t)kt * nant * nch};
    const cuuint32_t box[4] = {kKc, (cuuint32_t)tail_rows(nant), 1, 2};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = enc(&maps[1], CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<int8_t*>(planes), dims,
                     strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     kKc == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? MIXER_OK : MIXER_EINVAL;
}

// Dynamic shared memory of a launch: the transpose area only when it holds
// ragged-block tiles (measured: the larger carve-out slows the int64
// epilogue of other launches by up to 5 %).
static int launch_smem(bool ragged) {
    return kSmemBase + (ragged ? kXposeBytes : 0);
}

static int set_smem_attr() {
    static uint64_t attr_set = 0;   // one bit per device ordinal
    int dev = 0;
    MIXER_CK(cudaGetDevice(&dev));
    if (dev < 64 && !(attr_set & (1ull << dev))) {
        MIXER_CK(cudaFuncSetAttribute(k_xcorr_tri, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      kSmemBytes));
        attr_set |= 1ull << dev;
    }
    return MIXER_OK;
}

// Pair kernel set-up, once per device: its shared-memory attribute and how
// many clusters of two CTAs can be resident at once (0: pairs unusable).
static int pair_clusters() {
    static int clusters[64];
    static uint64_t done = 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return 0;
    if (!(done & (1ull << dev))) {
        int n = 0;
        if (cudaFuncSetAttribute(k_xcorr_pair, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kPairSmemBytes) == cudaSuccess) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = 2;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            cfg.gridDim = dim3(2 * 74);
            cfg.blockDim = dim3(kPairThreads);
            cfg.dynamicSmemBytes = kPairSmemBytes;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            if (cudaOccupancyMaxActiveClusters(&n, k_xcorr_pair, &cfg) != cudaSuccess) n = 0;
        }
        cudaGetLastError();   // a refused query leaves no error behind
        clusters[dev] = n;
        done |= 1ull << dev;
    }
    return clusters[dev];
}

// The pair kernel is opt-in (MIXER_XCORR_PAIRS=1 in the environment), from
// three 128-row blocks up (at most one discarded half per channel).  Measured
// on one B200 it is no faster than the one-SM kernel at boost clock and
// slower under the power cap (the clock settles lower: each SM still needs
// all of B, half of it from the peer), so the one-SM kernel is the default.
static bool pairs_wanted(int nblk) {
    if (kKc != 128 || nblk < 3) return false;
    const char* e = getenv("MIXER_XCORR_PAIRS");
    return e && e[0] == '1';
}

static int pair_launch(const CUtensorMap& map, int32_t nant, int32_t nch, int64_t kbeg,
                       int64_t klen, int32_t mode, void* vis, int32_t max_ctas, int32_t* err,
                       int clusters, cudaStream_t st) {
    PairArgs a;
    memset(&a, 0, sizeof(a));
    a.nant = nant;
    a.nch = nch;
    a.nblk = (nant + kTile - 1) / kTile;
    a.ntiles = a.nblk * (a.nblk + 1) / 2;
    a.kbeg = (int32_t)kbeg;
    a.nkc = (int32_t)((klen + kKc - 1) / kKc);
    a.mode = mode;
    a.nreg = a.nblk * a.nblk / 4;
    a.npairs = a.nreg + ((a.nblk + 1) / 2 + 1) / 2;
    a.nwork = (int64_t)nch * a.npairs;
    a.vis = vis;
    a.err = err;
    int64_t ncl = clusters;
    if (max_ctas > 0 && max_ctas / 2 < ncl) ncl = max_ctas / 2;
    if (a.nwork < ncl) ncl = a.nwork;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(2 * ncl));
    cfg.blockDim = dim3(kPairThreads);
    cfg.dynamicSmemBytes = kPairSmemBytes;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    MIXER_CK(cudaLaunchKernelEx(&cfg, k_xcorr_pair, map, a));
    return MIXER_OK;
}

// K ranges of the last round's tiles.  The tiles left over after whole rounds of
// the CTAs, when they are at most half a round, are split over all of them: the
// MMAs get shorter by the parts, for as many more adds (a tile's 256 KB an
// item), which other SMs send side by side.  Stored tiles cannot be split.  One
// B200, whole -> split, int64, 128 elements: 16 channels, K 1024 13.1 -> 10.3
// us, K 8192 45.5 -> 16.0; 164, K 4096 62.1 -> 49.8, K 16384 204 -> 132; 312, K
// 16384 367 -> 247; 64 elements x 16, K 4096 22.3 -> 8.7.  A launch that is all
// last round gains down to two chunks a part (64 x 16, K 1024: 6.6 us, 7.4 with
// four, 9.0 with eight); behind whole rounds, whose adds are still under way,
// the parts have to be longer: in two parts of four chunks 222 channels take
// 36.1 us instead of 34.8, in two of eight 42.1 instead of 44.8.
// The parts serve the launch that has the GPU to itself.  Several small launches
// side by side on streams of one graph take longer in parts, whole -> split:
// eight of 64 x 16, K 4096 27 -> 50 us (one after the other 132 -> 60), four of
// 256 x 16, K 1024 33 -> 49 (60 -> 55).  A CTA limit of as many CTAs as the
// launch has tiles keeps them whole.
constexpr int kPartChunks = 2, kPartChunksBehind = 6;

static void split_last_round(XcorrArgs& a, int64_t tiles, int32_t max_ctas) {
    a.nwhole = a.nwork = tiles;
    a.nsplit = 0;
    a.kpart = a.nkc;
    int64_t ctas = sm_count();
    if (max_ctas > 0 && max_ctas < ctas) ctas = max_ctas;
    const int64_t rest = tiles % ctas;
    if (a.mode == MIXER_VIS_STORE_I32 || rest == 0) return;
    int64_t parts = ctas / rest;
    const int64_t most = a.nkc / (tiles == rest ? kPartChunks : kPartChunksBehind);
    if (parts > most) parts = most;
    if (parts < 2) return;
    a.kpart = (int32_t)((a.nkc + parts - 1) / parts);
    parts = (a.nkc + a.kpart - 1) / a.kpart;
    a.nsplit = (int32_t)rest;
    a.nwhole = tiles - rest;
    a.nwork = a.nwhole + rest * parts;
}

// Grid of a launch, and how its CTAs find their items.  Round robin leaves the
// SMs that reach their memory more slowly behind: at 1024 elements, K 1024,
// where the cube's read-modify-write is the bound, the SMs were busy for 82 %
// of the launch.  Taken over one by one the items even that out.  One B200,
// round robin -> taken over, int64: 1024 x 64, K 1024 256 -> 238 us; 4096 x 8,
// K 1024 457 -> 410 us; 640 x 48 (4.9 items an SM) the same.  Below four items
// an SM there is little to even out, and which SMs get the last round's items
// matters more: 256 x 128 (2.6 an SM), K 1024 55 -> 57 us, so those stay round
// robin.  So do int32 stores, which wait for no memory and gain from CTAs that
// keep in step on a channel's row blocks: taken over -> round robin, 971 x 32, K
// 192 50.1 -> 44.2 us, 640 x 48, K 1024 55 -> 42, 4096 x 8, K 512 142 -> 136, but
// 1024 x 64, K 256 60.8 -> 64.8.  Table launches hold items of different lengths and are always taken
// over; a launch with a CTA limit cannot be, since its grid would be the items.
// A CTA fills its SM's registers either way, so a kernel on another stream
// starts when the launch runs out of items unless the limit leaves it SMs: a
// small flush beside 1024 x 64, K 8192 is done after 830 us, with 144 CTAs
// after 42 (the GEMM 2-5 % slower).
static int64_t launch_grid(XcorrArgs& a, int32_t max_ctas) {
    const int64_t sms = sm_count();
    a.dynamic = max_ctas <= 0 && a.nwork <= INT32_MAX &&
                (a.work ? a.nwork > sms : a.nwork > 4 * sms && a.mode != MIXER_VIS_STORE_I32);
    if (a.dynamic) return a.nwork;
    const int64_t grid = max_ctas > 0 && max_ctas < sms ? max_ctas : sms;
    return a.nwork < grid ? a.nwork : grid;
}

// Launch over samples [kbeg, kbeg + klen) with klen <= MIXER_KMAX_I32.
// At most max_ctas persistent CTAs (<= 0: every SM).
static int xcorr_launch(const int8_t* planes, int32_t nant, int32_t nch, int64_t kt, int64_t kbeg,
                        int64_t klen, int32_t mode, void* vis, int32_t max_ctas, int32_t* err,
                        cudaStream_t st) {
    CUtensorMap maps[2];
    int rc = xcorr_encode_maps(maps, planes, nant, nch, kt, kbeg + klen);
    if (rc != MIXER_OK) return rc;
    if (max_ctas != 1 && pairs_wanted((nant + kTile - 1) / kTile)) {
        const int clusters = pair_clusters();
        if (clusters > 0)
            return pair_launch(maps[0], nant, nch, kbeg, klen, mode, vis, max_ctas, err, clusters, st);
    }
    rc = set_smem_attr();
    if (rc != MIXER_OK) return rc;
    XcorrArgs a;
    a.nant = nant;
    a.ntiles = mixer_vis_tiles(nant);
    a.kbeg = (int32_t)kbeg;
    a.nkc = (int32_t)((klen + kWorkChunk - 1) / kWorkChunk);
    a.mode = mode;
    split_last_round(a, (int64_t)nch * a.ntiles, max_ctas);
    a.vis = vis;
    a.err = err;
    a.tmaps = nullptr;
    a.probs = nullptr;
    a.work = nullptr;
    const int64_t grid = launch_grid(a, max_ctas);
    MIXER_CK(launch_dependent(k_xcorr_tri, dim3((unsigned)grid), dim3(kThreads),
                              launch_smem(nant % kTile != 0), st, maps[0], maps[1], a));
    return MIXER_OK;
}

int xcorr_launch_table(const CUtensorMap* d_tmaps, const XcorrProblem* d_probs,
                       const XcorrWork* d_work, int64_t nwork, int32_t* err, bool ragged,
                       cudaStream_t st) {
    if (nwork <= 0) return MIXER_EINVAL;
    int rc = set_smem_attr();
    if (rc != MIXER_OK) return rc;
    XcorrArgs a;
    memset(&a, 0, sizeof(a));
    a.nwork = nwork;
    a.err = err;
    a.tmaps = d_tmaps;
    a.probs = d_probs;
    a.work = d_work;
    CUtensorMap unused;
    memset(&unused, 0, sizeof(unused));
    const int64_t grid = launch_grid(a, 0);
    MIXER_CK(launch_dependent(k_xcorr_tri, dim3((unsigned)grid), dim3(kThreads),
                              launch_smem(ragged), st, unused, unused, a));
    return MIXER_OK;
}

}  // namespace mixer

extern "C" int32_t mixer_vis_tiles(int32_t nant) {
    if (nant <= 0) return 0;
    const int32_t nb = (nant + 127) / 128;
    return nb * (nb + 1) / 2;
}

extern "C" int64_t mixer_vis_elems(int32_t nant, int32_t nch) {
    if (nant <= 0 || nch <= 0) return 0;
    return (int64_t)nch * mixer_vis_tiles(nant) * 2 * 128 * 128;
}

extern "C" int mixer_xcorr_tri_ex(const int8_t* planes, int32_t nant, int32_t nch, int64_t kt,
                                  int64_t kbeg, int64_t klen, int32_t mode, void* vis,
                                  int32_t max_ctas, int32_t* err, void* stream) {
    if (!planes || !vis || nant <= 0 || nch <= 0 || kt <= 0 || kt % 16 != 0) return MIXER_EINVAL;
    if (kbeg < 0 || kbeg % 16 != 0 || klen <= 0 || kbeg + klen > kt) return MIXER_EINVAL;
    if (mode != MIXER_VIS_STORE_I32 && mode != MIXER_VIS_ACC_I32 && mode != MIXER_VIS_ACC_I64)
        return MIXER_EINVAL;
    if (kt > (int64_t)INT32_MAX || nant > 65536 || nch > 65536) return MIXER_EINVAL;
    if (reinterpret_cast<uintptr_t>(planes) % 16 != 0) return MIXER_EINVAL;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (mode != MIXER_VIS_ACC_I64) {
        if (klen > MIXER_KMAX_I32) return MIXER_EOVERFLOW;
        return mixer::xcorr_launch(planes, nant, nch, kt, kbeg, klen, mode, vis, max_ctas, err, st);
    }
    for (int64_t k = 0; k < klen; k += MIXER_KMAX_I32) {
        const int64_t len = (klen - k) < MIXER_KMAX_I32 ? (klen - k) : MIXER_KMAX_I32;
        const int rc =
            mixer::xcorr_launch(planes, nant, nch, kt, kbeg + k, len, mode, vis, max_ctas, err, st);
        if (rc != MIXER_OK) return rc;
    }
    return MIXER_OK;
}

extern "C" int mixer_mma_peak(int64_t iters, int32_t ctas, int32_t* err, void* stream) {
    if (iters <= 0) return MIXER_EINVAL;
    const int64_t n = ctas > 0 ? ctas : mixer::sm_count();
    constexpr int smem = mixer::kStageBytes + 1024 + 64;
    static uint64_t attr_set = 0;
    int dev = 0;
    MIXER_CK(cudaGetDevice(&dev));
    if (dev < 64 && !(attr_set & (1ull << dev))) {
        MIXER_CK(cudaFuncSetAttribute(mixer::k_mma_peak, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      smem));
        attr_set |= 1ull << dev;
    }
    mixer::k_mma_peak<<<(unsigned)n, 128, smem, static_cast<cudaStream_t>(stream)>>>(iters, err);
    MIXER_CK(cudaGetLastError());
    return MIXER_OK;
}

extern "C" int mixer_xcorr_tri(const int8_t* planes, int32_t nant, int32_t nch, int64_t kt,
                               int64_t kbeg, int64_t klen, int32_t mode, void* vis, int32_t* err,
                               void* stream) {
    return mixer_xcorr_tri_ex(planes, nant, nch, kt, kbeg, klen, mode, vis, 0, err, stream);
}
