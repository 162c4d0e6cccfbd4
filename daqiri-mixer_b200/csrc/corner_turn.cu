// corner_turn.cu -- packets (wire format) -> per-channel int8 planes.
//
// Replaces k_packAB (reference src/rx_host_corr.cu:61-72), which reads one
// byte per thread and writes four planes (A = X and B = conj(X), both
// [ch][ant][k]) one byte at a time.  Here one CTA owns one antenna and `hg`
// consecutive heaps of it (the last group what is left), for a group of nchg
// channels:
//   1. one thread issues 2 x `hg` bulk TMA copies (cp.async.bulk) of the
//      group's re and im bytes of each payload into shared memory (heap stride
//      padded by tpkt bytes so the read-out below is free of bank conflicts);
//   2. all threads write the two planes re / im [C][N][kt] with 16-byte
//      stores, hg*tpkt contiguous bytes (whole cache lines) per (plane,
//      channel) row;
//   3. the first hg threads check each packet's big-endian seq at byte 48
//      against its position (the reference checks only the first packet of a
//      burst, src/rx_host_corr.cu:134).
// HBM-bound: algorithmic bytes = packets read + planes written.
#include "common.cuh"

namespace mixer {
namespace {

__global__ void __launch_bounds__(256)
    k_corner_turn(const uint8_t* pk, int64_t pkt_stride, int hdr, int nant, int nch,
                  int tpkt, int nheaps, int hg, int nchg, uint32_t seq0,
                  int8_t* planes, int64_t kt, int64_t k0, uint32_t* seq_err,
                  int32_t* err) {
    extern __shared__ __align__(128) uint8_t sm[];
    __shared__ __align__(8) uint64_t bar_store;
    const int a = blockIdx.x;
    const int g = blockIdx.y;
    const int c0 = blockIdx.z * nchg;      // first channel of this CTA's group
    const int nh = min(hg, nheaps - g * hg);   // the last groups may be smaller
    const int nc = min(nchg, nch - c0);
    const int half = nch * tpkt;           // bytes per re or im plane of a payload
    const int part = nc * tpkt;            // bytes of one plane staged per heap
    const int hstride = 2 * part + tpkt;   // padded heap stride in shared memory
    const uint32_t bar = smem_u32(&bar_store);

    pdl_wait();
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
        mbar_expect_tx(bar, (uint32_t)(nh * 2 * part));
        for (int hl = 0; hl < nh; ++hl) {
            const int64_t p = (int64_t)(g * hg + hl) * nant + a;
            const uint8_t* src = pk + p * pkt_stride + hdr + (int64_t)c0 * tpkt;
            bulk_g2s(smem_u32(sm + hl * hstride), src, (uint32_t)part, bar);                // re
            bulk_g2s(smem_u32(sm + hl * hstride + part), src + half, (uint32_t)part, bar);  // im
        }
    }
    if (seq_err && blockIdx.z == 0 && threadIdx.x < nh) {
        const int64_t p = (int64_t)(g * hg + threadIdx.x) * nant + a;
        const uint8_t* h = pk + p * pkt_stride + MIXER_WIRE_SEQ_BYTE;
        const uint32_t s = ((uint32_t)h[0] << 24) | ((uint32_t)h[1] << 16) |
                           ((uint32_t)h[2] << 8) | (uint32_t)h[3];
        if (s != seq0 + (uint32_t)p) atomicAdd(seq_err, 1u);
    }
    __syncthreads();   // barrier initialised before anyone polls it
    if (!mbar_wait(bar, 0)) {
        if (err) atomicOr(err, 8);
        mbar_wait(bar, 0);   // second bounded wait for the copies in flight
        return;
    }

    const int V = nh * tpkt / 16;              // 16-byte vectors per (plane, channel) row
    const int64_t kcol = k0 + (int64_t)g * hg * tpkt;
    const int64_t cstride = (int64_t)nant * kt;   // one channel row to the next
    // Each thread keeps one column v of the rows and walks the channel rows of
    // each plane with pointer increments only (no multiply per store); rows
    // wider than the block are walked in slices of its width.
    for (int v0 = 0; v0 < V; v0 += blockDim.x) {
        const int W = min(V - v0, (int)blockDim.x);
        const int rstep = blockDim.x / W;
        const int cl0 = threadIdx.x / W;
        if (cl0 >= rstep) continue;            // blockDim.x is no multiple of W
        const int kb = (v0 + threadIdx.x - cl0 * W) * 16;
        const int hl = kb / tpkt;
        const int64_t dstep = (int64_t)rstep * cstride;
        const int sstep = rstep * tpkt;
#pragma unroll 1
        for (int plane = 0; plane < 2; ++plane) {
            const uint8_t* src = sm + hl * hstride + (kb - hl * tpkt) + plane * part + cl0 * tpkt;
            int8_t* dst = planes + ((int64_t)plane * nch + c0 + cl0) * cstride + (int64_t)a * kt +
                          kcol + kb;
#pragma unroll 4
            for (int cl = cl0; cl < nc; cl += rstep) {
                *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src);
                src += sstep;
                dst += dstep;
            }
        }
    }
}

// Heaps per CTA (hg): output rows of up to kRowBytes contiguous bytes, whole
// cache lines when the packets allow it; the last group takes what is left, so
// that any heap count gets them (a divisor of it would leave 45 heaps, or any
// odd number, with rows of one packet).  Channels per CTA (nchg): equal parts
// of nch whose staging fits the limit, so that several CTAs share an SM and
// one's loads overlap another's stores.  One B200, divisors only -> this form:
// 300 elements x 128 channels, 45 heaps of 32 samples 48.1 -> 35.8 us (4.6 ->
// 6.2 TB/s); 1000 x 41, 21 heaps of 48 samples 50.1 -> 29.6 us; 500 x 127, 17
// heaps 37.9 -> 23.5 us; whole groups (1024 x 256, 512 heaps) unchanged.
// Equal groups instead of whole ones with a remainder measured 0-7 % slower.
constexpr int kRowBytes = 256;
// Staging of a CTA: three on an SM, or four where the grid is short of four
// rounds of those and the last round weighs more.  73 -> 48 KB: 200 x 128, 48
// heaps 27.6 -> 25.6 us, 500 x 127, 17 heaps 27.6 -> 23.5 us, but 1024 x 256,
// 512 heaps 1373 -> 1393 us; 24 KB is 5-9 % slower again.
constexpr int kStageMax = 73 * 1024, kStageShort = 48 * 1024;
constexpr int64_t kShortGrid = 4 * 3 * 148;

int split_channels(int hg, int nch, int tpkt, int limit) {
    int parts = 1;
    while (parts < nch &&
           hg * (2LL * ((nch + parts - 1) / parts) * tpkt + tpkt) > limit)
        ++parts;
    return (nch + parts - 1) / parts;
}

void pick_split(int nant, int nheaps, int nch, int tpkt, int& hg, int& nchg) {
    hg = 1;
    while (hg * tpkt < kRowBytes && hg < nheaps && (hg * 2) * 3 * tpkt <= kStageMax) hg *= 2;
    if (hg > nheaps) hg = nheaps;
    nchg = split_channels(hg, nch, tpkt, kStageMax);
    const int64_t ctas = (int64_t)nant * ((nheaps + hg - 1) / hg) * ((nch + nchg - 1) / nchg);
    if (ctas < kShortGrid) nchg = split_channels(hg, nch, tpkt, kStageShort);
}

}  // namespace
}  // namespace mixer

extern "C" int mixer_corner_turn(const uint8_t* packets, int64_t pkt_stride, int32_t hdr_bytes,
                                 int32_t nant, int32_t nch, int32_t tpkt, int32_t nheaps,
                                 uint32_t seq0, int8_t* planes, int64_t kt, int64_t k0,
                                 uint32_t* seq_errors, int32_t* err, void* stream) {
    if (!packets || !planes || nant <= 0 || nch <= 0 || tpkt <= 0 || nheaps <= 0) return MIXER_EINVAL;
    if (tpkt % 16 != 0 || pkt_stride % 16 != 0 || hdr_bytes % 16 != 0 || kt % 16 != 0 ||
        k0 % 16 != 0 || k0 < 0)
        return MIXER_EINVAL;
    const int64_t P = 2LL * nch * tpkt;
    if (hdr_bytes < MIXER_WIRE_SEQ_BYTE + 4 || hdr_bytes + P > pkt_stride) return MIXER_EINVAL;
    if (P + tpkt > 200 * 1024) return MIXER_EINVAL;
    if (k0 + (int64_t)nheaps * tpkt > kt) return MIXER_EINVAL;
    if (reinterpret_cast<uintptr_t>(packets) % 16 || reinterpret_cast<uintptr_t>(planes) % 16)
        return MIXER_EINVAL;
    int hg, nchg;
    mixer::pick_split(nant, nheaps, nch, tpkt, hg, nchg);
    const int ngroups = (nheaps + hg - 1) / hg;
    // Longest burst: 65535 groups (grid.y) of a power of two that divides it.
    int dg = 1;
    while (dg < hg && nheaps % (dg * 2) == 0) dg *= 2;
    if (nheaps / dg > 65535) return MIXER_EINVAL;
    const size_t smem = (size_t)hg * (size_t)(2 * nchg * tpkt + tpkt);
    if (smem > 48 * 1024)
        MIXER_CK(cudaFuncSetAttribute(mixer::k_corner_turn,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid((unsigned)nant, (unsigned)ngroups, (unsigned)((nch + nchg - 1) / nchg));
    MIXER_CK(mixer::launch_dependent(mixer::k_corner_turn, grid, dim3(256), smem,
                                     static_cast<cudaStream_t>(stream), packets, pkt_stride,
                                     hdr_bytes, nant, nch, tpkt, nheaps, hg, nchg, seq0, planes, kt,
                                     k0, seq_errors, err));
    return MIXER_OK;
}
