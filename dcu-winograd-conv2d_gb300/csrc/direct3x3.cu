// Direct 3x3 convolution as an implicit GEMM on the 5th-generation tensor
// cores, one fused kernel: no Winograd-domain tensor is written.
//
// Pixels are numbered in a flattened, zero-padded space: position
//     z = (n * PH + i) * PW + j      (i, j: padded row and column)
// with PW = W + max(q, 2q - 2) and PH = H + max(p, 2p - 2), so that the zero
// columns right of one row are those left of the next, and the zero rows
// below one image those above the next.  Output (n, oh, ow) sits at
// z = (n * PH + oh) * PW + ow and its tap (r, s) reads position
// z + r * PW + s.  A block of consecutive output positions therefore needs
// one window of consecutive positions, and in the tcgen05 canonical K-major
// layout (16-byte granules of 8 channels, one per position) each tap is the
// same window at another start address: nothing is copied per tap.
//
// Work item: 256 output positions x bn output channels (bn a multiple of 32,
// at most 256), computed by a pair of CTAs (cta_group::2, M = 256): each CTA
// holds the window of its own 128 positions and half of the filter rows.
// Per 16 input channels:
//   * producer warps (three groups of four, chunks round robin) read the
//     window's pixels of 16 channels straight from the caller's tensor --
//     2-byte loads of 8 planes per granule from NCHW, one 16-byte load from
//     channels-last -- and write the granules, zeros where padded;
//   * one TMA box per CTA brings its half of the nine taps' filter rows;
//   * one thread of the even CTA issues nine MMAs.
// Accumulators are double-buffered in TMEM (2 x 256 columns), so the epilogue
// warps store one item while the next is computed.  fp16 or bf16 products are
// exact and summed in fp32; each output is rounded once.
//
// Why a pair and why this tile: per 16 channels an item of 128 positions per
// CTA x 256 channels takes 1,152 cycles of MMAs, and in that time a CTA reads
// 9 x (4 + 4) KB of operands from shared memory (576 cycles at 128 bytes),
// receives 37 KB of filter (288) and writes its window (about 200 with the
// loads): without the pair the filter side doubles and shared memory, not the
// tensor cores, sets the time.  Narrow channel tiles are bound there all the
// same (the window is read nine times for few columns), so they take several
// blocks of 128 positions per item, which share the filter rows and the
// window's halo.  Measured, back to back with rotating buffers, against the
// tuner's choice without this kernel: 32x256x56^2 -> 256 70 us (1,690 TFLOP/s;
// 82 under the power cap) against 102; 32x256x28^2 -> 256 22.8 against 35;
// 32x256x14^2 -> 256 11.6 against 18.7; 16x64x128^2 -> 64 30.7 against 36.6;
// 1x64x56^2 -> 64 5.1 against 9.5; bf16 32x256x28^2 -> 256 22.9 against 52.8;
// channels-last 32x128x56^2 -> 128 26.7 against 42.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <utility>
#include <vector>

#include "wg_kernels.h"
#include "wg_launch.h"
#include "wg_ptx.cuh"

namespace wg {

namespace {

constexpr int kTaps9 = 9;
constexpr int kChunkC = 16;                       // input channels per stage
constexpr int kRows = 128;                        // output positions per CTA
constexpr int kGroups = 3, kGroupWarps = 4;       // producer groups
constexpr int kProdWarps = kGroups * kGroupWarps;
constexpr int kEpiWarps = 4, kEpiHalves = kEpiWarps / 4;
constexpr int kTmaWarp = kProdWarps + kEpiWarps, kMmaWarpD = kTmaWarp + 1;
constexpr int kTables = 2, kTableWarp = kMmaWarpD + 1;   // channels-last: item tables, each filled by a warp of its own
// more warps than 20 would leave fewer than 96 registers per thread
template <bool NHWC>
constexpr int kDirectThreads = 32 * (NHWC ? kTableWarp + kTables : kTableWarp);
constexpr int kMaxRingA = 12, kMaxRingB = 12;
constexpr int kHeader = 512;                      // barriers
constexpr int kMaxSmem = 227 * 1024;
// one CTA per SM (each takes all of TMEM), whatever the rings need
constexpr int kMinSmem = 116 * 1024;

// Element offset (from image n0) of the input pixel at flattened position z,
// or -1 where the position is padding or past the last image.
template <bool NHWC>
__device__ __forceinline__ int pixel_offset(const DirectDesc& d, int z, int n0) {
    const int n = static_cast<int>(fast_div(d.fd_img, static_cast<uint32_t>(z)));
    const int rem = z - n * d.img;
    const int i = static_cast<int>(fast_div(d.fd_pw, static_cast<uint32_t>(rem)));
    const int y = i - d.pad_h, x = rem - i * d.pw - d.pad_w;
    const bool in = n < d.n && static_cast<unsigned>(y) < static_cast<unsigned>(d.h) &&
                    static_cast<unsigned>(x) < static_cast<unsigned>(d.w);
    const int pix = y * d.w + x;
    return in ? (n - n0) * (d.c * d.h * d.w) + (NHWC ? pix * d.c : pix) : -1;
}

__device__ __forceinline__ uint32_t ldg16(const uint16_t* p) {
    uint16_t v;
    asm volatile("ld.global.nc.b16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ldg32(const uint16_t* p) {
    uint32_t v;
    asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void ldg128(const uint16_t* p, uint32_t* v) {
    asm volatile("ld.global.nc.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "l"(p));
}

struct DItem {
    int tile, nb;
};

__device__ __forceinline__ DItem locate_direct(const DirectDesc* __restrict__ descs, int ndesc, int t, int& pi) {
    while (pi + 1 < ndesc && t >= descs[pi + 1].item_begin) ++pi;
    const DirectDesc& d = descs[pi];
    const uint32_t local = static_cast<uint32_t>(t - d.item_begin);
    DItem it;
    it.tile = static_cast<int>(fast_div(d.fd_nb, local));
    it.nb = static_cast<int>(local) - it.tile * d.n_blocks;
    return it;
}

// ---- producers ----------------------------------------------------------------
// A group of four warps writes the windows of every kGroups-th chunk (NHWC:
// pair of chunks).  Its work is a sequence of steps (item, chunk, block of
// positions), each 16 registers of loads per thread; a step's loads are issued
// before the step ahead of it is stored, so one load latency covers two steps
// whether or not a stage is free.  Per block and thread:
//   pairs   two neighbouring pixels of 16 planes (4-byte loads; W even, x
//           4-byte aligned), 128 pairs; the padding of the window is cleared
//           by the threads whose positions it is
//   single  one position of 16 planes (2-byte loads), 128 positions
//   NHWC    four positions of one of the pair's four granules (16-byte loads),
//           128 positions: a pixel's 64 bytes are half a line, one chunk's 32
//           would make twice the requests to L2
constexpr int kGroupThreads = 32 * kGroupWarps;
constexpr int kMaxPadBits = 32;      // pairs: positions per thread the pad mask covers

// Channels-last: where the pixels of an item's window lie in the input, worked
// out once per item by warps that do nothing else (items take the two tables in
// turn; all warps share the first item).  Worked out by the threads of each
// producer group, and kept in 12 of their registers, it stood in the way of
// their loads: 32x256x56^2 -> 256 75.4 -> 69.9 us, 32x128x56^2 -> 128 28.0 -> 26.7,
// 32x256x14^2 -> 256 12.3 -> 11.2.  (NCHW gains nothing, 16x64x128^2 -> 64 30.6 ->
// 30.4 and 32x256x28^2 -> 256 23.1 -> 24.2: a table of pixel pairs and padding takes
// a warp three times as long.)
struct ItemTable {
    const uint16_t* xi;   // image of the window's first position
    int chunks, win, channels;
    // then the element offset of each position from xi, or -1; whole blocks of 128
};
__host__ __device__ __forceinline__ int table_bytes(int win) {
    return static_cast<int>(sizeof(ItemTable)) + 4 * ((win + 127) / 128 * 128);
}
// longest window that a stage of a_bytes holds
__host__ __device__ __forceinline__ int max_window(int a_bytes) { return a_bytes / 32; }

// by `threads` threads
__device__ __forceinline__ void build_table(const DirectDesc& d, const DItem& it, uint32_t rank, ItemTable* tab, int tid,
                                            int threads) {
    const int z0 = d.pos0 + (2 * it.tile + static_cast<int>(rank)) * d.cta_rows;
    const int n0 = min(static_cast<int>(fast_div(d.fd_img, static_cast<uint32_t>(z0))), d.n - 1), win = d.win;
    if (tid == 0) {
        tab->xi = static_cast<const uint16_t*>(d.x) + static_cast<long long>(n0) * d.c * d.h * d.w;
        tab->chunks = d.c_chunks;
        tab->win = win;
        tab->channels = d.c;
    }
    for (int p = tid; p < (win + 127) / 128 * 128; p += threads) reinterpret_cast<int*>(tab + 1)[p] = p < win ? pixel_offset<true>(d, z0 + p, n0) : -1;
}

struct Step {
    uint32_t r[16];
    int p;             // pairs, single: position of the first granule; NHWC: of the block's first
    uint32_t pads;     // pairs: bit i set where position gt + 128 i is padding (last block of a chunk only);
                       // NHWC: the first of the two chunks, counted over the CTA's items
    uint32_t flags;    // bit 0: first block of the chunk, 1: last, 2: pairs (NHWC: there is a second
                       // chunk), 4..7: zero the granule (single: 4); the window's length above bit 16
};

// Bytes of one granule's window in shared memory: 4 mod 8 positions, so that
// the two granules of a channels-last pixel fall in different bank groups.
__host__ __device__ __forceinline__ int granule_bytes(int win) { return ((win + 7) / 8 * 8 + 4) * 16; }

template <bool NHWC>
struct Producer {
    const DirectDesc* __restrict__ descs;
    int ndesc, total_items, step, grp, gt;
    uint32_t rank;
    // load cursor; NHWC: c counts pairs of chunks (gu0: those of earlier items)
    int t, pi, c, chunks, gc0, blk, blocks, gu0;
    int z0, n0, win, channels;
    int pairs;
    uint32_t plane;
    const uint16_t* xi;
    // the item's first blocks: element offset from xi (-1: nothing to load) and position
    static constexpr int kKeep = 4;
    int off[kKeep];
    uint32_t pos2[2];   // positions of blocks 0, 1 and 2, 3 as 16-bit halves (-1 as 0xffff)
    uint32_t pads;
    // NHWC: the tables, the item of this CTA and its table
    unsigned char* tables;
    int table_size, k;
    const int* table;
    uint64_t *tabfull, *tabempty;
    volatile int* abort_flag;
    DevErr* err;
    bool failed;

    // pairs: pair number gt + 128 i of the window, decoded from scratch (blocks past kKeep)
    __device__ __forceinline__ void locate_pair(const DirectDesc& d, int i, int& o, int& p) const {
        const int g = d_first(d) + 2 * (gt + kGroupThreads * i);
        const int hw = d.h * d.w, n = static_cast<int>(fast_div(d.fd_hw, static_cast<uint32_t>(g))), m = g - n * hw;
        const int y = static_cast<int>(fast_div(d.fd_w, static_cast<uint32_t>(m)));
        p = n * d.img + (y + d.pad_h) * d.pw + (m - y * d.w) + d.pad_w - z0;
        o = n < d.n && p < win ? (n - n0) * (d.c * hw) + m : -1;
        if (o < 0) p = win;
    }
    // index (over all images, in memory order of one channel) of the first
    // pixel pair that reaches into the window
    __device__ __forceinline__ int d_first(const DirectDesc& d) const {
        const int n = static_cast<int>(fast_div(d.fd_img, static_cast<uint32_t>(z0)));
        const int rem = z0 - n * d.img;
        const int i = static_cast<int>(fast_div(d.fd_pw, static_cast<uint32_t>(rem)));
        const int y = i - d.pad_h, x = rem - i * d.pw - d.pad_w;
        const int m = y < 0 ? 0 : min(y, d.h) * d.w + (y < d.h ? min(max(x, 0), d.w) : 0);
        return (n * (d.h * d.w) + m) & ~1;
    }

    __device__ __forceinline__ void decode(const DirectDesc& d) {
        if (pairs) {
            // pairs 128 apart: a step of qy rows and rx columns
            const int hw = d.h * d.w, w = d.w, h = d.h, chw = d.c * hw;
            const int g = d_first(d) + 2 * gt;
            int n = static_cast<int>(fast_div(d.fd_hw, static_cast<uint32_t>(g)));
            const int m = g - n * hw;
            int y = static_cast<int>(fast_div(d.fd_w, static_cast<uint32_t>(m))), x = m - y * w;
#pragma unroll
            for (int i = 0; i < kKeep; ++i) {
                const int p = n * d.img + (y + d.pad_h) * d.pw + x + d.pad_w - z0;
                const bool in = n < d.n && p < win;
                off[i] = in ? (n - n0) * chw + y * w + x : -1;
                const uint32_t q = static_cast<uint32_t>(in ? p : win) & 0xffffu;
                pos2[i / 2] = (i & 1) ? pos2[i / 2] | (q << 16) : q;
                x += d.step_x;
                y += d.step_y;
                if (x >= w) x -= w, ++y;
                while (y >= h && n < d.n) y -= h, ++n;
            }
            // positions 128 apart: the window's padding among this thread's
            int zn = static_cast<int>(fast_div(d.fd_img, static_cast<uint32_t>(z0 + gt)));
            const int rem = z0 + gt - zn * d.img;
            int zi = static_cast<int>(fast_div(d.fd_pw, static_cast<uint32_t>(rem))), zj = rem - zi * d.pw;
            pads = 0;
            for (int i = 0, p = gt; p < win; ++i, p += kGroupThreads) {
                const bool in = zn < d.n && static_cast<unsigned>(zi - d.pad_h) < static_cast<unsigned>(h) &&
                                static_cast<unsigned>(zj - d.pad_w) < static_cast<unsigned>(w);
                pads |= (in ? 0u : 1u) << i;
                zj += d.pad_step_j;
                zi += d.pad_step_i;
                if (zj >= d.pw) zj -= d.pw, ++zi;
                while (zi >= d.ph) zi -= d.ph, ++zn;
            }
        } else {
#pragma unroll
            for (int i = 0; i < kKeep; ++i) {
                const uint32_t q = static_cast<uint32_t>(gt + kGroupThreads * i);
                pos2[i / 2] = (i & 1) ? pos2[i / 2] | (q << 16) : q;
                off[i] = pixel_offset<false>(d, z0 + static_cast<int>(q), n0);
            }
        }
    }

    // the current item's chunks, or pairs of them
    __device__ __forceinline__ int units() const { return NHWC ? (chunks + 1) / 2 : chunks; }

    // moves to the group's next step of the item; false when there is none
    __device__ __forceinline__ bool advance() {
        if (++blk < blocks) return true;
        blk = 0;
        c += kGroups;
        return c < units();
    }

    // moves to the first step in the items that follow; false when there is none
    __device__ __forceinline__ bool next_item() {
        while (c >= units()) {
            if (NHWC && k >= 0) {   // its table is read
                __syncwarp();
                if ((gt & 31) == 0) mbar_arrive(&tabempty[k % kTables]);
            }
            gu0 += units();
            gc0 += chunks;
            chunks = 0;
            t += step;
            if (t >= total_items) return false;
            if constexpr (NHWC) {
                ++k;
                if (!mbar_wait(&tabfull[k % kTables], (k / kTables) & 1, abort_flag, err, ERR_SITE_FULL)) {
                    failed = true;
                    return false;
                }
                const ItemTable& tab = *reinterpret_cast<const ItemTable*>(tables + (k % kTables) * table_size);
                chunks = tab.chunks;
                c = (grp - gu0 % kGroups + kGroups) % kGroups;
                table = reinterpret_cast<const int*>(&tab + 1);
                xi = tab.xi;
                win = tab.win;
                channels = tab.channels;
                blocks = (win + 127) / 128;
                continue;
            }
            const DItem it = locate_direct(descs, ndesc, t, pi);
            const DirectDesc& d = descs[pi];
            chunks = d.c_chunks;
            c = (grp - gc0 % kGroups + kGroups) % kGroups;
            if (c >= units()) continue;
            z0 = d.pos0 + (2 * it.tile + static_cast<int>(rank)) * d.cta_rows;
            n0 = min(static_cast<int>(fast_div(d.fd_img, static_cast<uint32_t>(z0))), d.n - 1);
            win = d.win;
            channels = d.c;
            pairs = d.pairs;
            plane = static_cast<uint32_t>(d.h * d.w);
            xi = static_cast<const uint16_t*>(d.x) + static_cast<long long>(n0) * channels * plane;
            // blocks that reach into the window, for this warp's part of them
            blocks = max(((pairs ? win / 2 + 1 : win) - (gt & ~31) + kGroupThreads - 1) / kGroupThreads, 1);
            pads = 0;
            decode(d);
        }
        return true;
    }

    __device__ __forceinline__ void load(Step& s) {
        s.flags = (static_cast<uint32_t>(win) << 16) | (blk == 0 ? 1u : 0u) | (blk == blocks - 1 ? 2u : 0u);
        if constexpr (NHWC) {
            const int ch = c * 2 * kChunkC + 8 * (gt & 3);
            const bool cin = ch < channels;
            if (2 * c + 1 < chunks) s.flags |= 4u;
            s.pads = static_cast<uint32_t>(gc0 + 2 * c);
            s.p = blk * 128 + (gt >> 2);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                int o = table[s.p + 32 * k];
                if (o < 0 || !cin) {
                    o = 0;
                    s.flags |= 16u << k;
                }
                ldg128(xi + o + (cin ? ch : 0), s.r + 4 * k);
            }
            return;
        }
        if (pairs) s.flags |= 4u;
        s.pads = blk == blocks - 1 ? pads : 0u;
        const int left = channels - c * kChunkC;   // channels from this chunk on
        int o = off[0];
        o = blk == 1 ? off[1] : o;
        o = blk == 2 ? off[2] : o;
        o = blk == 3 ? off[3] : o;
        const uint32_t pq = blk < 2 ? pos2[0] : pos2[1];
        int p = static_cast<int16_t>((blk & 1) ? pq >> 16 : pq);
        if (blk >= kKeep) {
            if (pairs) {
                locate_pair(descs[pi], blk, o, p);
            } else {
                p = gt + kGroupThreads * blk;
                o = pixel_offset<false>(descs[pi], z0 + p, n0);
            }
        }
        s.p = p;
        if (o < 0) s.flags |= 16u;
        // padding reads the image's first pixel (cleared or not stored later)
        const uint16_t* src = xi + max(o, 0) + static_cast<unsigned long long>(c * kChunkC) * plane;
        if (left >= kChunkC) {
            if (pairs) {
#pragma unroll
                for (int j = 0; j < kChunkC; ++j) s.r[j] = ldg32(src + static_cast<unsigned long long>(j) * plane);
            } else {
#pragma unroll
                for (int j = 0; j < kChunkC; ++j) s.r[j] = ldg16(src + static_cast<unsigned long long>(j) * plane);
            }
        } else {
            // the last chunk of a C that is not a multiple of 16
#pragma unroll
            for (int j = 0; j < kChunkC; ++j) {
                const uint16_t* q = src + static_cast<unsigned long long>(min(j, left - 1)) * plane;
                const uint32_t v = pairs ? ldg32(q) : ldg16(q);
                s.r[j] = j < left ? v : 0u;
            }
        }
    }

    // writes a loaded step's granules into the window stage at A
    __device__ __forceinline__ void store(const Step& s, unsigned char* A) const {
        const int s_win = static_cast<int>(s.flags >> 16), s_gran = granule_bytes(s_win);
        if (s.flags & 4u) {
            // lanes 4-7 of every 8 store their second pixel first: the 8 lanes
            // of a store phase then write 8 different 16-byte bank groups
            const uint32_t sel0 = (gt & 4) ? 0x7632u : 0x5410u, sel1 = sel0 ^ 0x2222u;
            const int p0 = s.p + ((gt >> 2) & 1), p1 = s.p + 1 - ((gt >> 2) & 1);
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                const uint32_t* r = s.r + 8 * g;
                unsigned char* dst = A + g * s_gran;
                if (static_cast<unsigned>(p0) < static_cast<unsigned>(s_win))
                    *reinterpret_cast<uint4*>(dst + p0 * 16) =
                        make_uint4(__byte_perm(r[0], r[1], sel0), __byte_perm(r[2], r[3], sel0),
                                   __byte_perm(r[4], r[5], sel0), __byte_perm(r[6], r[7], sel0));
                if (static_cast<unsigned>(p1) < static_cast<unsigned>(s_win) && s.p < s_win)
                    *reinterpret_cast<uint4*>(dst + p1 * 16) =
                        make_uint4(__byte_perm(r[0], r[1], sel1), __byte_perm(r[2], r[3], sel1),
                                   __byte_perm(r[4], r[5], sel1), __byte_perm(r[6], r[7], sel1));
            }
            for (uint32_t m = s.pads; m; m &= m - 1) {
                unsigned char* dst = A + (gt + kGroupThreads * (__ffs(m) - 1)) * 16;
                *reinterpret_cast<uint4*>(dst) = make_uint4(0u, 0u, 0u, 0u);
                *reinterpret_cast<uint4*>(dst + s_gran) = make_uint4(0u, 0u, 0u, 0u);
            }
        } else {
            const bool z = (s.flags & 16u) != 0;
            if (s.p < s_win)
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    const uint32_t* r = s.r + 8 * g;
                    *reinterpret_cast<uint4*>(A + g * s_gran + s.p * 16) =
                        z ? make_uint4(0u, 0u, 0u, 0u)
                          : make_uint4(__byte_perm(r[0], r[1], 0x5410), __byte_perm(r[2], r[3], 0x5410),
                                       __byte_perm(r[4], r[5], 0x5410), __byte_perm(r[6], r[7], 0x5410));
                }
        }
    }
};

template <bool BF16>
__device__ __forceinline__ uint32_t pack2(uint32_t a, uint32_t b) {
    if constexpr (BF16) {
        __nv_bfloat162 v = __floats2bfloat162_rn(__uint_as_float(a), __uint_as_float(b));
        return *reinterpret_cast<uint32_t*>(&v);
    } else {
        __half2 v = __floats2half2_rn(__uint_as_float(a), __uint_as_float(b));
        return *reinterpret_cast<uint32_t*>(&v);
    }
}

// NHWC: stores a loaded step once its two stages (st, st2) are free, and hands
// them over after its last block.
__device__ __forceinline__ bool flush_step2(const Producer<true>& pr, const Step& s, unsigned char* astage, int a_bytes,
                                            int na, int& st, int& st2, uint64_t* afull, uint64_t* aempty,
                                            volatile int* abort_flag, DevErr* err) {
    const bool two = (s.flags & 4u) != 0;
    if (s.flags & 1u) {
        const int use = static_cast<int>(s.pads) / na;
        st = static_cast<int>(s.pads) - use * na;
        st2 = st + 1 == na ? 0 : st + 1;
        const uint32_t ph = (use & 1) ^ 1, ph2 = st2 == 0 ? ph ^ 1u : ph;
        if (!mbar_wait(&aempty[st], ph, abort_flag, err, ERR_SITE_EMPTY)) return false;
        if (two && !mbar_wait(&aempty[st2], ph2, abort_flag, err, ERR_SITE_EMPTY)) return false;
    }
    const int win = static_cast<int>(s.flags >> 16), sub = pr.gt & 3;
    unsigned char* dst = astage + (sub < 2 ? st : st2) * a_bytes + (sub & 1) * granule_bytes(win);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int p = s.p + 32 * k;
        const bool z = (s.flags >> (4 + k)) & 1u;
        if (p < win && (two || sub < 2))
            *reinterpret_cast<uint4*>(dst + p * 16) =
                make_uint4(z ? 0u : s.r[4 * k], z ? 0u : s.r[4 * k + 1], z ? 0u : s.r[4 * k + 2], z ? 0u : s.r[4 * k + 3]);
    }
    if (s.flags & 2u) {
        fence_proxy_async_smem();     // the windows are read by the tensor core
        __syncwarp();
        if ((pr.gt & 31) == 0) {
            mbar_arrive_cluster(map_to_rank(&afull[st], 0));
            if (two) mbar_arrive_cluster(map_to_rank(&afull[st2], 0));
        }
    }
    return true;
}

// Stores a loaded step once its stage is free; after a chunk's last block
// hands the stage to the MMAs and moves to the group's next one.
__device__ __forceinline__ bool flush_step(const Producer<false>& pr, const Step& s, unsigned char* astage, int a_bytes,
                                           int na, int& sa, uint32_t& ph, uint64_t* afull, uint64_t* aempty,
                                           volatile int* abort_flag, DevErr* err) {
    if ((s.flags & 1u) && !mbar_wait(&aempty[sa], ph, abort_flag, err, ERR_SITE_EMPTY)) return false;
    pr.store(s, astage + sa * a_bytes);
    if (s.flags & 2u) {
        fence_proxy_async_smem();     // the window is read by the tensor core
        __syncwarp();
        if ((pr.gt & 31) == 0) mbar_arrive_cluster(map_to_rank(&afull[sa], 0));
        sa += kGroups;
        while (sa >= na) sa -= na, ph ^= 1u;
    }
    return true;
}

// LATE: the kernel ahead on the stream is waited for only where its data is
// first touched, so that the set-up (barriers, TMEM, the first item's decoding)
// overlaps its end.  Not with descriptors in global memory, which that kernel
// or copy may have written.
template <bool NHWC, bool BF16, bool LATE>
__device__ __forceinline__ void direct_body(const DirectDesc* __restrict__ descs, int ndesc, int total_items,
                                            const DirectRing& ring, DevErr* err) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    unsigned char* bstage = smem;                              // filter ring
    unsigned char* astage = smem + ring.nb * ring.b_bytes;     // window ring
    uint64_t* bars = reinterpret_cast<uint64_t*>(astage + ring.na * ring.a_bytes);
    uint64_t* afull = bars;                        // even CTA: windows of both CTAs written
    uint64_t* aempty = afull + kMaxRingA;          // MMAs done with the window
    uint64_t* bfull = aempty + kMaxRingA;          // even CTA: filter halves of both CTAs landed
    uint64_t* bempty = bfull + kMaxRingB;          // MMAs done with the filter rows
    uint64_t* tfull = bempty + kMaxRingB;          // [2] accumulator ready
    uint64_t* tempty = tfull + 2;                  // [2] even CTA: accumulator drained in both CTAs
    uint64_t* tabfull = tempty + 2;                // item table written
    uint64_t* tabempty = tabfull + kTables;        // read by every producer warp
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tabempty + kTables);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int first = blockIdx.x >> 1, step = gridDim.x >> 1;
    const int na = ring.na, nb = ring.nb;
    unsigned char* tables = reinterpret_cast<unsigned char*>(bars) + kHeader;
    const int table_size = table_bytes(max_window(ring.a_bytes));

    if (threadIdx.x == 0) {
        for (int i = 0; i < kMaxRingA; ++i) {
            mbar_init(&afull[i], 2 * kGroupWarps);
            mbar_init(&aempty[i], 1);
        }
        for (int i = 0; i < kMaxRingB; ++i) {
            mbar_init(&bfull[i], 1);
            mbar_init(&bempty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&tfull[i], 1);
            mbar_init(&tempty[i], 2 * kEpiWarps);
        }
        for (int i = 0; i < kTables; ++i) {
            mbar_init(&tabfull[i], 1);
            mbar_init(&tabempty[i], kProdWarps);
        }
        *abort_flag = 0;
        fence_barrier_init();
    }
    if constexpr (!LATE) pdl_wait();
    if (warp == kMmaWarpD) tmem_alloc_pair(tmem_slot, 512);
    if (NHWC && first < total_items) {
        int pi = 0;
        const DItem it = locate_direct(descs, ndesc, first, pi);
        build_table(descs[pi], it, rank, reinterpret_cast<ItemTable*>(tables), static_cast<int>(threadIdx.x),
                    kDirectThreads<NHWC>);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // input and filter written, earlier readers of the output done
    auto start = [&] {
        if constexpr (LATE) pdl_wait();
        pdl_trigger();
    };

    if (warp < kProdWarps) {
        Producer<NHWC> pr;
        pr.descs = descs;
        pr.ndesc = ndesc;
        pr.total_items = total_items;
        pr.step = step;
        pr.grp = warp / kGroupWarps;
        pr.gt = static_cast<int>(threadIdx.x) - pr.grp * kGroupThreads;
        pr.rank = rank;
        pr.tables = tables;
        pr.table_size = table_size;
        pr.k = -1;
        pr.tabfull = tabfull;
        pr.tabempty = tabempty;
        pr.abort_flag = abort_flag;
        pr.err = err;
        pr.failed = false;
        pr.t = first - step;
        pr.pi = pr.c = pr.chunks = pr.gc0 = pr.gu0 = pr.blk = pr.blocks = 0;
        int sa = pr.grp;             // this group's next window stage and its phase
        uint32_t ph = 1;
        while (sa >= na) sa -= na, ph ^= 1u;
        int st = 0, st2 = 0;
        auto flush = [&](const Step& s) {
            if constexpr (NHWC)
                return flush_step2(pr, s, astage, ring.a_bytes, na, st, st2, afull, aempty, abort_flag, err);
            else
                return flush_step(pr, s, astage, ring.a_bytes, na, sa, ph, afull, aempty, abort_flag, err);
        };
        // Steps alternate between s0 and s1.
        bool ok = true, more = pr.next_item();
        start();
        Step s0, s1;
        if constexpr (NHWC) {
            auto next = [&] { return pr.advance() || pr.next_item(); };
            if (more) pr.load(s0);
            while (more) {
                more = next();
                if (more) pr.load(s1);
                ok = flush(s0);
                if (!ok || !more) break;
                more = next();
                if (more) pr.load(s0);
                ok = flush(s1);
                if (!ok) break;
            }
        } else {
            // moving to another item is one copy of code for both: the warps of
            // an SM share a small instruction cache, and the NCHW loads and
            // packing alone fill it (32x128x56^2 -> 128 28.5 -> 26.5 us;
            // channels-last, with a quarter of that code, gains nothing)
            bool first_step = true, boundary = false;
            for (int odd = 0;;) {
                if (boundary) more = pr.next_item();
                if (odd == 0) {
                    if (more) pr.load(s0);
                    if (!first_step) ok = flush(s1);
                    if (!ok || !more) break;
                    first_step = false;
                    odd = 1;
                    if ((boundary = !pr.advance())) continue;
                }
                if (more) pr.load(s1);
                ok = flush(s0);
                if (!ok || !more) break;
                odd = 0;
                boundary = !pr.advance();
            }
        }
        // the last commits on this CTA's window barriers must land before it exits
        if (ok && !pr.failed && warp == 0 && lane == 0)
            for (int k = max(0, pr.gc0 - na); k < pr.gc0; ++k)
                if (!mbar_wait(&aempty[k % na], (k / na) & 1, abort_flag, err, ERR_SITE_DRAIN)) break;
    } else if (warp == kTmaWarp) {
        // ---- filter halves: one box per chunk, counted on the even CTA's barrier
        start();
        if (lane == 0) {
            int gc = 0, pi = 0, prefetched = -1;
            bool ok = true;
            for (int t = first; t < total_items && ok; t += step) {
                const DItem it = locate_direct(descs, ndesc, t, pi);
                const DirectDesc& d = descs[pi];
                if (prefetched != pi) {
                    tma_prefetch_desc(&d.tmU);
                    prefetched = pi;
                }
                const uint32_t bytes = static_cast<uint32_t>(kTaps9 * 2 * (d.bn / 2) * 16);
                const int row = (it.nb * d.bn + static_cast<int>(rank) * (d.bn / 2)) / 8;
                const int chunks = d.c_chunks;
                for (int c = 0; c < chunks; ++c, ++gc) {
                    const int sb = gc % nb;
                    if (!mbar_wait(&bempty[sb], ((gc / nb) & 1) ^ 1, abort_flag, err, ERR_SITE_EMPTY)) {
                        ok = false;
                        break;
                    }
                    if (rank == 0) mbar_arrive_expect_tx(&bfull[sb], 2 * bytes);
                    tma_load_4d_pair(bstage + sb * ring.b_bytes, &d.tmU, map_to_rank(&bfull[sb], 0), 0, row, c * 2, 0);
                }
            }
            if (ok)
                for (int k = max(0, gc - nb); k < gc; ++k)
                    if (!mbar_wait(&bempty[k % nb], (k / nb) & 1, abort_flag, err, ERR_SITE_DRAIN)) break;
        }
    } else if (warp == kMmaWarpD) {
        // ---- MMAs of the pair, issued by one elected thread of the even CTA.
        //      The whole warp walks the loop with warp-uniform control flow and
        //      values, so descriptors stay in uniform registers: with one lane
        //      in the loop every MMA first moved its operands there
        start();
        if (rank == 0) {
            int pi = 0, k = 0, sa = 0, sb = 0;
            uint32_t aph = 0, bph = 0;
            const int a_step = ring.a_bytes / 16, b_step = ring.b_bytes / 16;
            const uint64_t a_lo = make_smem_desc(smem_u32(astage), 0, 128, Swz::None);
            const uint64_t b_lo = make_smem_desc(smem_u32(bstage), 0, 128, Swz::None);
            const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
            const bool elected = elect_one();
            bool ok = true;
            for (int t = first; t < total_items && ok; t += step, ++k) {
                locate_direct(descs, ndesc, t, pi);
                const DirectDesc& d = descs[pi];
                const int acc = k & 1;
                if (!mbar_wait_warp(&tempty[acc], ((k >> 1) & 1) ^ 1, abort_flag, err, ERR_SITE_TMEM_EMPTY)) break;
                tc_fence_after();
                const uint32_t idesc = make_idesc_f16(2 * kRows, d.bn, BF16);
                const uint32_t d_tmem = tmem_u + static_cast<uint32_t>(acc * 256);
                // descriptors of stage 0, tap 0; stages and taps only move the
                // start address (the low 14 bits, in 16-byte units)
                const int chunks = d.c_chunks, bn = d.bn, pw = d.pw, mb = d.mb;
                const uint64_t ad0 = a_lo | (static_cast<uint64_t>(d.gran >> 4) << 16);
                const uint64_t bd0 = b_lo | (static_cast<uint64_t>(bn >> 1) << 16);
                for (int c = 0; c < chunks; ++c) {
                    if (!mbar_wait_warp(&bfull[sb], bph, abort_flag, err, ERR_SITE_FULL) ||
                        !mbar_wait_warp(&afull[sa], aph, abort_flag, err, ERR_SITE_FULL)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t as = ad0 + static_cast<uint32_t>(sa * a_step);
                    const uint64_t bs = bd0 + static_cast<uint32_t>(sb * b_step);
                    if (elected) {
                        for (int m = 0; m < mb; ++m) {
                            const uint64_t am = as + static_cast<uint32_t>(m * kRows);
#pragma unroll
                            for (int tap = 0; tap < kTaps9; ++tap)
                                tc_mma_f16_pair(d_tmem + static_cast<uint32_t>(m * bn),
                                                am + static_cast<uint32_t>((tap / 3) * pw + tap % 3),
                                                bs + static_cast<uint32_t>(tap * bn), idesc, (c | tap) != 0 ? 1u : 0u);
                        }
                        tc_commit_pair(&aempty[sa]);
                        tc_commit_pair(&bempty[sb]);
                    }
                    __syncwarp();
                    if (++sa == na) sa = 0, aph ^= 1u;
                    if (++sb == nb) sb = 0, bph ^= 1u;
                }
                if (ok && elected) tc_commit_pair(&tfull[acc]);
                __syncwarp();
            }
        }
    } else if (NHWC && warp >= kTableWarp) {
        // ---- item tables; the first is written
        int pi = 0, k = warp - kTableWarp;
        if (k == 0) {
            if (lane == 0) mbar_arrive(&tabfull[0]);
            k = kTables;
        }
        // nothing here needs the kernel ahead, but the bounded waits below end only
        // after the producers, who do, have read a table: its remaining time must
        // not count against them
        start();
        for (int t = first + k * step; t < total_items; t += kTables * step, k += kTables) {
            const DItem it = locate_direct(descs, ndesc, t, pi);
            if (!mbar_wait_warp(&tabempty[k % kTables], ((k / kTables) & 1) ^ 1, abort_flag, err, ERR_SITE_EMPTY)) break;
            build_table(descs[pi], it, rank, reinterpret_cast<ItemTable*>(tables + (k % kTables) * table_size), lane, 32);
            __syncwarp();
            if (lane == 0) mbar_arrive(&tabfull[k % kTables]);
        }
    } else {
        // ---- epilogue: kEpiHalves warps per TMEM lane quarter, taking blocks
        //      of 16 columns in turn
        start();
        const int quarter = warp & 3, half = (warp - kProdWarps) >> 2;
        int pi = 0, k = 0;
        for (int t = first; t < total_items; t += step, ++k) {
            const DItem it = locate_direct(descs, ndesc, t, pi);
            const DirectDesc& d = descs[pi];
            const int acc = k & 1;
            if (!mbar_wait(&tfull[acc], (k >> 1) & 1, abort_flag, err, ERR_SITE_TMEM_FULL)) break;
            __syncwarp();
            tc_fence_after();
            uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(acc * 256 + half * 16);
            const int K = d.k, bn = d.bn, mb = d.mb, ow_n = d.ow;
            const int oplane = d.oh * ow_n;
            const bool vec = d.vec != 0;
            const int zb = d.pos0 + (2 * it.tile + static_cast<int>(rank)) * d.cta_rows + quarter * 32 + lane;
            for (int m = 0; m < mb; ++m) {
                const int z = zb + m * kRows;
                const int n = static_cast<int>(fast_div(d.fd_img, static_cast<uint32_t>(z)));
                const int rem = z - n * d.img;
                const int oh = static_cast<int>(fast_div(d.fd_pw, static_cast<uint32_t>(rem)));
                const int ow = rem - oh * d.pw;
                const bool valid = n < d.n && oh < d.oh && ow < ow_n;
                const int opix = oh * ow_n + ow;
                int k0 = it.nb * bn + half * 16;
                uint16_t* o = static_cast<uint16_t*>(d.y);
                if constexpr (NHWC)
                    o += (static_cast<long long>(n) * oplane + opix) * K + k0;
                else
                    o += (static_cast<long long>(n) * K + k0) * oplane + opix;
                for (int b = half; b < bn / 16; b += kEpiHalves, k0 += 16 * kEpiHalves, taddr += 16 * kEpiHalves) {
                    uint32_t r[16];
                    tmem_ld_x16(taddr, r);
                    tc_wait_ld16(r);
                    if (m == mb - 1 && b + kEpiHalves >= bn / 16) {   // this warp's last read of the accumulators
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_cluster(map_to_rank(&tempty[acc], 0));
                    }
                    if (valid) {
                        if constexpr (NHWC) {
                            if (vec && k0 + 16 <= K) {
#pragma unroll
                                for (int j = 0; j < 2; ++j)
                                    reinterpret_cast<uint4*>(o)[j] = make_uint4(
                                        pack2<BF16>(r[8 * j], r[8 * j + 1]), pack2<BF16>(r[8 * j + 2], r[8 * j + 3]),
                                        pack2<BF16>(r[8 * j + 4], r[8 * j + 5]), pack2<BF16>(r[8 * j + 6], r[8 * j + 7]));
                            } else {
#pragma unroll
                                for (int j = 0; j < 16; ++j)
                                    if (k0 + j < K) o[j] = static_cast<uint16_t>(pack2<BF16>(r[j], 0u));
                            }
                        } else {
                            // a warp's 32 positions of one channel are (nearly) contiguous
                            const uint32_t op = static_cast<uint32_t>(oplane);
                            if (k0 + 16 <= K) {
#pragma unroll
                                for (int j = 0; j < 16; j += 2) {
                                    const uint32_t v = pack2<BF16>(r[j], r[j + 1]);
                                    o[static_cast<unsigned long long>(j) * op] = static_cast<uint16_t>(v);
                                    o[static_cast<unsigned long long>(j + 1) * op] = static_cast<uint16_t>(v >> 16);
                                }
                            } else {
#pragma unroll
                                for (int j = 0; j < 16; ++j) {
                                    if (k0 + j < K)
                                        o[static_cast<unsigned long long>(j) * op] = static_cast<uint16_t>(pack2<BF16>(r[j], 0u));
                                }
                            }
                        }
                    }
                    o += NHWC ? 16LL * kEpiHalves : 16LL * kEpiHalves * oplane;
                    __syncwarp();
                }
                // (bn / 16 is even: every warp of a quarter takes as many blocks)
            }
        }
    }

    __syncthreads();
    if (*abort_flag) {
        // let any copy or MMA still in flight land before the pair retires
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) {
        }
    }
    tc_fence_before();
    cluster_sync();   // the peer's MMAs, copies and arrivals on this CTA are done
    tc_fence_after();
    if (warp == kMmaWarpD) tmem_dealloc_pair(tmem_base, 512);
}

template <bool NHWC, bool BF16>
__global__ void __launch_bounds__(kDirectThreads<NHWC>, 1)
    direct3x3_kernel(const __grid_constant__ DirectParts parts, const __grid_constant__ DirectRing ring, DevErr* err) {
    direct_body<NHWC, BF16, true>(parts.d, parts.count, parts.items, ring, err);
}

// Many problems (fp16 NCHW) as one work queue; descs device-resident, sorted by item_begin.
__global__ void __launch_bounds__(kDirectThreads<false>, 1)
    direct3x3_grouped(const DirectDesc* __restrict__ descs, int ndesc, int items, const __grid_constant__ DirectRing ring,
                      DevErr* err) {
    direct_body<false, false, false>(descs, ndesc, items, ring, err);
}

// U9[tap][Cp/8][Kp][8]: the KCRS filter as granules of 8 input channels, zero
// past C and K.  One thread per (output channel, granule).
__global__ void __launch_bounds__(256) direct_filter_kernel(const uint16_t* __restrict__ w, uint16_t* __restrict__ U, int K,
                                                           int C, int CG, int Kp) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= CG * Kp) return;
    const int g = idx / Kp, k = idx - g * Kp;
    uint16_t v[8][kTaps9];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int c = g * 8 + j;
        const uint16_t* src = w + (static_cast<long long>(k) * C + c) * kTaps9;
#pragma unroll
        for (int t = 0; t < kTaps9; ++t) v[j][t] = (k < K && c < C) ? src[t] : static_cast<uint16_t>(0);
    }
#pragma unroll
    for (int t = 0; t < kTaps9; ++t) {
        uint4 q;
        q.x = v[0][t] | (static_cast<uint32_t>(v[1][t]) << 16);
        q.y = v[2][t] | (static_cast<uint32_t>(v[3][t]) << 16);
        q.z = v[4][t] | (static_cast<uint32_t>(v[5][t]) << 16);
        q.w = v[6][t] | (static_cast<uint32_t>(v[7][t]) << 16);
        *reinterpret_cast<uint4*>(U + ((static_cast<long long>(t) * CG + g) * Kp + k) * 8) = q;
    }
}

// The KCRS filter back from U9, one thread per value.
__global__ void __launch_bounds__(256) direct_unfilter_kernel(const uint16_t* __restrict__ U, uint16_t* __restrict__ w, int K,
                                                             int C, int CG, int Kp) {
    const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= static_cast<long long>(K) * C * kTaps9) return;
    const int t = static_cast<int>(idx % kTaps9), c = static_cast<int>(idx / kTaps9 % C);
    const int k = static_cast<int>(idx / kTaps9 / C);
    w[idx] = U[((static_cast<long long>(t) * CG + c / 8) * Kp + k) * 8 + (c & 7)];
}

// Output positions of n images, up to the last one.
long long positions(const DirectDesc& d, long long n) {
    return (n - 1) * d.img + static_cast<long long>(d.oh - 1) * d.pw + d.ow;
}

int window_of(int mb, int pw) { return kRows * mb + 2 * pw + 2; }

// One window stage: two granules; 32 more than a multiple of 128, so that the
// four granules of a channels-last pixel, in two stages, fall in different banks.
int window_bytes(int win) { return (2 * granule_bytes(win) + 127) / 128 * 128 + 32; }

int b_stage_bytes(int bn) { return kTaps9 * bn * 16; }

// Fewest window stages.  A producer group waits for the release of a stage by
// the parity of its use, which tells one use from the next but not from the one
// after: when the group comes to its next chunk, the use before last of that
// chunk's stage has to be over.  What it knows to be over is the use that freed
// the stage of its last chunk, na chunks before that one.  So na may not be less
// than the chunks it moves on by: three, or channels-last, by pairs of chunks,
// five from the second of one pair to the first of the next.
constexpr int least_stages(bool nhwc) { return nhwc ? 2 * kGroups - 1 : kGroups; }

// Ring depths for one window size and channel tile; false when the fewest
// window stages and two of the filter do not fit.
bool size_ring(DirectRing& r, int a_bytes, int b_bytes, bool nhwc) {
    const int fixed = 1024 + kHeader + (nhwc ? kTables * table_bytes(max_window(a_bytes)) : 0), room = kMaxSmem - fixed;
    r.a_bytes = a_bytes;
    r.b_bytes = b_bytes;
    // as many chunks ahead on both sides; what is left over goes to the windows
    for (int nb = std::min(kMaxRingB, room / (a_bytes + b_bytes)); nb >= 2; --nb) {
        const int na = std::min(kMaxRingA, (room - nb * b_bytes) / a_bytes);
        if (na >= least_stages(nhwc)) {
            r.nb = nb;
            r.na = na;
            r.smem_bytes = std::max(kMinSmem, nb * b_bytes + na * a_bytes + fixed);
            return true;
        }
    }
    return false;
}

// Cycles of one item of mb x 256 positions x bn channels: per chunk the longer
// of its 9 mb MMAs (each bn / 2 cycles of tensor time for 256 x bn x 16 on a
// pair, or the shared-memory reads of its operands: 4 KB of window and 16 bn
// bytes of filter per CTA at 128 bytes per cycle) and the producers' time for
// the window; plus what an item costs however short.
double item_cycles(int bn, int mb, int pw, int chunks) {
    const double mma = 9.0 * mb * std::max(bn / 2.0, 36.0 + bn / 8.0);
    const double prod = 150.0 + 2.0 * window_of(mb, pw);
    return chunks * std::max(mma, prod) + 1200.0 + 120.0 * mb * bn / 32;
}

template <auto Kernel, class... Args>
cudaError_t launch_cluster(int pairs, int threads, int smem, cudaStream_t s, const Args&... args) {
    const cudaError_t e = allow_smem<Kernel>(kMaxSmem);
    return e == cudaSuccess ? launch_pairs(Kernel, pairs, threads, smem, s, args...) : e;
}

// CTA pairs that run at once (one CTA per SM; a cluster stays within a GPC)
int max_pairs(int num_sms) {
    auto kern = direct3x3_kernel<false, false>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem) != cudaSuccess) return num_sms / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (num_sms / 2));
    cfg.blockDim = dim3(kDirectThreads<false>);
    cfg.dynamicSmemBytes = kMaxSmem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
        cudaGetLastError();
        return num_sms / 2;
    }
    return std::min(n, num_sms / 2);
}

}  // namespace

int direct_threads(bool nhwc) { return nhwc ? kDirectThreads<true> : kDirectThreads<false>; }

long long direct_filter_bytes(int K, int C) {
    return static_cast<long long>(kTaps9) * ((C + 7) / 8 * 8) * ((K + 7) / 8 * 8) * 2;
}

namespace {

// One way to cut a problem: items of mb x 256 positions x bn channels, and the
// positions past the last whole round of items in smaller ones.
struct Split {
    int bn = 0, mb = 0;
    long long main_tiles = 0;     // tiles of the main part
    int tail_bn = 0, tail_mb = 0; // 0: no tail
    double cycles = 0;
};

bool tile_fits(int bn, int mb, int pw, DirectRing* ring, bool nhwc) {
    if (bn * mb > 256) return false;
    const int a = window_bytes(window_of(mb, pw));
    DirectRing r;
    if (!size_ring(r, a, b_stage_bytes(bn), nhwc)) return false;
    if (ring) *ring = r;
    return true;
}

// Cycles of every item shape that fits (0: does not), by log2 mb and bn / 32 - 1.
struct TileCosts {
    double one[4][8];
    TileCosts(int pw, int chunks, int only_bn, int only_mb, bool nhwc) {
        for (int i = 0; i < 4; ++i)
            for (int j = 0; j < 8; ++j) {
                const int mb = 1 << i, bn = 32 * (j + 1);
                const bool out = (only_mb && mb != only_mb) || (only_bn && bn != only_bn) || !tile_fits(bn, mb, pw, nullptr, nhwc);
                one[i][j] = out ? 0 : item_cycles(bn, mb, pw, chunks);
            }
    }
};

// Least rounds x cycles for `pos` positions over `pairs` pairs; with `tail`,
// the positions past the last whole round may take another shape.
Split best_split(long long pos, int K, int pairs, const TileCosts& cost, const TileCosts* tail) {
    Split best;
    for (int i = 0; i < 4; ++i)
        for (int j = 0; j < 8; ++j) {
            const double one = cost.one[i][j];
            if (one == 0) continue;
            Split s;
            s.mb = 1 << i;
            s.bn = 32 * (j + 1);
            const long long rows = 2LL * kRows * s.mb;
            const long long tiles = (pos + rows - 1) / rows, nb = (K + s.bn - 1) / s.bn, items = tiles * nb;
            s.main_tiles = tiles;
            s.cycles = static_cast<double>((items + pairs - 1) / pairs) * one;
            if (best.bn == 0 || s.cycles < best.cycles) best = s;
            // whole rounds in the main part, the rest in items that take less than one more round
            const long long main = items / pairs * pairs / nb;
            const double main_cycles = static_cast<double>((main * nb + pairs - 1) / pairs) * one;
            if (!tail || main <= 0 || main >= tiles || main_cycles >= best.cycles) continue;
            const Split t = best_split(pos - main * rows, K, pairs, *tail, nullptr);
            s.main_tiles = main;
            s.tail_bn = t.bn;
            s.tail_mb = t.mb;
            s.cycles = main_cycles + t.cycles;
            if (s.cycles < best.cycles) best = s;
        }
    return best;
}

cudaError_t encode_filter(DirectDesc& d, const void* U, bool bf16) {
    const cuuint64_t CG = static_cast<cuuint64_t>((d.c + 7) / 8), Kr = static_cast<cuuint64_t>((d.k + 7) / 8);
    cuuint64_t dims[4] = {64, Kr, CG, kTaps9};
    cuuint64_t strides[3] = {128, Kr * 128, CG * Kr * 128};
    cuuint32_t box[4] = {64, static_cast<cuuint32_t>(d.bn / 16), 2, kTaps9};
    return encode_tiled(&d.tmU, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
                        const_cast<void*>(U), dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE) == CUDA_SUCCESS
               ? cudaSuccess
               : cudaErrorInvalidValue;
}

// fields of an item shape
void set_tile(DirectDesc& d, int bn, int mb) {
    d.bn = bn;
    d.mb = mb;
    d.cta_rows = kRows * mb;
    d.win = window_of(mb, d.pw);
    d.gran = granule_bytes(d.win);
    d.n_blocks = (d.k + bn - 1) / bn;
    d.fd_nb = make_fastdiv(static_cast<uint32_t>(d.n_blocks));
}

cudaError_t describe_direct(DirectDesc& d, const Geom& g, bool nhwc) {
    d = DirectDesc{};
    if (nhwc && g.c % 8 != 0) return cudaErrorNotSupported;   // a pixel's granule is one 16-byte load
    d.n = g.n;
    d.c = g.c;
    d.h = g.h;
    d.w = g.w;
    d.k = g.k;
    d.pad_h = g.pad_h;
    d.pad_w = g.pad_w;
    d.oh = g.oh;
    d.ow = g.ow;
    const long long pw = static_cast<long long>(g.w) + std::max(g.pad_w, 2 * g.pad_w - 2);
    const long long ph = static_cast<long long>(g.h) + std::max(g.pad_h, 2 * g.pad_h - 2), img = ph * pw;
    // positions (with what the last items reach past them) and the window's
    // element offsets from its first image, in 32 bits
    if (g.n * img + 4 * pw + 8192 >= (1LL << 31)) return cudaErrorNotSupported;
    d.pw = static_cast<int>(pw);
    d.ph = static_cast<int>(ph);
    d.img = static_cast<int>(img);
    const long long imgs = std::min<long long>(g.n, (window_of(8, d.pw) + 2048) / img + 2);
    if (imgs * g.c * g.h * g.w >= (1LL << 31)) return cudaErrorNotSupported;
    // items of the smallest tile
    if ((positions(d, g.n) / (2 * kRows) + 1) * ((g.k + 31) / 32) >= (1LL << 30)) return cudaErrorNotSupported;
    d.c_chunks = (g.c + kChunkC - 1) / kChunkC;
    d.step_y = (2 * kGroupThreads) / g.w;
    d.step_x = (2 * kGroupThreads) % g.w;
    d.pad_step_i = kGroupThreads / d.pw;
    d.pad_step_j = kGroupThreads % d.pw;
    d.fd_img = make_fastdiv(static_cast<uint32_t>(d.img));
    d.fd_pw = make_fastdiv(static_cast<uint32_t>(d.pw));
    d.fd_hw = make_fastdiv(static_cast<uint32_t>(static_cast<long long>(g.h) * g.w));
    d.fd_w = make_fastdiv(static_cast<uint32_t>(g.w));
    return cudaSuccess;
}

// the descriptor's tensors, and its items [begin, begin + tiles * n_blocks) from position pos0
void place(DirectDesc& d, const void* x, void* y, bool nhwc, long long pos0, long long tiles, int begin) {
    d.x = x;
    d.y = y;
    d.pos0 = static_cast<int>(pos0);
    d.item_begin = begin;
    d.items = static_cast<int>(tiles * d.n_blocks);
    // (the mask of padding positions covers 32 per thread)
    d.pairs = !nhwc && d.w % 2 == 0 && reinterpret_cast<uintptr_t>(x) % 4 == 0 && d.win <= kMaxPadBits * kGroupThreads;
    d.vec = d.k % 8 == 0 && reinterpret_cast<uintptr_t>(y) % 16 == 0;
}

}  // namespace

int direct_max_pairs(int num_sms) {
    static std::atomic<int> cached{0};   // one device type per process; the same answer from every thread
    int n = cached.load();
    if (n == 0) cached.store(n = max_pairs(num_sms));
    return n;
}

bool direct_supported(const Geom& g, bool nhwc) {
    DirectDesc d;
    return describe_direct(d, g, nhwc) == cudaSuccess && tile_fits(32, 1, d.pw, nullptr, nhwc);
}

cudaError_t plan_direct(DirectPlan& dp, const Geom& g, bool nhwc, bool bf16, const void* U, int tile, int num_sms) {
    DirectDesc d;
    if (cudaError_t e = describe_direct(d, g, nhwc); e != cudaSuccess) return e;
    dp.max_pairs = direct_max_pairs(num_sms);
    const int bn = tile & 0x1ff, mb = tile >> 9;
    const TileCosts any(d.pw, d.c_chunks, 0, 0, nhwc), asked(d.pw, d.c_chunks, bn, mb, nhwc);
    const Split s = best_split(positions(d, g.n), g.k, dp.max_pairs, asked, &any);
    if (s.bn == 0 || !tile_fits(s.bn, s.mb, d.pw, &dp.ring, nhwc)) return cudaErrorNotSupported;
    set_tile(d, s.bn, s.mb);
    dp.main = d;
    dp.tail = d;
    dp.has_tail = s.tail_bn != 0;
    if (dp.has_tail) {
        set_tile(dp.tail, s.tail_bn, s.tail_mb);
        DirectRing r;
        // one ring serves both parts: the larger stages
        const int a = std::max(window_bytes(d.win), window_bytes(dp.tail.win));
        if (size_ring(r, a, std::max(b_stage_bytes(d.bn), b_stage_bytes(dp.tail.bn)), nhwc))
            dp.ring = r;
        else
            dp.has_tail = false;
    }
    dp.main_tiles = static_cast<int>(s.main_tiles);
    dp.nhwc = nhwc;
    dp.bf16 = bf16;
    if (!U) return cudaSuccess;
    cudaError_t e = encode_filter(dp.main, U, bf16);
    if (e == cudaSuccess && dp.has_tail) e = encode_filter(dp.tail, U, bf16);
    return e;
}

cudaError_t launch_direct_unfilter(const void* U, void* weight, int K, int C, cudaStream_t stream) {
    const int CG = (C + 7) / 8, Kp = (K + 7) / 8 * 8;
    const long long n = static_cast<long long>(K) * C * kTaps9;
    direct_unfilter_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(
        static_cast<const uint16_t*>(U), static_cast<uint16_t*>(weight), K, C, CG, Kp);
    return cudaGetLastError();
}

cudaError_t launch_direct_filter(const void* weight, void* U, int K, int C, cudaStream_t stream) {
    const int CG = (C + 7) / 8, Kp = (K + 7) / 8 * 8;
    const long long n = static_cast<long long>(CG) * Kp;
    direct_filter_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(
        static_cast<const uint16_t*>(weight), static_cast<uint16_t*>(U), K, C, CG, Kp);
    return cudaGetLastError();
}

int direct_parts(const DirectPlan& dp, const void* x, void* y, int n_images, DirectParts& out) {
    const long long pos = positions(dp.main, n_images);
    auto part = [&](const DirectDesc& d, long long pos0, long long tiles, int begin) {
        DirectDesc& o = out.d[out.count++];
        o = d;
        o.n = n_images;
        place(o, x, y, dp.nhwc, pos0, tiles, begin);
        return begin + o.items;
    };
    const long long rows = 2LL * dp.main.cta_rows, tiles = (pos + rows - 1) / rows;
    out.count = 0;
    if (!dp.has_tail || tiles <= dp.main_tiles) {
        out.items = part(dp.main, 0, tiles, 0);
    } else {
        const long long done = dp.main_tiles * rows, trows = 2LL * dp.tail.cta_rows;
        out.items = part(dp.main, 0, dp.main_tiles, 0);
        out.items = part(dp.tail, done, (pos - done + trows - 1) / trows, out.items);
    }
    return out.items;
}

// Item shapes for queues of many problems: throughput decides (items x
// cycles), not rounds, as the problems fill each other's; but no item longer
// than a third of the queue's time where a shorter one is to be had.  Longest
// items first, so that the pairs, which take the items in turn, end together.
//
// Problems share a queue where one ring has room for the widest window and the
// widest filter tile of all, three stages of each (or as many as a problem's own
// ring has): up to rows of about 220 columns always.  The problems with wider
// windows get queues of their own.  32x256x56^2 -> 256, 16x128x28^2 -> 128 and
// 8x512x14^2 -> 512 take 84-88 us together; with 64x560^2 -> 64, 56 us by itself,
// they took 199 in one queue of two filter stages and take 138 in two; with
// 64x760^2 -> 64 (108) 323 when its items were held to one block of positions, now
// 181; with 64x300^2 -> 64 (20) 102-104 in one.  Each problem's own stages fit
// (choose), so every set of problems has its queues.
cudaError_t make_direct_queues(const DirectProblem* p, int n, int pairs, DirectDesc* out, std::vector<DirectQueue>& queues) {
    struct Pick {
        DirectDesc d;
        double one;
        int i, queue;
    };
    std::vector<Pick> picks(n);
    // stages small enough for four of each; of wide rows, whose windows are too
    // long for that anyway, any that fit (several blocks share the window's halo)
    auto fits = [](int bn, int mb, int pw) {
        DirectRing r;
        constexpr int kShared = 18 * 1024;
        return tile_fits(bn, mb, pw, &r, false) &&
               (mb == 1 || r.a_bytes <= kShared || window_bytes(window_of(1, pw)) > kShared);
    };
    auto choose = [&](Pick& k, double longest) {
        const long long pos = positions(k.d, k.d.n);
        double best = 0;
        int bbn = 0, bmb = 0;
        for (int mb = 1; mb <= 8; mb *= 2)
            for (int bn = 32; bn <= 256; bn += 32) {
                if (!fits(bn, mb, k.d.pw)) continue;
                const double one = item_cycles(bn, mb, k.d.pw, k.d.c_chunks);
                const long long rows = 2LL * kRows * mb;
                double t = static_cast<double>((pos + rows - 1) / rows * ((k.d.k + bn - 1) / bn)) * one;
                if (longest > 0 && one > longest) t *= one / longest;
                if (bbn == 0 || t < best) {
                    best = t;
                    bbn = bn;
                    bmb = mb;
                }
            }
        if (bbn == 0) return -1.0;
        set_tile(k.d, bbn, bmb);
        k.one = item_cycles(bbn, bmb, k.d.pw, k.d.c_chunks);
        return best;
    };
    double total = 0;
    for (int i = 0; i < n; ++i) {
        if (cudaError_t e = describe_direct(picks[i].d, p[i].g, false); e != cudaSuccess) return e;
        picks[i].i = i;
        const double t = choose(picks[i], 0);
        if (t < 0) return cudaErrorNotSupported;
        total += t;
    }
    const double longest = total / pairs / 3;
    for (Pick& k : picks)
        if (k.one > longest) choose(k, longest);
    // narrower windows first, each problem into the first queue whose ring has room for it
    std::stable_sort(picks.begin(), picks.end(), [](const Pick& x, const Pick& y) { return x.d.win < y.d.win; });
    queues.clear();
    constexpr int kEnough = 3;
    std::vector<std::pair<int, int>> least;   // stages that a queue's ring keeps
    for (Pick& k : picks) {
        const int a = window_bytes(k.d.win), b = b_stage_bytes(k.d.bn);
        DirectRing own, r;
        if (!size_ring(own, a, b, false)) return cudaErrorNotSupported;
        for (k.queue = 0;; ++k.queue) {
            if (k.queue == static_cast<int>(queues.size())) {
                queues.push_back(DirectQueue{});
                least.push_back({0, 0});
            }
            DirectQueue& q = queues[k.queue];
            const int na = std::max(least[k.queue].first, std::min(kEnough, own.na));
            const int nb = std::max(least[k.queue].second, std::min(kEnough, own.nb));
            if (size_ring(r, std::max(a, q.ring.a_bytes), std::max(b, q.ring.b_bytes), false) && r.na >= na && r.nb >= nb) {
                q.ring = r;
                least[k.queue] = {na, nb};
                ++q.n;
                break;
            }
        }
    }
    std::sort(picks.begin(), picks.end(), [](const Pick& x, const Pick& y) {
        return x.queue != y.queue ? x.queue < y.queue : x.one != y.one ? x.one > y.one : x.i < y.i;
    });
    int next = 0;
    for (DirectQueue& q : queues) {
        q.first = next;
        long long begin = 0;
        for (; next < q.first + q.n; ++next) {
            DirectDesc& d = picks[next].d;
            const DirectProblem& pr = p[picks[next].i];
            if (pr.U)
                if (cudaError_t e = encode_filter(d, pr.U, false); e != cudaSuccess) return e;
            const long long rows = 2LL * d.cta_rows;
            place(d, pr.x, pr.y, false, 0, (positions(d, d.n) + rows - 1) / rows, static_cast<int>(begin));
            begin += d.items;
            if (begin >= (1LL << 31)) return cudaErrorNotSupported;
            out[next] = d;
        }
        q.items = static_cast<int>(begin);
    }
    return cudaSuccess;
}

cudaError_t launch_direct_grouped(const DirectDesc* descs, const DirectQueue& q, int pairs, DevErr* err, cudaStream_t stream) {
    return launch_cluster<direct3x3_grouped>(std::min(q.items, pairs), kDirectThreads<false>, q.ring.smem_bytes, stream,
                                             descs + q.first, q.n, q.items, q.ring, err);
}

cudaError_t launch_direct(const DirectPlan& dp, const void* x, void* y, int n_images, DevErr* err, cudaStream_t stream) {
    DirectParts p;
    const int pairs = std::min(direct_parts(dp, x, y, n_images, p), dp.max_pairs);
    const int threads = direct_threads(dp.nhwc), smem = dp.ring.smem_bytes;
    if (dp.nhwc)
        return launch_cluster<direct3x3_kernel<true, false>>(pairs, threads, smem, stream, p, dp.ring, err);
    return dp.bf16 ? launch_cluster<direct3x3_kernel<false, true>>(pairs, threads, smem, stream, p, dp.ring, err)
                   : launch_cluster<direct3x3_kernel<false, false>>(pairs, threads, smem, stream, p, dp.ring, err);
}

}  // namespace wg
