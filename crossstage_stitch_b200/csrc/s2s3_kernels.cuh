// S2 (FAST-9 + NMS + 2K pre-selection + Harris + top-K) and S3 (7x7 blur +
// IC angle + rBRIEF-256) kernels for sm_100a.
//
// Every kernel reads its image and buffers from a "job". A job source is
// either one job passed by value (the per-image stage call) or a device table
// of jobs plus a block-prefix array (the batched chain, where one launch
// covers every image of every pair). Results are identical either way, but for
// the blur: the pyramid and batched paths fuse its products and sums, the
// per-image S3 call rounds each as the reference does, and on noise some 3 blurred
// pixels of a million differ by one (first_taps).
//
// Reference semantics (file:line in the reference tree):
//   FAST score        src/s2_s3/s2.cu:37-67   (cornerScore<16>, circle order)
//   NMS + histogram   src/s2_s3/s2.cu:81-106
//   2K threshold      src/s2_s3/s2.cu:108-139 (SelectParams)
//   raster compaction src/s2_s3/s2.cu:141-235 (all above, then first ties)
//   Harris            src/s2_s3/s2.cu:247-285 (no-FMA float formula, key)
//   top-K order       src/s2_s3/s2.cu:287-310 (descending key)
//   blur              src/s2_s3/s3.cu:41-73
//   describe          src/s2_s3/s3.cu:75-157
#pragma once

#include <type_traits>

#include "common.cuh"

namespace stitch::b200::s2s3 {

// ---------------------------------------------------------------- jobs

struct SelectParams {
    std::uint32_t threshold;  // FAST score at the 2K boundary
    std::uint32_t above;      // maxima with score > threshold
    std::uint32_t ties;       // maxima at the threshold that are kept
    std::uint32_t selected;   // above + ties
};

// Keys of the jobs of a batch that the sort takes, summed up by the selection
// (zeroed per run).
struct RankTotals {
    unsigned long long squares;
    std::uint32_t sum, largest;
};

// Per-job counters of the detect kernels, after the 256 histogram bins. kTies
// counts the maxima at the threshold written behind the keys above it, or listed
// (TieList). Scores start at 1, so bin 0 of the histogram counts the select blocks
// that have finished: a word more would take the smallest workspaces.
enum DetectCounter { kListed, kAboveWritten, kTies, kTileQueue, kDetectCounters };
constexpr int kSelectDoneBin = 0;
constexpr int kHistWords = 256 + kDetectCounters;  // one job's histogram and counters

struct alignas(16) DetectJob {  // 16-byte multiple: copied into shared memory in 16-byte chunks
    const std::uint8_t* image;
    int width, height, pitch;
    int threshold, max_keypoints;
    float harris_k;
    // workspace
    std::uint64_t* maxima;         // NMS maxima listed by the FAST kernel: (score << 32) | raster index
    int max_maxima;                // capacity of `maxima`
    std::uint32_t* hist;           // [256] scores of the listed maxima (bin 0: kSelectDoneBin), then DetectCounter words;
                                   // all zeroed before the FAST launch
    SelectParams* params;
    std::uint64_t* keys;           // [candidates]
    // output
    float* x;
    float* y;
    float* response;  // may be null
    int* count;
    // On-demand S3 blur (pyramid and batched paths; null elsewhere): the
    // blur tiles that final keypoints sample are flagged in blur_marks
    // (one word per tile, zeroed every run) and listed once each in
    // blur_list as (describe job, tile) behind the launch-wide *blur_count.
    std::uint32_t* blur_marks;
    uint2* blur_list;
    std::uint32_t* blur_count;
    int job;  // this job's index in the describe table of the launch
    // launch bookkeeping
    int tiles_x, tiles, select_blocks, candidates;
    std::uint32_t tiles_x_magic;  // ceil(2^32 / tiles_x), 0 for one tile column (see fast_origin)
    __host__ __device__ std::uint32_t* counters() const { return hist + 256; }
};

struct DescribeJob {
    const std::uint8_t* image;
    int width, height, pitch;
    std::uint8_t* blurred;  // rows of blur_pitch bytes
    int blur_pitch;
    const float* x;
    const float* y;
    const int* count;
    int capacity;
    std::uint8_t* out;  // rows of row_stride bytes
    int row_stride;
    int tiles_x, tiles;  // blur tiles
    // Pyramid layer (level_counts != null): the layer's keypoints are in
    // layer coordinates in x/y/response; the describe kernel writes them,
    // multiplied by `scale`, and their descriptors to the image's
    // concatenated outputs after the keypoints of lower layers
    // (level_counts[0..level-1]) and adds the layer's count to *out_count.
    const float* response;
    float* out_x;
    float* out_y;
    float* out_response;  // may be null
    int* out_count;
    const int* level_counts;
    int level;
    float scale;
};

// One pyramid layer: `dst` (dense) resized from `src` by fixed-point
// bilinear interpolation (cv::resize INTER_LINEAR_EXACT on 8-bit images).
struct ResizeJob {
    const std::uint8_t* src;
    int src_width, src_height, src_pitch;
    std::uint8_t* dst;
    int width, height, pitch;
    int tiles_x, tiles;
    double scale_x, scale_y;  // linear_exact_scale of each axis, computed by the host
};

// Per-image job passed by value.
template <class Job> struct OneJob {
    Job job;
    __device__ bool find(int block, int /*kind*/, Job* j, int* local) const {
        *j = job;
        *local = block;
        return true;
    }
    __device__ Job at(int /*index*/) const { return job; }
    __device__ int count() const { return 1; }
};

// Device table: prefix[kind * (n + 1) + i] is the first block of job i for
// launch kind `kind`; blocks past the end are idle. With map[kind] set, entry
// b of it is (job << 16 | block within the job) for block b of that kind, so
// a block finds its job in one load instead of a binary search over the
// prefix (each step of which waits on the previous one).
constexpr int kMapKinds = 16;
template <class Job> struct JobTable {
    const Job* jobs;
    const int* prefix;
    int n;
    const std::uint32_t* map[kMapKinds] = {};
    int map_blocks[kMapKinds] = {};
    __device__ bool find(int block, int kind, Job* j, int* local) const {
        if (const std::uint32_t* m = map[kind]) {
            if (block >= map_blocks[kind]) return false;
            const std::uint32_t e = __ldg(m + block);
            *j = jobs[e >> 16];
            *local = static_cast<int>(e & 0xffffu);
            return true;
        }
        const int* p = prefix + kind * (n + 1);
        if (block >= p[n]) return false;
        int lo = 0, hi = n - 1;
        while (lo < hi) {  // largest i with p[i] <= block
            const int mid = (lo + hi + 1) >> 1;
            if (p[mid] <= block) lo = mid; else hi = mid - 1;
        }
        *j = jobs[lo];
        *local = block - p[lo];
        return true;
    }
    __device__ Job at(int index) const { return jobs[index]; }
    __device__ int count() const { return n; }
};

// A few jobs passed by value (the layers of one image's pyramid):
// first[kind][i] is the first block of job i; linear search.
template <class Job, int kJobs, int kKinds> struct InlineTable {
    Job jobs[kJobs];
    int first[kKinds][kJobs + 1];
    int n;
    __device__ bool find(int block, int kind, Job* j, int* local) const {
        if (block >= first[kind][n]) return false;
        int i = 0;
        while (i + 1 < n && first[kind][i + 1] <= block) ++i;
        *j = jobs[i];
        *local = block - first[kind][i];
        return true;
    }
    __device__ Job at(int index) const { return jobs[index]; }
    __device__ int count() const { return n; }
};

// Launch kinds of the detect table: kFastKind entries are the FAST tiles of
// each job (looked up by tile index from the persistent FAST kernel's
// queue), kSelectKind blocks walk a job's maxima list (a job's last one picks its
// ties), kHarrisKind blocks have kHarrisThreads candidates each (the ranking divides
// them further), kSortKind is one block per job, the top-K sort.
enum DetectKind { kFastKind = 0, kSelectKind = 1, kHarrisKind = 2, kSortKind = 3, kDetectKinds = 4 };
enum DescribeKind { kBlurKind = 0, kDescKind = 1, kDescribeKinds = 2 };

constexpr int kFastTileW = 64, kFastTileH = 64;

// Origin (x0, y0) of FAST tile `local` of a job: local / tiles_x by a
// multiply-high with ceil(2^32 / tiles_x), which is the quotient or one
// above it (the error term local * (magic - 2^32 / tiles_x) / 2^32 is below
// 1), then corrected.
__device__ __forceinline__ int2 fast_origin(const DetectJob& j, int local) {
    int ty = j.tiles_x_magic ? static_cast<int>(__umulhi(static_cast<std::uint32_t>(local), j.tiles_x_magic)) : local;
    if (ty * j.tiles_x > local) --ty;
    return make_int2((local - ty * j.tiles_x) * kFastTileW, ty * kFastTileH);
}
constexpr int kFastInW = kFastTileW + 8, kFastInH = kFastTileH + 8;  // halo 4 = FAST 3 + NMS 1
constexpr int kFastScW = kFastTileW + 2, kFastScH = kFastTileH + 2;
constexpr int kSelectPx = 65536;   // image pixels per select block (a job's maxima list is walked
                                   // by ceil(W * H / kSelectPx) blocks)
constexpr int kFastThreads = 256;
constexpr int kFastCtasPerSm = 7;  // resident FAST blocks per SM (shared memory); the persistent grid is 148 x this
constexpr int kTieCap = 16384;      // most tie list entries; more ties are picked from the maxima list itself
constexpr int kTieRank = 1024;      // ties ranked against each other in shared memory
// Largest offset of a rotated rBRIEF sample from its keypoint: the pattern's
// coordinates lie within a radius of 18.39 px (|x|, |y| <= 13), so a rotated
// coordinate rounds to at most 18.
constexpr int kSampleRadius = 18;
constexpr int kHarrisThreads = 128;  // candidates of a harris (and rank) block: small blocks spread one image's few
                                     // thousand candidates over the chip
constexpr int kRankKeys = 32;        // keys a rank block ranks: small blocks, so that one image's largest layer
                                     // spreads over the chip
constexpr int kRankThreads = 512;
constexpr int kRankPer = kHarrisThreads / kRankKeys;  // rank blocks per harris block
constexpr int kRankTile = 1024;      // keys staged at a time
constexpr int kSortCap = 16384;    // candidates sorted in shared memory by one block
constexpr int kSortThreads = 1024;
// Threads of a batch's sort blocks: few where a job has few keys for them or many
// jobs share an SM. Noise of 500x400, us with 256, 512 and 1024 threads: 64 jobs of 1000
// candidates 24, 18, 18; 512 jobs of up to 868 (8 layers) 37, 31, 39; 1024 of them 46,
// 46, 59, and at 512x512 29, 31, 45; 512 jobs of up to 434 19, 23, 28.
constexpr int sort_threads(int max_candidates, int jobs) {
    return max_candidates <= 512 || (max_candidates <= 1024 && jobs >= 6 * 148) ? 256 : max_candidates <= 1024 ? 512 : kSortThreads;
}
constexpr int kSortChunk = 64;      // keys a warp sorts in registers (2 per lane)
constexpr int kBlurTileW = 64, kBlurTileH = 64;
constexpr int kDescWarps = 8;
// Keypoints per warp of a describe block: as many as leave the chip's block
// slots filled, up to 8, so that a block's tables and a warp's angle pass are
// shared by more. 512x512, K = 1000, one image: 20 us at 4, 14 us at 1; 64
// pairs, K = 2000: 174 us at 4, 166 at 8, 174 at 16.
constexpr int kDescMaxRounds = 8;
constexpr int kDescCtasPerSm = 5;
__host__ __device__ inline int desc_keys(long long keypoints) {
    int rounds = kDescMaxRounds;
    while (rounds > 1 && keypoints < static_cast<long long>(kDescWarps) * rounds * 148 * kDescCtasPerSm) rounds /= 2;
    return kDescWarps * rounds;
}
constexpr int kEdge = 31;
constexpr int kResizeTileW = 128, kResizeTileH = 64;  // the tile of a launch over many images
constexpr int kResizeTallH = 128;                     // and of one with tiles enough for it (resize_tile_rows)
constexpr int kMaxLevels = 16;
static_assert(kMaxLevels <= kMapKinds && kDetectKinds <= kMapKinds, "block map kinds");

// ------------------------------------------------------------- FAST + NMS

// float32 taps of a 7-tap, sigma-2 Gaussian (exp in float64, normalised,
// rounded to float32); equal to cv::getGaussianKernel(7, 2, CV_32F).
__device__ __forceinline__ float blur_tap(int i) {
    switch (i) {
        case 0: case 6: return 0x1.1f5f62p-4f;
        case 1: case 5: return 0x1.0c70fcp-3f;
        case 2: case 4: return 0x1.869472p-3f;
        default: return 0x1.ba95c0p-3f;
    }
}

// Border reflection without repeating the edge pixel (BORDER_REFLECT_101).
__device__ __forceinline__ int reflect101(int i, int n) {
    if (n == 1) return 0;
    while (i < 0 || i >= n) i = i < 0 ? -i : 2 * n - 2 - i;
    return i;
}

// FAST-9 score of the pixel at p (row stride `stride`), 0 when it is not a
// corner. With d_k = centre - ring_k over the 16-pixel circle, a 9-pixel arc
// scores min(d) when darker and min(-d) when brighter; the raw score is the
// largest over the 16 arcs of both kinds, the pixel is a corner iff the raw
// score exceeds the threshold, and it then scores raw - 1. Both kinds run
// at once as unsigned 16-bit lanes q_k = (d_k + 256) | (256 - d_k) << 16
// (all in [1, 511]), which is c + r_k * 0xffff for c = (v + 256) |
// (256 - v) << 16: one multiply-add per ring pixel, no borrow between the
// lanes. 9-wide arc minima come from 3-wide ones through the 3-input 16x2
// minimum (min3(m3[k], m3[k+3], m3[k+6])), and the 16 arcs are folded with
// the 3-input maximum. (CUDA 12.9 ptxas at -O1 and above miscompiles the
// signed max(min(arc), -max(arc)) form of this score on sm_100; this
// unsigned form is exact at every optimisation level.)
__device__ __forceinline__ int fast_score(const std::uint8_t* p, int stride, int thr) {
    const unsigned v = p[0];
    const unsigned c = (v + 256u) | ((256u - v) << 16);
    const unsigned r[16] = {p[3 * stride],      p[3 * stride + 1],  p[2 * stride + 2],  p[stride + 3],
                            p[3],               p[-stride + 3],     p[-2 * stride + 2], p[-3 * stride + 1],
                            p[-3 * stride],     p[-3 * stride - 1], p[-2 * stride - 2], p[-stride - 3],
                            p[-3],              p[stride - 3],      p[2 * stride - 2],  p[3 * stride - 1]};
    unsigned q[16], m3[16], m9[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) q[k] = c + r[k] * 0xffffu;
#pragma unroll
    for (int k = 0; k < 16; ++k) m3[k] = __vimin3_u16x2(q[k], q[(k + 1) & 15], q[(k + 2) & 15]);
#pragma unroll
    for (int k = 0; k < 16; ++k) m9[k] = __vimin3_u16x2(m3[k], m3[(k + 3) & 15], m3[(k + 6) & 15]);
    const unsigned b0 = __vimax3_u16x2(m9[0], m9[1], m9[2]), b1 = __vimax3_u16x2(m9[3], m9[4], m9[5]);
    const unsigned b2 = __vimax3_u16x2(m9[6], m9[7], m9[8]), b3 = __vimax3_u16x2(m9[9], m9[10], m9[11]);
    const unsigned b4 = __vimax3_u16x2(m9[12], m9[13], m9[14]);
    const unsigned best = __vmaxu2(__vimax3_u16x2(b0, b1, b2), __vimax3_u16x2(b3, b4, m9[15]));
    const unsigned lo = best & 0xffffu, hi = best >> 16;
    const int score = static_cast<int>(lo > hi ? lo : hi) - 256;
    return score > thr ? score - 1 : 0;
}

// Compass test of four pixels, a necessary condition for a FAST-9 corner: every
// 9-pixel arc of the circle holds one of the compass pixels s0, s8 (3 below, 3
// above) and one of s4, s12 (3 right, 3 left), so an arc brighter than v + t
// needs hi = min(max(s0, s8), max(s4, s12)) >= v + t + 1 and one darker than v -
// t needs lo = max(min(s0, s8), min(s4, s12)) <= v - t - 1.
// Two pixels per word, their bytes in the high bytes of the 16-bit lanes: the
// minima and maxima of such lanes are right in the high byte whatever the low
// bytes hold, so the odd pixels' words are taken as loaded, the even pixels'
// shifted left by 8, and only hi, lo and v are masked. In the masked lanes
// hi + 0x8000 - v - (t + 1) and v + 0x8000 - lo - (t + 1) have their top bit
// set exactly when the test passes, with no borrow between lanes.
// The kernel is bound by the ALU pipe and by issue slots: the sums are
// multiply-adds, which run on the FMA pipe (`one` and `minus` are 1 and -1
// where the compiler cannot see them). FAST of 64 pairs at 512x512 with 8
// layers: 252 -> 240 us with this test, 221 with eight pixels per thread (the
// list bookkeeping once per eight), 217 with the staging's chunk per thread
// fixed; 30 mixed pairs: 1300, 1227, 1143, 1120 us.
struct Compass {
    std::uint32_t one, minus, top;  // top = 0x80008000 - (t + 1) in both lanes
};

__device__ __forceinline__ std::uint32_t mad32(std::uint32_t a, std::uint32_t b, std::uint32_t c) {
    std::uint32_t d;
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// Top bits of the lanes whose pixel passes; s0 .. s12 and v with the pixels in
// the high bytes, v with clear low bytes shifted down (masked).
__device__ __forceinline__ std::uint32_t compass_lanes(std::uint32_t v, std::uint32_t s0, std::uint32_t s4,
                                                       std::uint32_t s8, std::uint32_t s12, const Compass& k) {
    const std::uint32_t hi = __byte_perm(__vminu2(__vmaxu2(s0, s8), __vmaxu2(s4, s12)), 0, 0x4341);
    const std::uint32_t lo = __byte_perm(__vmaxu2(__vminu2(s0, s8), __vminu2(s4, s12)), 0, 0x4341);
    return mad32(hi, k.one, mad32(v, k.minus, k.top)) | mad32(lo, k.minus, mad32(v, k.one, k.top));
}

// Survivor bits 0 .. 3 of the four pixels of word v, with the words left and
// right of it and those three rows below and above; other bits are undefined.
__device__ __forceinline__ unsigned compass_bits(std::uint32_t l, std::uint32_t v, std::uint32_t r, std::uint32_t s0,
                                                 std::uint32_t s8, const Compass& k) {
    const std::uint32_t odd = compass_lanes(__byte_perm(v, 0, 0x4341), s0, __funnelshift_r(v, r, 24), s8,
                                            __funnelshift_r(l, v, 8), k);
    const std::uint32_t even = compass_lanes(v & 0x00ff00ffu, mad32(s0, 256u, 0u), __funnelshift_r(v, r, 16),
                                             mad32(s8, 256u, 0u), l, k);
    // bits 14, 15 (pixels 0, 1) and 30, 31 (pixels 2, 3), then together
    const std::uint32_t m = (((even >> 1) & 0x40004000u) | (odd & 0x80008000u)) >> 14;
    return m | (m >> 14);
}

constexpr int kInStride = 96;
// Score rows hold columns x0-4 .. x0+67 of a tile at x0: words aligned with the
// staged bytes (score column c is staged byte kInOff + c). The tile and its
// 1-pixel ring are columns kScRing .. kScRing + kFastScW - 1.
constexpr int kInOff = 12, kScStride = 72, kScRing = 3;
constexpr int kScGroups = kScStride / 8;  // groups of 8 positions per score row

// Bytes k of wa and wb as a float pair (rows r, r + 1 of one column), each
// exact: the float 2^23 + b (byte b placed in the low mantissa) minus 2^23.
__device__ __forceinline__ float2 byte_pair(std::uint32_t wa, std::uint32_t wb, int k) {
    const float2 biased = make_float2(__uint_as_float(__byte_perm(wa, 0x4B000000u, 0x7440u + k)),
                                      __uint_as_float(__byte_perm(wb, 0x4B000000u, 0x7440u + k)));
    return __fadd2_rn(biased, make_float2(-8388608.0f, -8388608.0f));
}

// A blur tap in both lanes of a packed pair: two rows (or two columns) of the
// blur in one instruction stream.
__device__ __forceinline__ float2 tap_pair(int t) { return make_float2(blur_tap(t), blur_tap(t)); }

// Taps 0 and 1, then tap t, of a pair of sums. Packed: one rounding less per
// tap, in the order that the pyramid and batched paths have always had (the
// compiler joined their packed products and sums so; written out, the bytes no
// longer depend on it). Scalar: every product and sum rounded on its own, as
// the reference does. On noise 3 pixels of a million differ by one.
template <bool kPacked> __device__ __forceinline__ float2 first_taps(float2 v0, float2 v1) {
    return kPacked ? __ffma2_rn(tap_pair(0), v0, __fmul2_rn(tap_pair(1), v1))
                   : make_float2(__fadd_rn(__fmul_rn(blur_tap(0), v0.x), __fmul_rn(blur_tap(1), v1.x)),
                                 __fadd_rn(__fmul_rn(blur_tap(0), v0.y), __fmul_rn(blur_tap(1), v1.y)));
}
template <bool kPacked> __device__ __forceinline__ float2 next_tap(float2 sum, int t, float2 v) {
    return kPacked ? __ffma2_rn(tap_pair(t), v, sum)
                   : make_float2(__fadd_rn(sum.x, __fmul_rn(blur_tap(t), v.x)),
                                 __fadd_rn(sum.y, __fmul_rn(blur_tap(t), v.y)));
}

// Rounds two blur sums half-to-even to integers, in the low mantissa bits:
// adding 1.5 * 2^23 rounds a float below 2^22 to an integer the way
// __float2int_rn does, on the FP32 pipe (the conversion instruction runs at a
// sixteenth of its rate). No clamp: the taps are positive and rounding is
// monotone, so a sum lies between 0 and that of an all-255 window, which is
// below 255.5 (tests/test_gpu_detect_edges.py checks that window).
__device__ __forceinline__ float2 round_pair(float2 v) {
    return __fadd2_rn(v, make_float2(12582912.0f, 12582912.0f));
}

// Low bytes of four rounded sums (round_pair), first in the low byte.
__device__ __forceinline__ std::uint32_t pack_bytes(float2 a, float2 b) {
    const std::uint32_t lo = __byte_perm(__float_as_uint(a.x), __float_as_uint(a.y), 0x0040);
    const std::uint32_t hi = __byte_perm(__float_as_uint(b.x), __float_as_uint(b.y), 0x0040);
    return __byte_perm(lo, hi, 0x5410);
}

// Asynchronous 16-byte copy, global to shared memory (both 16-byte aligned).
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(gmem) : "memory");
}

// The FAST kernel's block map and job array where its source has them
// (tables staged by a plan); elsewhere the job is looked up in place.
template <class S> __device__ __forceinline__ const std::uint32_t* fast_map(const S&) { return nullptr; }
template <class S> __device__ __forceinline__ const DetectJob* fast_jobs(const S&) { return nullptr; }
template <> __device__ __forceinline__ const std::uint32_t* fast_map(const JobTable<DetectJob>& s) {
    return s.map[kFastKind];
}
template <class S> __device__ __forceinline__ int fast_map_tiles(const S&) { return 0; }
template <> __device__ __forceinline__ int fast_map_tiles(const JobTable<DetectJob>& s) { return s.map_blocks[kFastKind]; }
template <> __device__ __forceinline__ const DetectJob* fast_jobs(const JobTable<DetectJob>& s) { return s.jobs; }

// Stages rows y0-4 .. y0+67 and columns x0-16 .. x0+79 of the job's image in
// `in` (byte c of row r = image (y0-4+r, x0-16+c)). The FAST test never reads
// a position outside the image, so rows are clamped into it and the bytes of
// columns outside it are left as they are. With a 16-byte aligned image (base
// and pitch) every 16-byte chunk within a row's pitch (within the width on
// the last row) is one asynchronous copy, and a chunk that straddles the end
// of the last row is copied byte by byte; other images are loaded byte by
// byte with clamped columns. Asynchronous copies complete at the caller's
// cp_async_wait_all.
__device__ __forceinline__ void stage_fast_tile(const DetectJob& j, int local, std::uint8_t (*in)[kInStride]) {
    const int tid = threadIdx.x;
    const int W = j.width, H = j.height;
    const int2 org = fast_origin(j, local);
    const int y0 = org.y, x0 = org.x;
    const bool vec = ((reinterpret_cast<std::uintptr_t>(j.image) | static_cast<std::uintptr_t>(j.pitch)) & 15) == 0;
    if (vec) {
        // thread (r, q): chunk q of rows r, r + 42
        constexpr int kChunks = kInStride / 16, kRows = kFastThreads / kChunks;  // 6, 42
        const int r0 = tid / kChunks, q = tid - r0 * kChunks, cx = x0 - 16 + 16 * q;
        if (r0 < kRows && cx >= 0 && cx < W) {
            const std::uint8_t* const column = j.image + cx;
#pragma unroll
            for (int r = r0; r < kFastInH; r += kRows) {
                const int gy = min(max(y0 - 4 + r, 0), H - 1);
                const std::uint8_t* from = column + static_cast<std::size_t>(gy) * j.pitch;
                // bytes of the row that may be read: the pitch, the width on the last row
                if (cx + 16 <= (gy == H - 1 ? W : j.pitch)) {
                    cp_async16(&in[r][16 * q], from);
                } else {
                    for (int b = 0; b < 16 && cx + b < W; ++b) in[r][16 * q + b] = from[b];
                }
            }
        }
    } else {
        for (int i = tid; i < kFastInH * kInStride; i += kFastThreads) {
            const int r = i / kInStride, c = i - r * kInStride;
            const int gy = min(max(y0 - 4 + r, 0), H - 1), gx = min(max(x0 - 16 + c, 0), W - 1);
            in[r][c] = j.image[static_cast<std::size_t>(gy) * j.pitch + gx];
        }
    }
}

// FAST-9 + strict 3x3 NMS, persistent: each block takes 64x64 tiles of
// every job of the launch from a device queue (`*queue`, zero at launch; tile
// t of `total` is looked up through the source's kFastKind entries), while
// the next tile's bytes are copied into the other half of a double buffer.
// The jobs of the current and the next tile sit in shared memory. Per tile:
//   1. the compass test on the tile plus a 1-pixel ring, 8 positions per
//      thread in 16-bit lanes; groups with a survivor are listed;
//   2. the groups are expanded into one list of survivor positions, scored
//      on full warps (every other position scores 0);
//   3. each survivor of the tile inside the 31-pixel edge margin that is a
//      strict 3x3 maximum goes into the job's maxima list as
//      (score << 32) | raster index (one atomic per warp), its score into the
//      tile's histogram, which is added to the job's at the end of the tile.
// No maxima map and no blur are written.
template <class Src>
__global__ __launch_bounds__(kFastThreads, kFastCtasPerSm) void fast_kernel(const __grid_constant__ Src src,
                                                                          std::uint32_t* queue, int total) {
    wait_for_previous();
    static_assert(sizeof(DetectJob) % 16 == 0, "jobs are copied in 16-byte chunks");
    __shared__ __align__(16) std::uint8_t in[2][kFastInH][kInStride];
    __shared__ __align__(16) std::uint8_t sc[kFastScH][kScStride];
    __shared__ std::uint32_t cand[kFastScH * kScGroups];
    __shared__ std::uint16_t pos[kFastScH * kFastScW];  // survivor positions r * kScStride + c
    __shared__ std::uint32_t hist[256];
    __shared__ DetectJob jobs[2];  // jobs of the tiles in in[0] and in[1] (kept here, not in registers)
    __shared__ int locals[2];
    __shared__ int n_cand, n_pos, next;
    __shared__ int ahead_tile;          // with a block map: the tile after `next`, taken from the queue
    __shared__ std::uint32_t ahead_entry;  // and its block-map entry (job << 16 | tile within the job)
    const int tid = threadIdx.x, lane = tid & 31;
    // With a block map, total is capped by the map; the job of the tile after
    // the current one is copied into shared memory asynchronously while the
    // current tile is tested, and the queue index and map entry of the tile
    // after that are fetched a tile ahead, so no thread waits on the lookup.
    std::uint32_t one = 1u, minus = ~0u;
    asm("" : "+r"(one), "+r"(minus));  // see Compass
    const std::uint32_t* map = fast_map(src);
    if (map) total = min(total, fast_map_tiles(src));
    hist[tid] = 0;
    if (tid == 0) {
        n_cand = 0;
        n_pos = 0;
        next = static_cast<int>(atomicAdd(queue, 1u));
        if (next < total && !src.find(next, kFastKind, &jobs[0], &locals[0])) next = total;
        if (map) {
            const int t = static_cast<int>(atomicAdd(queue, 1u));
            ahead_tile = t;
            if (t < total) cp_async4(&ahead_entry, map + t);
        }
    }
    __syncthreads();
    int tile = next, buf = 0;
    if (tile < total) stage_fast_tile(jobs[0], locals[0], in[0]);
    cp_async_wait_all();
    __syncthreads();
    while (tile < total) {
        const DetectJob& j = jobs[buf];
        const int local = locals[buf];
        const int W = j.width, H = j.height;
        const int2 org = fast_origin(j, local);
        const int y0 = org.y, x0 = org.x;
        std::uint8_t (*cur)[kInStride] = in[buf];
        int ahead = total;  // thread 0 with a block map: the queue index of the tile after next
        if (tid == 0) {
            if (map) {
                const int t = ahead_tile;
                next = t;
                if (t < total) {
                    const std::uint32_t e = ahead_entry;
                    locals[buf ^ 1] = static_cast<int>(e & 0xffffu);
                    const auto* g = reinterpret_cast<const char*>(fast_jobs(src) + (e >> 16));
                    auto* d = reinterpret_cast<char*>(&jobs[buf ^ 1]);
#pragma unroll
                    for (int k = 0; k < static_cast<int>(sizeof(DetectJob) / 16); ++k) cp_async16(d + 16 * k, g + 16 * k);
                    ahead = static_cast<int>(atomicAdd(queue, 1u));
                }
            } else {
                int t = static_cast<int>(atomicAdd(queue, 1u));
                if (t < total && !src.find(t, kFastKind, &jobs[buf ^ 1], &locals[buf ^ 1])) t = total;
                next = t;
            }
        }
        // 1. compass test: thread (q, rb) takes positions 8q .. 8q+7 of rows rb,
        // rb + 28, rb + 56; groups with a survivor are listed as
        // (group << 8 | survivor bits)
        const Compass compass{one, minus, 0x80008000u - static_cast<std::uint32_t>(j.threshold + 1) * 0x00010001u};
        {
            constexpr int kRowSets = 256 / kScGroups;  // 28
            const int q = tid % kScGroups, rb = tid / kScGroups, c = 8 * q;
            unsigned colmask = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int gx = x0 - 1 - kScRing + c + k;
                if (c + k >= kScRing && c + k < kScRing + kFastScW && gx >= 3 && gx < W - 3) colmask |= 1u << k;
            }
            for (int it = 0; it < (kFastScH + kRowSets - 1) / kRowSets; ++it) {  // same trip count everywhere
                const int r = rb + it * kRowSets;
                unsigned bits = 0;
                if (rb < kRowSets && r < kFastScH) {
                    *reinterpret_cast<uint2*>(&sc[r][c]) = make_uint2(0u, 0u);
                    const int gy = y0 - 1 + r;
                    if (colmask && gy >= 3 && gy < H - 3) {
                        const int w = 2 * q + kInOff / 4;  // the first centres' word
                        const auto* mid = reinterpret_cast<const std::uint32_t*>(&cur[r + 3][0]) + w;
                        const auto* bot = reinterpret_cast<const std::uint32_t*>(&cur[r + 6][0]) + w;
                        const auto* top = reinterpret_cast<const std::uint32_t*>(&cur[r][0]) + w;
                        const std::uint32_t m0 = mid[-1], m1 = mid[0], m2 = mid[1], m3 = mid[2];
                        const unsigned b0 = compass_bits(m0, m1, m2, bot[0], top[0], compass);
                        const unsigned b1 = compass_bits(m1, m2, m3, bot[1], top[1], compass);
                        bits = ((b0 & 0xfu) | (b1 << 4)) & colmask;
                    }
                }
                const unsigned m = __ballot_sync(0xffffffffu, bits != 0);
                int base = 0;
                if (lane == 0 && m) base = atomicAdd(&n_cand, __popc(m));
                base = __shfl_sync(0xffffffffu, base, 0);
                if (bits)
                    cand[base + __popc(m & ((1u << lane) - 1u))] = (static_cast<unsigned>(r * kScGroups + q) << 8) | bits;
            }
        }
        if (tid == 0 && map) cp_async_wait_all();  // the next tile's job
        __syncthreads();
        // the next tile's bytes travel while this one is scored
        const int nt = next;
        if (tid == 0 && map) {
            ahead_tile = ahead;
            if (ahead < total) cp_async4(&ahead_entry, map + ahead);
        }
        if (nt < total) stage_fast_tile(jobs[buf ^ 1], locals[buf ^ 1], in[buf ^ 1]);
        const int nc = n_cand;
        // 2. the survivor groups expanded into one position list (each warp
        // reserves its share with one shared atomic), then scored on full warps
        for (int base = 0; base < nc; base += kFastThreads) {  // block-uniform trip count
            const int i = base + tid;
            unsigned bits = 0;
            int pos0 = 0;
            if (i < nc) {
                const int e = static_cast<int>(cand[i]);
                const int grp = e >> 8, r = grp / kScGroups, c0 = 8 * (grp - r * kScGroups);
                bits = e & 0xffu;
                pos0 = r * kScStride + c0;
            }
            const int cnt = __popc(bits);
            int incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            int first = 0;
            if (lane == 31 && incl) first = atomicAdd(&n_pos, incl);
            first = __shfl_sync(0xffffffffu, first, 31);
            int o = first + incl - cnt;
            for (unsigned b = bits; b; b &= b - 1) pos[o++] = static_cast<std::uint16_t>(pos0 + __ffs(b) - 1);
        }
        __syncthreads();
        const int np = n_pos;
        for (int k = tid; k < np; k += kFastThreads) {
            const int e = pos[k];
            const int r = e / kScStride, c = e - r * kScStride;
            sc[r][c] = static_cast<std::uint8_t>(fast_score(&cur[r + 3][c + kInOff], kInStride, j.threshold));
        }
        __syncthreads();
        // 3. strict 3x3 maxima inside the 31-pixel edge margin: only listed
        // survivors can score above 0, so only they are tested (the ring
        // rows and columns hold neighbours only). Each warp appends its maxima
        // to the job's list with one atomic, and their scores to the tile's
        // histogram.
        for (int k0 = 0; k0 < np; k0 += kFastThreads) {  // block-uniform trip count
            const int k = k0 + tid;
            unsigned v = 0;
            std::uint32_t px = 0;
            if (k < np) {
                const int e = pos[k];
                const int r = e / kScStride, c = e - r * kScStride;
                const int gy = y0 - 1 + r, gx = x0 - 1 - kScRing + c;
                if (r >= 1 && r <= kFastTileH && c >= kScRing + 1 && c <= kScRing + kFastTileW && gy >= kEdge && gy < H - kEdge &&
                    gx >= kEdge && gx < W - kEdge) {
                    const unsigned s0 = sc[r][c];
                    if (s0 && s0 > sc[r - 1][c - 1] && s0 > sc[r - 1][c] && s0 > sc[r - 1][c + 1] &&
                        s0 > sc[r][c - 1] && s0 > sc[r][c + 1] && s0 > sc[r + 1][c - 1] && s0 > sc[r + 1][c] &&
                        s0 > sc[r + 1][c + 1]) {
                        v = s0;
                        px = static_cast<std::uint32_t>(gy) * static_cast<std::uint32_t>(W) + static_cast<std::uint32_t>(gx);
                    }
                }
            }
            const unsigned m = __ballot_sync(0xffffffffu, v != 0);
            if (m) {
                const int leader = __ffs(m) - 1;
                std::uint32_t first = 0;
                if (lane == leader) first = atomicAdd(&j.counters()[kListed], static_cast<std::uint32_t>(__popc(m)));
                first = __shfl_sync(0xffffffffu, first, leader);
                if (v) {
                    const std::uint32_t slot = first + static_cast<std::uint32_t>(__popc(m & ((1u << lane) - 1u)));
                    if (slot < static_cast<std::uint32_t>(j.max_maxima))
                        j.maxima[slot] = (static_cast<std::uint64_t>(v) << 32) | px;
                    atomicAdd(&hist[v], 1u);
                }
            }
        }
        __syncthreads();
        // the tile's histogram into the job's
        if (hist[tid]) {
            atomicAdd(&j.hist[tid], hist[tid]);
            hist[tid] = 0;
        }
        if (tid == 0) {
            n_cand = 0;
            n_pos = 0;
        }
        cp_async_wait_all();
        __syncthreads();
        tile = nt;
        buf ^= 1;
    }
}

// --------------------------------------------------------- 2K selection

// All 256 threads: suffix[s] = number of maxima with score >= s (s >= 1),
// then the unique threshold s with suffix[s] >= cap > suffix[s + 1]; with at
// most cap maxima, everything is kept (threshold 1).
__device__ __forceinline__ SelectParams select_params(const std::uint32_t* hist, std::uint32_t cap,
                                                     std::uint32_t* suffix /*[257] shared*/,
                                                     SelectParams* out /*shared*/) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    __shared__ std::uint32_t warp_total[8];
    const std::uint32_t own = t ? hist[t] : 0u;
    std::uint32_t v = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const std::uint32_t n = __shfl_down_sync(0xffffffffu, v, o);
        if (lane + o < 32) v += n;
    }
    if (lane == 0) warp_total[warp] = v;
    __syncthreads();
    for (int w = warp + 1; w < 8; ++w) v += warp_total[w];
    suffix[t] = v;
    if (t == 0) suffix[256] = 0;
    __syncthreads();
    const std::uint32_t total = suffix[1];
    if (total <= cap) {
        if (t == 1) *out = SelectParams{1u, total - own, own, total};
    } else if (t >= 1 && suffix[t] >= cap && suffix[t + 1] < cap) {
        *out = SelectParams{static_cast<std::uint32_t>(t), suffix[t + 1], cap - suffix[t + 1], cap};
    }
    __syncthreads();
    return *out;
}

// The list of the maxima at the selection threshold (their raster indices), in
// the entries of the maxima list that its n maxima leave over.
struct TieList {
    std::uint32_t* at;
    std::uint32_t room;
};

__device__ __forceinline__ TieList tie_list(const DetectJob& j, std::uint32_t n) {
    const std::uint32_t left = static_cast<std::uint32_t>(j.max_maxima) - n;  // two ties fit an entry
    return {reinterpret_cast<std::uint32_t*>(j.maxima + n), min(left, kTieCap / 2u) * 2u};
}

// The first `p.ties` maxima at the threshold score in raster order, when they
// cannot all be kept (the reference's raster-order scatter of the first ties,
// src/s2_s3/s2.cu:182-235), by the 256 threads of one block, into keys[above,
// selected). The listed ties are walked, or the maxima list when the ties
// outgrew their list (then an entry counts only with the threshold's score).
// A few ties are ranked against each other; more go through a
// most-significant-digit radix select of the p.ties-th smallest raster index.
__device__ __forceinline__ void pick_ties(const DetectJob& j, const SelectParams& p, std::uint32_t listed,
                                          const TieList& list) {
    __shared__ __align__(16) std::uint32_t buf[kTieRank];  // staged ties, or the 256 radix bins
    __shared__ std::uint32_t pick[2];        // digit, maxima before it
    __shared__ std::uint32_t written;
    const std::uint32_t T = p.threshold, total = j.hist[T];
    const int t = threadIdx.x;
    if (total <= kTieRank && total <= list.room) {
        const int n = static_cast<int>(total), padded = (n + 3) / 4 * 4;
        for (int i = t; i < padded; i += 256) buf[i] = i < n ? __ldcg(list.at + i) : 0xffffffffu;
        __syncthreads();
        for (int i = t; i < n; i += 256) {
            const std::uint32_t px = buf[i];
            std::uint32_t rank = 0;
            for (int k = 0; k < padded; k += 4) {
                const uint4 q = *reinterpret_cast<const uint4*>(buf + k);
                rank += (q.x < px) + (q.y < px) + (q.z < px) + (q.w < px);
            }
            if (rank < p.ties) j.keys[p.above + rank] = px;
        }
        return;
    }
    const bool own = total <= list.room;
    const std::uint32_t n = own ? total : listed;
    const auto entry = [&](std::uint32_t i, std::uint32_t& px) {  // whether entry i is a tie
        if (own) {
            px = __ldcg(list.at + i);
            return true;
        }
        const std::uint64_t e = j.maxima[i];
        px = static_cast<std::uint32_t>(e);
        return static_cast<std::uint32_t>(e >> 32) == T;
    };
    std::uint32_t prefix = 0, need = p.ties;
    for (int shift = 24; shift >= 0; shift -= 8) {
        const std::uint32_t high = shift == 24 ? 0u : (0xffffffffu << (shift + 8));
        buf[t] = 0;
        __syncthreads();
#pragma unroll 4
        for (std::uint32_t i = t; i < n; i += 256) {
            std::uint32_t px;
            if (entry(i, px) && (px & high) == prefix) atomicAdd(&buf[(px >> shift) & 255u], 1u);
        }
        __syncthreads();
        if (t == 0) {
            std::uint32_t run = 0, d = 0;
            while (d < 255 && run + buf[d] < need) run += buf[d++];
            pick[0] = d;
            pick[1] = run;
            written = 0;
        }
        __syncthreads();
        prefix |= pick[0] << shift;
        need -= pick[1];
        __syncthreads();
    }
    const int lane = t & 31;
    const unsigned below = (1u << lane) - 1u;
    for (std::uint32_t i0 = 0; i0 < n; i0 += 256) {  // block-uniform
        const std::uint32_t i = i0 + t;
        std::uint32_t px = 0;
        const bool keep = i < n && entry(i, px) && px <= prefix;
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        std::uint32_t b = 0;
        if (lane == 0 && m) b = atomicAdd(&written, static_cast<std::uint32_t>(__popc(m)));
        b = __shfl_sync(0xffffffffu, b, 0) + __popc(m & below);
        if (keep && b < p.ties) j.keys[p.above + b] = px;
    }
}

// Pre-selection over a job's maxima list: every block of the job derives the
// same threshold from the histogram; block 0 publishes the parameters and
// the keypoint count min(selected, K). The maxima above the threshold go to
// keys[0, above), and when every maximum at the threshold is kept (selected
// below the cap, or the cap falls exactly on a score boundary) those go to
// keys[above, selected); otherwise they are listed, and the job's last block
// to finish picks the first of them in raster order. The order inside each
// range is not the raster order: the keys are sorted later by (response,
// raster index), which no order of equal sets changes.
//
// Latency-bound. The ties used to be picked by a kernel of one block per job
// that walked the whole maxima list five times (512x512, 8 layers: 15 us; 4K:
// 60 us); the list of the ties alone is some hundred entries, and picking
// them in the last block saves a launch. Select and ties together, 512x512:
// 18.5 -> 7 us, 4K: 67 -> 23 us.
template <class Src>
__global__ __launch_bounds__(256) void select_kernel(const __grid_constant__ Src src, RankTotals* totals) {
    wait_for_previous();
    __shared__ std::uint32_t suffix[257];
    __shared__ SelectParams sp;
    __shared__ bool last;
    DetectJob j;
    int local;
    if (!src.find(blockIdx.x, kSelectKind, &j, &local)) return;
    const SelectParams p = select_params(j.hist, static_cast<std::uint32_t>(j.candidates), suffix, &sp);
    if (local == 0 && threadIdx.x == 0) {
        *j.params = p;
        *j.count = static_cast<int>(min(p.selected, static_cast<std::uint32_t>(j.max_keypoints)));
        if (totals && p.selected <= kSortCap) {
            atomicAdd(&totals->squares, static_cast<unsigned long long>(p.selected) * p.selected);
            atomicAdd(&totals->sum, p.selected);
            atomicMax(&totals->largest, p.selected);
        }
    }
    const bool all_ties = p.ties == j.hist[p.threshold];
    std::uint32_t* ctr = j.counters();
    const std::uint32_t n = min(ctr[kListed], static_cast<std::uint32_t>(j.max_maxima));
    const TieList list = tie_list(j, n);
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    // ties go behind the keys above the threshold, or to their list
    std::uint32_t* const tie_count = &ctr[kTies];
    const std::uint32_t stride = static_cast<std::uint32_t>(j.select_blocks) * 256u;
    for (std::uint32_t i0 = static_cast<std::uint32_t>(local) * 256u; i0 < n; i0 += stride) {  // block-uniform
        const std::uint32_t i = i0 + threadIdx.x;
        bool above = false, tie = false;
        std::uint32_t px = 0;
        if (i < n) {
            const std::uint64_t e = j.maxima[i];
            const auto score = static_cast<std::uint32_t>(e >> 32);
            px = static_cast<std::uint32_t>(e);
            above = score > p.threshold;
            tie = score == p.threshold;
        }
        const unsigned ma = __ballot_sync(0xffffffffu, above), mt = __ballot_sync(0xffffffffu, tie);
        std::uint32_t ba = 0, bt = 0;
        if (lane == 0) {
            if (ma) ba = atomicAdd(&ctr[kAboveWritten], static_cast<std::uint32_t>(__popc(ma)));
            if (mt) bt = atomicAdd(tie_count, static_cast<std::uint32_t>(__popc(mt)));
        }
        ba = __shfl_sync(0xffffffffu, ba, 0) + __popc(ma & below);
        bt = __shfl_sync(0xffffffffu, bt, 0) + __popc(mt & below);
        if (above && ba < p.above) j.keys[ba] = px;  // always true when list and histogram agree
        if (tie && all_ties && bt < p.ties) j.keys[p.above + bt] = px;
        if (tie && !all_ties && bt < list.room) list.at[bt] = px;
    }
    if (all_ties || p.selected == 0) return;
    __threadfence();  // this block's list entries, before it counts as done
    __syncthreads();
    if (threadIdx.x == 0)
        last = atomicAdd(&j.hist[kSelectDoneBin], 1u) == static_cast<std::uint32_t>(j.select_blocks) - 1u;
    __syncthreads();
    if (!last) return;
    __threadfence();
    pick_ties(j, p, n, list);
}

// ------------------------------------------------------------- Harris

// Monotone float -> unsigned order (never 0 for a finite input).
__device__ __forceinline__ std::uint32_t order_bits(float v) {
    const std::uint32_t u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_order_bits(std::uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// (1 / (4 * 7 * 255))^4 evaluated in float32, as ORB's HarrisResponses does.
constexpr float kHarrisScale4 = 0x1.bb9da2p-52f;

// Harris response over the 7x7 window of 3x3 Sobel gradients centred on
// (x, y): integer sums, then det - k * trace^2 in float32 with every product
// and sum rounded separately. The gradients are separable: ix is the
// horizontal difference of the columns' 1-2-1 sums, iy the vertical
// difference of the rows' 1-2-1 sums. With 4-byte aligned rows (words) a
// row's nine bytes come from three word loads, else from nine byte loads: the
// lanes of a warp look at scattered patches, so the loads are what the kernel
// takes its time for (64 pairs at 512x512: 37 -> 20 us; one image: 9 -> 6 us).
__device__ __forceinline__ float harris_response(const std::uint8_t* img, int pitch, int x, int y, float k, bool words) {
    const int x0 = x - 4, off = words ? x0 & 3 : 0;
    const std::uint8_t* base = img + static_cast<std::size_t>(y - 4) * pitch + (x0 - off);
    std::uint32_t raw[9][3];  // bytes 0..8 of each row
    if (words) {
#pragma unroll
        for (int r = 0; r < 9; ++r)
#pragma unroll
            for (int w = 0; w < 3; ++w)
                raw[r][w] = __ldg(reinterpret_cast<const unsigned int*>(base + static_cast<std::size_t>(r) * pitch) + w);
#pragma unroll
        for (int r = 0; r < 9; ++r) {
            raw[r][0] = __funnelshift_r(raw[r][0], raw[r][1], 8 * off);
            raw[r][1] = __funnelshift_r(raw[r][1], raw[r][2], 8 * off);
            raw[r][2] >>= 8 * off;
        }
    } else {
#pragma unroll
        for (int r = 0; r < 9; ++r) {
            const std::uint8_t* q = base + static_cast<std::size_t>(r) * pitch;
            raw[r][0] = q[0] | q[1] << 8 | q[2] << 16 | static_cast<std::uint32_t>(q[3]) << 24;
            raw[r][1] = q[4] | q[5] << 8 | q[6] << 16 | static_cast<std::uint32_t>(q[7]) << 24;
            raw[r][2] = q[8];
        }
    }
    int p[3][9], h[3][7];  // the last three rows: bytes, 1-2-1 sums
    int a = 0, b = 0, cc = 0;
#pragma unroll
    for (int r = 0; r < 9; ++r) {
#pragma unroll
        for (int c = 0; c < 9; ++c) p[r % 3][c] = static_cast<int>((raw[r][c / 4] >> (8 * (c % 4))) & 0xffu);
#pragma unroll
        for (int c = 0; c < 7; ++c) h[r % 3][c] = p[r % 3][c] + 2 * p[r % 3][c + 1] + p[r % 3][c + 2];
        if (r < 2) continue;
        int v[9];
#pragma unroll
        for (int c = 0; c < 9; ++c) v[c] = p[(r + 1) % 3][c] + 2 * p[(r + 2) % 3][c] + p[r % 3][c];
#pragma unroll
        for (int c = 0; c < 7; ++c) {
            const int ix = v[c + 2] - v[c], iy = h[r % 3][c] - h[(r + 1) % 3][c];
            a += ix * ix;
            b += iy * iy;
            cc += ix * iy;
        }
    }
    const float fa = static_cast<float>(a), fb = static_cast<float>(b), fc = static_cast<float>(cc);
    const float trace = __fadd_rn(fa, fb);
    const float det = __fsub_rn(__fmul_rn(fa, fb), __fmul_rn(fc, fc));
    const float penalty = __fmul_rn(__fmul_rn(k, trace), trace);
    return __fmul_rn(__fsub_rn(det, penalty), kHarrisScale4);
}

// Replaces each pre-selected pixel index by its sort key
// (order_bits(response) << 32) | (0xffffffff - index): larger key = better,
// equal responses prefer the smaller raster index.
template <class Src>
__global__ __launch_bounds__(kHarrisThreads) void harris_kernel(const __grid_constant__ Src src) {
    wait_for_previous();
    DetectJob j;
    int local;
    if (!src.find(blockIdx.x, kHarrisKind, &j, &local)) return;
    const int slot = local * kHarrisThreads + threadIdx.x;
    if (slot >= j.candidates) return;
    const std::uint32_t selected = j.params->selected;
    if (static_cast<std::uint32_t>(slot) >= selected) return;
    const auto px = static_cast<std::uint32_t>(j.keys[slot]);
    const int x = static_cast<int>(px % static_cast<std::uint32_t>(j.width));
    const int y = static_cast<int>(px / static_cast<std::uint32_t>(j.width));
    const bool words = ((reinterpret_cast<std::uintptr_t>(j.image) | static_cast<std::uintptr_t>(j.pitch)) & 3) == 0;
    const float r = harris_response(j.image, j.pitch, x, y, j.harris_k, words);
    j.keys[slot] = (static_cast<std::uint64_t>(order_bits(r)) << 32) | (0xffffffffu - px);
}

// ------------------------------------------------------------- top-K

// Flags the blur tiles within kSampleRadius of the keypoint at (x, y) (the
// describe kernel samples nothing else of the blurred layer around it) and
// lists each newly flagged tile once for blur_tiles_kernel.
__device__ __forceinline__ void mark_blur_tiles(const DetectJob& j, int x, int y) {
    const int tx0 = max(x - kSampleRadius, 0) / kBlurTileW, tx1 = min(x + kSampleRadius, j.width - 1) / kBlurTileW;
    const int ty0 = max(y - kSampleRadius, 0) / kBlurTileH, ty1 = min(y + kSampleRadius, j.height - 1) / kBlurTileH;
    const int tiles_x = (j.width + kBlurTileW - 1) / kBlurTileW;
    for (int ty = ty0; ty <= ty1; ++ty)
        for (int tx = tx0; tx <= tx1; ++tx) {
            const int t = ty * tiles_x + tx;
            if (atomicExch(&j.blur_marks[t], 1u) == 0u)
                j.blur_list[atomicAdd(j.blur_count, 1u)] = make_uint2(static_cast<unsigned>(j.job), static_cast<unsigned>(t));
        }
}

__device__ __forceinline__ void write_keypoint(const DetectJob& j, int rank, std::uint64_t key) {
    const std::uint32_t px = 0xffffffffu - static_cast<std::uint32_t>(key);
    const std::uint32_t x = px % static_cast<std::uint32_t>(j.width), y = px / static_cast<std::uint32_t>(j.width);
    j.x[rank] = static_cast<float>(x);
    j.y[rank] = static_cast<float>(y);
    if (j.response) j.response[rank] = from_order_bits(static_cast<std::uint32_t>(key >> 32));
    if (j.blur_marks) mark_blur_tiles(j, static_cast<int>(x), static_cast<int>(y));
}

// Time of ranking `jobs` jobs with `sum` keys in all, `squares` comparisons and
// `largest` keys in one, by that of sorting them. Measured in ns: the ranking takes 8 us,
// 4 ns per 32 keys and a rate, 4 comparisons per ps in slices of 32 keys and 6.4 in
// wide ones; the sort 6 us and 10.2 ns per key of the largest job, padded to a power of
// two, for every wave of blocks (one per job, two per SM). 800x600 noise, K keypoints
// at one level, ranked and sorted: 4 pairs, K = 1000 18 and 26 us, 4000 102 and 90, 8000
// 315 and 186; 8 pairs, K = 2000 57 and 45; 16 pairs, K = 4000 312 and 90.
__host__ __device__ inline float rank_cost(float squares, float sum, int largest, int jobs, bool wide) {
    int keys = 1024;
    while (keys < largest) keys *= 2;
    const float rank = 8000.0f + 0.125f * sum + 4.0f * jobs + (wide ? 0.156e-3f : 0.25e-3f) * squares;
    return rank / (6000.0f + 10.2f * keys * ((jobs + 2 * 148 - 1) / (2 * 148)));
}

// Where the capacities leave it open (totals not null), the kernels of both ways are
// launched and decide by the keys that are there: the idle one costs 3 to 5 us.
struct RankChoice {
    const RankTotals* totals;
    int jobs;
    bool wide;
    __device__ __forceinline__ bool ranked() const {
        return rank_cost(static_cast<float>(totals->squares), static_cast<float>(totals->sum), static_cast<int>(totals->largest), jobs, wide) <= 1.0f;
    }
};

// One block per job: bitonic sort (descending) of up to kSortCap keys in
// shared memory, then the first min(K, selected) become the keypoints. Bound by
// instruction issue and barriers on the SMs that have a block; sort_threads has the
// batched blocks' sizes (30 mixed pairs, K up to 8000, want 1024 threads: 83 us, 86
// with 512, 100 with 256, and 106 in two launches that divide the jobs).
template <class Src, int kThreads>
__global__ __launch_bounds__(kThreads) void sort_topk_kernel(const __grid_constant__ Src src, RankChoice choice) {
    wait_for_previous();
    if (choice.totals && choice.ranked()) return;
    extern __shared__ std::uint64_t sk[];
    DetectJob j;
    int local;
    if (!src.find(blockIdx.x, kSortKind, &j, &local)) return;
    const int n = static_cast<int>(j.params->selected);
    if (n > kSortCap || n == 0) return;
    int N = kSortChunk;  // at least one 64-key chunk (zero keys pad and sort last)
    while (N < n) N <<= 1;
    for (int i = threadIdx.x; i < N; i += kThreads) sk[i] = i < n ? j.keys[i] : 0ull;
    __syncthreads();
    // Bitonic network, keys unique: a compare-exchange of i < q = i + s puts
    // the larger key first where (i & k) == 0 (those runs end up descending).
    // Exchanges closer than 64 keys run in registers, a warp holding keys
    // c*64 + lane and c*64 + lane + 32 of chunk c; wider ones in shared memory.
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto chunk_pass = [&](int k_lo, int k_hi, int s_top) {
        for (int c = warp; c < N / kSortChunk; c += kThreads / 32) {
            const int e0 = c * kSortChunk + lane;
            std::uint64_t v0 = sk[e0], v1 = sk[e0 + 32];
            for (int k = k_lo; k <= k_hi; k <<= 1) {
                for (int s = min(k >> 1, s_top); s > 0; s >>= 1) {
                    if (s == 32) {  // v0 (key e0) is the lower of the pair
                        const bool desc = (e0 & k) == 0;
                        const std::uint64_t hi = v0 > v1 ? v0 : v1, lo = v0 > v1 ? v1 : v0;
                        v0 = desc ? hi : lo;
                        v1 = desc ? lo : hi;
                    } else {
                        const bool lower = (lane & s) == 0;
                        const std::uint64_t p0 = __shfl_xor_sync(0xffffffffu, v0, s);
                        const std::uint64_t p1 = __shfl_xor_sync(0xffffffffu, v1, s);
                        const bool keep_hi0 = lower == ((e0 & k) == 0);
                        const bool keep_hi1 = lower == (((e0 + 32) & k) == 0);
                        v0 = keep_hi0 ? (v0 > p0 ? v0 : p0) : (v0 > p0 ? p0 : v0);
                        v1 = keep_hi1 ? (v1 > p1 ? v1 : p1) : (v1 > p1 ? p1 : v1);
                    }
                }
            }
            sk[e0] = v0;
            sk[e0 + 32] = v1;
        }
        __syncthreads();
    };
    chunk_pass(2, kSortChunk, kSortChunk / 2);  // runs up to 64 keys: registers only
    for (int k = 2 * kSortChunk; k <= N; k <<= 1) {
        for (int s = k >> 1; s >= kSortChunk; s >>= 1) {
            for (int t = threadIdx.x; t < (N >> 1); t += kThreads) {
                const int i = 2 * t - (t & (s - 1));  // the t-th key without bit s
                const int q = i + s;
                const std::uint64_t a = sk[i], b = sk[q];
                const bool descending = (i & k) == 0;
                if (descending ? (a < b) : (a > b)) { sk[i] = b; sk[q] = a; }
            }
            __syncthreads();
        }
        chunk_pass(k, k, kSortChunk / 2);
    }
    const int limit = min(n, j.max_keypoints);
    for (int i = threadIdx.x; i < limit; i += kThreads) write_keypoint(j, i, sk[i]);
}

// Top-K by counting: the rank of a key is the number of larger keys (keys are
// unique). A block ranks kRankKeys keys, one per lane; its 16 warps share the
// comparisons with every key of the job, staged kRankTile at a time. Jobs with
// more than `below` keys are left to rank_wide_kernel. Counting n keys costs n^2
// comparisons, but spread over the whole chip, where the sort has one block
// per job: one 512x512 image, 8 layers: 12 -> 6 us; 4K, K = 8000: 46 -> 14 us.
// rank_pays draws the line between the two.
template <class Src>
__global__ __launch_bounds__(kRankThreads) void rank_topk_kernel(const __grid_constant__ Src src, int below, RankChoice choice) {
    wait_for_previous();
    if (choice.totals && !choice.ranked()) return;
    __shared__ __align__(16) std::uint64_t tile[kRankTile];
    __shared__ int part[kRankThreads / 32][kRankKeys];
    static_assert(kRankKeys == 32, "one key per lane");
    DetectJob j;
    int local;
    if (!src.find(blockIdx.x / kRankPer, kHarrisKind, &j, &local)) return;
    const int first = (local * kRankPer + static_cast<int>(blockIdx.x % kRankPer)) * kRankKeys;
    const int n = static_cast<int>(j.params->selected);
    if (n > below || first >= n) return;  // block-uniform
    const int t = threadIdx.x, k = t % kRankKeys, slice = t / kRankKeys;
    const int slot = first + k;
    const std::uint64_t key = slot < n ? j.keys[slot] : ~0ull;
    int rank = 0;
    for (int b0 = 0; b0 < n; b0 += kRankTile) {
        if (b0) __syncthreads();
#pragma unroll
        for (int i = t; i < kRankTile; i += kRankThreads) tile[i] = b0 + i < n ? j.keys[b0 + i] : 0ull;
        __syncthreads();
        const int m = min(kRankTile, (n - b0 + 1) / 2 * 2);  // keys past n are 0, never larger
#pragma unroll 4
        for (int i = 2 * slice; i < m; i += 2 * (kRankThreads / 32)) {
            const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(tile + i);
            rank += (q.x > key) + (q.y > key);
        }
    }
    part[slice][k] = rank;
    __syncthreads();
    if (slice == 0 && slot < n) {
#pragma unroll
        for (int v = 1; v < kRankThreads / 32; ++v) rank += part[v][k];
        if (rank < j.max_keypoints) write_keypoint(j, rank, key);
    }
}

// The same with kRankGrid blocks, each of which looks for the harris blocks that
// hold keys among its share of the launch with all its threads, and kRankWide keys per
// lane, for two kinds of launches:
// - of batches that would take more than kRankDirect blocks above. A slice without
//   keys, whose job lookup is a chain of loads, costs 2.2 ns as a block of its own:
//   32 pairs of 800x600, K = 20000, some 400 keypoints each, sort and rank 210 us
//   so, 54 here (an image's own launch has no lookup: 0.4 ns);
// - of jobs of very many keys, which fill the chip's block slots all the same: a key
//   read from shared memory is compared four times. 64 jobs of 40000 keys: 18.3 ms
//   above, 14.4 here; one of 400000: 27.1 and 22.0.
constexpr int kRankDirect = 12 * 148, kRankGrid = 8 * 148, kRankWide = 4;
constexpr int kRankMany = 1 << 17;  // an image's jobs of more keys are ranked here
static_assert(kRankKeys * kRankWide == kHarrisThreads, "a block ranks a harris block's keys");

template <class Src>
__global__ __launch_bounds__(kRankThreads, 3) void rank_wide_kernel(const __grid_constant__ Src src, int above, int below, int harris_blocks,
                                                                     RankChoice choice) {
    wait_for_previous();
    if (choice.totals && !choice.ranked()) return;
    __shared__ __align__(16) std::uint64_t tile[kRankTile];
    __shared__ int part[kRankThreads / 32][kHarrisThreads];
    __shared__ int found[kRankThreads], n_found;
    const int t = threadIdx.x, lane = t % 32, warp = t / 32, grid = gridDim.x;
    // first key and key count of harris block b; false when it has nothing to rank
    const auto lookup = [&](int b, DetectJob* j, int* first, int* n) {
        int local;
        if (!src.find(b, kHarrisKind, j, &local)) return false;
        *first = local * kHarrisThreads;
        *n = static_cast<int>(j->params->selected);
        return *n > above && *n <= below && *first < *n;
    };
    for (int base = blockIdx.x; base < harris_blocks; base += grid * kRankThreads) {
        if (t == 0) n_found = 0;
        __syncthreads();
        {
            const long long mine = base + static_cast<long long>(grid) * t;
            DetectJob j;
            int first, n;
            if (mine < harris_blocks && lookup(static_cast<int>(mine), &j, &first, &n))
                found[atomicAdd(&n_found, 1)] = static_cast<int>(mine);
        }
        __syncthreads();
        const int todo = n_found;
        for (int f = 0; f < todo; ++f) {
            DetectJob j;
            int first, n;
            lookup(found[f], &j, &first, &n);
            std::uint64_t key[kRankWide];
            int rank[kRankWide];
#pragma unroll
            for (int p = 0; p < kRankWide; ++p) {
                const int slot = first + 32 * p + lane;
                key[p] = slot < n ? j.keys[slot] : ~0ull;
                rank[p] = 0;
            }
            for (int b0 = 0; b0 < n; b0 += kRankTile) {
                if (b0 || f) __syncthreads();
#pragma unroll
                for (int i = t; i < kRankTile; i += kRankThreads) tile[i] = b0 + i < n ? j.keys[b0 + i] : 0ull;
                __syncthreads();
                const int m = min(kRankTile, (n - b0 + 1) / 2 * 2);  // keys past n are 0, never larger
#pragma unroll 4
                for (int i = 2 * warp; i < m; i += 2 * (kRankThreads / 32)) {
                    const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(tile + i);
#pragma unroll
                    for (int p = 0; p < kRankWide; ++p) rank[p] += (q.x > key[p]) + (q.y > key[p]);
                }
            }
#pragma unroll
            for (int p = 0; p < kRankWide; ++p) part[warp][32 * p + lane] = rank[p];
            __syncthreads();
            if (t < kHarrisThreads && first + t < n) {
                int r = 0;
#pragma unroll
                for (int v = 0; v < kRankThreads / 32; ++v) r += part[v][t];
                if (r < j.max_keypoints) write_keypoint(j, r, j.keys[first + t]);
            }
        }
        __syncthreads();  // found, n_found and part are read before they are written again
    }
}

// Launches the ranking of one image's jobs of up to max_candidates candidates, in
// all `harris_blocks` blocks of them, through go(kernel, blocks, arguments after
// the source ...). Returns the launches.
template <class Src, class Go> inline int launch_rank(int harris_blocks, int max_candidates, Go go) {
    const bool many = max_candidates > kRankMany;
    go(rank_topk_kernel<Src>, harris_blocks * kRankPer, many ? kRankMany : INT_MAX, RankChoice{});
    if (many) go(rank_wide_kernel<Src>, kRankGrid, kRankMany, INT_MAX, harris_blocks, RankChoice{});
    return many ? 2 : 1;
}

// ------------------------------------------------------ pyramid layers

// Source index and 8-bit weight of the right neighbour for destination
// index v of a src -> dst linear resize: f = (v + 0.5) * scale - 0.5 in
// double with scale = 1 / (dst / src), weight rint((f - floor f) * 256).
// Indices left of the source (every index when src == 1) read pixel 0 with
// weight 0, indices past the last interval read pixel src - 1 with weight 0.
__host__ __device__ inline double linear_exact_scale(int src, int dst) {
    return 1.0 / (static_cast<double>(dst) / static_cast<double>(src));
}

__device__ __forceinline__ int2 linear_exact_tap(int v, int src, double scale) {
    const double f = scale * (static_cast<double>(v) + 0.5) - 0.5;
    const double fl = floor(f);
    if (src == 1 || fl < 0.0) return make_int2(0, 0);
    if (fl >= static_cast<double>(src - 1)) return make_int2(src - 1, 0);
    return make_int2(static_cast<int>(fl), static_cast<int>(rint((f - fl) * 256.0)));
}

// One block = one tile of 128 x kTileH (16..128) layer pixels:
//   1. per-column and per-row taps in shared memory (double, as above);
//   2. the tile's exact source window (rows of the first and last row taps,
//      columns from the first column tap rounded down to 16 bytes) is
//      staged in shared memory with 16-byte asynchronous copies;
//   3. warp w makes the band of kTileH / 8 consecutive rows starting at row
//      w * kTileH / 8, lane l columns 4l .. 4l + 3:
//        h(r, c) = src[r][c0] * (256 - wx) + src[r][c0 + 1] * wx   (< 2^16)
//        out = (h(ra, c) * (256 - wy) + h(rb, c) * wy + 2^15) >> 16,
//      the integer form of the 8-bit fixed-point horizontal pass followed by
//      the vertical pass with one final rounding. A source row's h comes from
//      two byte permutes of aligned shared-memory words and one 16x8-bit dot
//      product per column; it is kept when the next output row's upper source
//      row is this one's lower (four of five rows at 1.2). The rounded sum is
//      below 2^24, so out is its byte 2 and the four bytes are gathered by
//      permutes. A whole warp shares one band, so its lanes take the same
//      branches.
// Blocks whose source is not 16-byte aligned or whose window exceeds the
// staging buffer (layer ratios above about 1.45), and lanes whose bytes do
// not fit two 8-byte pools, read the source bytes from global memory per
// output row instead, with the same result.
// Bound by issue slots and the latency of job, tap and window loads. Layers
// 1..7 of 128 images of 512x512: 133 us walking every source row with the
// output rows tested inside (34 instructions per pixel), 104 with this loop
// (21), 96 with six blocks per SM instead of five; 30 mixed pairs: 442, 328
// and 303 us. A third of that is made per tile (taps, window, selectors), so
// tiles of 128 rows take 94 and 268 us.
constexpr int kRawStride = 208;  // bytes of a staged source row: 13 chunks of 16
template <int kTileH> __host__ __device__ constexpr int resize_raw_rows() { return kTileH * 3 / 2 + 6; }

// A source byte read in place. Read-only loads may pass the stores to the other layer
// (2 pairs of 799x601, ratio 2, 4 layers: layers 22 us with them, 25 with plain ones),
// but a chained launch may overlap the one that writes its source (launch_chained).
template <class Src> __device__ __forceinline__ std::uint32_t source_byte(const std::uint8_t* p) {
    if constexpr (std::is_same_v<Src, JobTable<ResizeJob>>) return __ldg(p);
    else return *p;
}

// Four output pixels of one row from the h of its upper and lower source rows.
__device__ __forceinline__ std::uint32_t resize_quad(const std::uint32_t (&ha)[4], const std::uint32_t (&hb)[4], std::uint32_t wy) {
    std::uint32_t v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = hb[k] * wy + (ha[k] * (256u - wy) + 32768u);
    return __byte_perm(__byte_perm(v[0], v[1], 0x0062), __byte_perm(v[2], v[3], 0x0062), 0x5410);
}

template <class Src, int kTileH>
__global__ __launch_bounds__(256, kTileH > kResizeTileH ? 5 : 6) void resize_kernel(const __grid_constant__ Src src, int kind) {
    static_assert(kTileH >= 16 && kTileH <= kResizeTallH && kResizeTileW + kTileH <= 256 && kTileH % 16 == 0, "resize tile height");
    constexpr int kBand = kTileH / 8, kRows = resize_raw_rows<kTileH>();
    __shared__ int2 xtap[kResizeTileW];
    __shared__ int2 ytap[kTileH];
    __shared__ __align__(16) std::uint8_t raw[kRows][kRawStride];
    ResizeJob j;
    int local;
    if (!src.find(blockIdx.x, kind, &j, &local)) {
        wait_for_previous();
        return;
    }
    const int y0 = (local / j.tiles_x) * kTileH;
    const int x0 = (local % j.tiles_x) * kResizeTileW;
    const int t = threadIdx.x;
    // 1. taps (columns and rows past the layer edge repeat the last one)
    if (t < kResizeTileW) xtap[t] = linear_exact_tap(min(x0 + t, j.width - 1), j.src_width, j.scale_x);
    else if (t < kResizeTileW + kTileH)
        ytap[t - kResizeTileW] = linear_exact_tap(min(y0 + t - kResizeTileW, j.height - 1), j.src_height, j.scale_y);
    wait_for_previous();  // what stands above depends on the job alone
    __syncthreads();
    // 2. source window: rows ry0 .. ry1, 16-byte chunks from column rx0
    const int ry0 = ytap[0].x, ry1 = min(ytap[kTileH - 1].x + 1, j.src_height - 1);
    const int rx0 = xtap[0].x & ~15, rx1 = min(xtap[kResizeTileW - 1].x + 1, j.src_width - 1);
    const int nrow = ry1 - ry0 + 1, nchunk = (rx1 - rx0) / 16 + 1;
    const bool staged = ((reinterpret_cast<std::uintptr_t>(j.src) | static_cast<std::uintptr_t>(j.src_pitch)) & 15) == 0 &&
                        nrow <= kRows && nchunk <= kRawStride / 16;  // block-uniform
    if (staged) {
        const int q = t & 15, col = rx0 + 16 * q;
        if (q < nchunk) {
            // rows whose 16 bytes may be read: within the pitch, on the last image row within the width
            const int whole = col + 16 <= j.src_width ? nrow : col + 16 <= j.src_pitch ? min(nrow, j.src_height - 1 - ry0) : 0;
            int r = t >> 4;
            const std::uint8_t* p = j.src + static_cast<std::size_t>(ry0 + r) * j.src_pitch + col;
            const std::size_t step = static_cast<std::size_t>(j.src_pitch) * 16;
            for (; r < whole; r += 16, p += step) cp_async16(&raw[r][16 * q], p);
            for (; r < nrow; r += 16, p += step) {
#pragma unroll
                for (int k = 0; k < 16; ++k) raw[r][16 * q + k] = col + k < j.src_width ? p[k] : 0;
            }
        }
        cp_async_wait_all();
    }
    __syncthreads();
    // 3. bands
    const int r0 = (t >> 5) * kBand;
    const int r_end = r0 + min(kBand, j.height - y0 - r0);  // band rows inside the layer
    const int c = 4 * (t & 31), x = x0 + c;
    if (r_end <= r0 || x >= j.width) return;
    int2 tx[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) tx[k] = xtap[c + k];
    std::uint32_t wx[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) wx[k] = (256u - tx[k].y) | (static_cast<std::uint32_t>(tx[k].y) << 16);
    const int nx = min(4, j.width - x);
    std::uint8_t* dst = j.dst + static_cast<std::size_t>(y0 + r0) * j.pitch + x;
    const bool word_store = nx == 4 && ((reinterpret_cast<std::uintptr_t>(j.dst) | static_cast<std::uintptr_t>(j.pitch)) & 3) == 0;
    auto emit = [&](std::uint32_t quad) {
        if (word_store) {
            *reinterpret_cast<std::uint32_t*>(dst) = quad;
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < nx) dst[k] = static_cast<std::uint8_t>(quad >> (8 * k));
        }
        dst += j.pitch;
    };
    // the lane's bytes: pool A = 8 bytes at column `base` (columns 0, 1),
    // pool B = 8 bytes at base + 4 * kb (columns 2, 3)
    const int base = tx[0].x & ~3;
    const int o0 = tx[0].x - base, o1 = tx[1].x - base;
    const int kb = (tx[2].x - base) >> 2;
    const int o2 = tx[2].x - base - 4 * kb, o3 = tx[3].x - base - 4 * kb;
    const bool fits = staged && o1 + 1 <= 7 && o3 + 1 <= 7 && base - rx0 + 4 * kb + 8 <= kRawStride;
    if (!fits) {
        int xb[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) xb[k] = min(tx[k].x + 1, j.src_width - 1);
        for (int rr = r0; rr < r_end; ++rr) {
            const int2 ty = ytap[rr];
            const std::uint8_t* A = j.src + static_cast<std::size_t>(ty.x) * j.src_pitch;
            const std::uint8_t* B = j.src + static_cast<std::size_t>(min(ty.x + 1, j.src_height - 1)) * j.src_pitch;
            std::uint32_t ha[4], hb[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const std::uint32_t wa = source_byte<Src>(A + tx[k].x) | (source_byte<Src>(A + xb[k]) << 8);
                const std::uint32_t wb = source_byte<Src>(B + tx[k].x) | (source_byte<Src>(B + xb[k]) << 8);
                ha[k] = __dp2a_lo(wx[k], wa, 0u);
                hb[k] = __dp2a_lo(wx[k], wb, 0u);
            }
            emit(resize_quad(ha, hb, static_cast<std::uint32_t>(ty.y)));
        }
        return;
    }
    const std::uint32_t sel_a = static_cast<std::uint32_t>(o0 | ((o0 + 1) << 4) | (o1 << 8) | ((o1 + 1) << 12));
    const std::uint32_t sel_b = static_cast<std::uint32_t>(o2 | ((o2 + 1) << 4) | (o3 << 8) | ((o3 + 1) << 12));
    const std::uint8_t* lane_bytes = &raw[0][0] + (base - rx0);
    const int last = j.src_height - 1 - ry0;
    auto row_h = [&](int row, std::uint32_t (&h)[4]) {  // h of staged row `row`
        const auto* w = reinterpret_cast<const std::uint32_t*>(lane_bytes + row * kRawStride);
        const std::uint32_t pool_a = __byte_perm(w[0], w[1], sel_a), pool_b = __byte_perm(w[kb], w[kb + 1], sel_b);
        h[0] = __dp2a_lo(wx[0], pool_a, 0u);
        h[1] = __dp2a_hi(wx[1], pool_a, 0u);
        h[2] = __dp2a_lo(wx[2], pool_b, 0u);
        h[3] = __dp2a_hi(wx[3], pool_b, 0u);
    };
    // two rows per step, the h of the lower source rows changing places
    std::uint32_t h0[4], h1[4];
    int have = -1;  // staged row whose h is in h0
    for (int rr = r0; rr < r_end; rr += 2) {
        const int2 ta = ytap[rr];
        const int ua = ta.x - ry0, la = min(ua + 1, last);
        if (have != ua) row_h(ua, h0);
        row_h(la, h1);
        emit(resize_quad(h0, h1, static_cast<std::uint32_t>(ta.y)));
        if (rr + 1 == r_end) break;
        const int2 tb = ytap[rr + 1];
        const int ub = tb.x - ry0, lb = min(ub + 1, last);
        if (la != ub) row_h(ub, h1);
        row_h(lb, h0);
        emit(resize_quad(h1, h0, static_cast<std::uint32_t>(tb.y)));
        have = lb;
    }
}

// ------------------------------------------------------------- S3 blur

// The S3 blur of 64x64 tiles: those listed by the keypoint writers (on-demand
// blur of the pyramid and batched paths, kPacked), or, without a list, the
// first all_tiles tiles of job 0 (the per-image S3 call, scalar). Per output
// the taps are summed first to last, then rounded half-to-even. Persistent:
// block b takes list entries b, b + gridDim.x, ... (the list is complete when
// the kernel starts). A tile is staged with its reflect-101 halo: 16-byte
// copies for 16-byte aligned images, reflected byte loads otherwise. The
// per-image call used to have a kernel with byte-wise loads of its own
// (640x480: 14 -> 5 us).
// Bound by issue slots and shared-memory wavefronts alike (66 and 64 % busy; the
// packed sums alone would take 45 %). 128 images of 512x512 with 8 layers: 160 us
// with the job, the origin and the halo made by every thread and 2x4 outputs
// per item of either pass; 143 with the descriptions, 8x2 and 4x4 items; 133
// with 5 blocks per SM instead of 6 (spills at 40 registers); 129 with the
// swizzled rows, the list read ahead and one row item per thread. 4 blocks: 127.
// 30 mixed pairs: 411 -> 330 us.
// One thread for each item of the rows pass (35 row pairs x 8 groups of 8
// columns = 280); the columns pass has 256, and the ninth warp makes the next
// but one tile's description beside it.
constexpr int kBlurThreads = 288;
constexpr int kBlurInH = kBlurTileH + 8;  // staged rows of a blur tile: rows y0-4 .. y0+kBlurTileH+3 (halo 3, rounded to 4)

// What the threads of a block need of a tile, in shared memory: one thread
// reads the list, the job and makes the origin, a tile ahead of the staging.
struct BlurTile {
    const std::uint8_t* image;
    std::uint8_t* blurred;  // the tile's first pixel
    int width, height, pitch, blur_pitch;
    int x0, y0;
    bool aligned;  // 16-byte copies and word-wise halo columns
    bool whole;    // 64x64 pixels inside the image, stored as words
};

template <class Src>
__device__ __forceinline__ void blur_tile_at(const Src& src, uint2 e, BlurTile* t) {
    const DescribeJob j = src.at(static_cast<int>(e.x));
    const int tiles_x = (j.width + kBlurTileW - 1) / kBlurTileW;
    const int y0 = (static_cast<int>(e.y) / tiles_x) * kBlurTileH, x0 = (static_cast<int>(e.y) % tiles_x) * kBlurTileW;
    t->image = j.image;
    t->blurred = j.blurred + static_cast<std::size_t>(y0) * j.blur_pitch + x0;
    t->width = j.width;
    t->height = j.height;
    t->pitch = j.pitch;
    t->blur_pitch = j.blur_pitch;
    t->x0 = x0;
    t->y0 = y0;
    // three columns are mirrored about the first and the last one
    t->aligned = ((reinterpret_cast<std::uintptr_t>(j.image) | static_cast<std::uintptr_t>(j.pitch)) & 15) == 0 && j.width >= 4;
    t->whole = x0 + kBlurTileW <= j.width && y0 + kBlurTileH <= j.height &&
               ((reinterpret_cast<std::uintptr_t>(j.blurred) | static_cast<std::uintptr_t>(j.blur_pitch)) & 3) == 0;
}

// Asynchronous staging of a blur tile of a 16-byte aligned image: row r of
// `in` is image row reflect101(y0 - 4 + r) (the reflected halo rows are whole
// image rows), byte c is column x0 - 16 + c. Chunks inside a row's pitch
// (inside the width on the last image row) are 16-byte copies, a chunk
// straddling the end of the last row is copied byte by byte; the reflected
// halo columns are filled by blur_fix_columns once the copies are complete.
// A thread has the same chunk of rows r and r + 48 in every tile.
__device__ __forceinline__ void blur_stage_async(const BlurTile& t, std::uint8_t (*in)[kInStride]) {
    constexpr int kChunks = kInStride / 16, kRows = kBlurThreads / kChunks;  // 6, 48
    const int r0 = static_cast<int>(threadIdx.x) / kChunks, q = static_cast<int>(threadIdx.x) - r0 * kChunks;
    const int cx = t.x0 - 16 + 16 * q;
    if (cx < 0 || cx >= t.width) return;
    for (int r = r0; r < kBlurInH; r += kRows) {
        const int gy = reflect101(t.y0 - 4 + r, t.height);
        const std::uint8_t* p = t.image + static_cast<std::size_t>(gy) * t.pitch + cx;
        if (cx + 16 <= (gy == t.height - 1 ? t.width : t.pitch)) {
            cp_async16(&in[r][16 * q], p);
        } else {
            for (int b = 0; b < 16 && cx + b < t.width; ++b) in[r][16 * q + b] = p[b];
        }
    }
}

// Whether the 7x7 blur of the tile at x0 reads columns outside the image.
__device__ __forceinline__ bool blur_needs_columns(int x0, int W) { return x0 < 3 || x0 + kBlurTileW + 3 > W; }

// Reflect-101 halo columns of a staged tile of an image of 4 columns or more:
// column -k is column k, column W - 1 + k is column W - 1 - k (k = 1..3),
// copied inside `in` (sources are interior columns, never written here).
__device__ __forceinline__ void blur_fix_columns(int x0, int W, std::uint8_t (*in)[kInStride]) {
    const int tid = threadIdx.x;
    static_assert(kBlurInH <= 128, "a side per half of the block");
    if (tid < kBlurInH) {
        auto* w = reinterpret_cast<std::uint32_t*>(in[tid]);
        if (x0 < 3) w[3] = __byte_perm(w[4], 0u, 0x1230);  // bytes 13..15 are bytes 19..17
    } else if (tid >= 128 && tid < 128 + kBlurInH && x0 + kBlurTileW + 3 > W) {
        std::uint8_t* b = &in[tid - 128][16 + W - x0];  // column W
        const std::uint8_t c0 = b[-2], c1 = b[-3], c2 = b[-4];
        b[0] = c0;
        b[1] = c1;
        b[2] = c2;
    }
}

// Where the four sums of columns 4c .. 4c+3 of a row stand: a thread of the
// rows pass writes 2q and 2q+1, one of the columns pass reads one, and eight
// lanes in turn meet no bank twice.
__device__ __forceinline__ int blur_quad(int c) { return c ^ (c >> 3); }

constexpr int kBlurCtasPerSm = 5;     // resident blur blocks per SM; the persistent grid is 148 x this
constexpr int kBlurMaxCtasPerSm = 6;  // the largest grid a tuning may ask for
template <class Src, bool kPacked>
__global__ __launch_bounds__(kBlurThreads, kBlurCtasPerSm) void blur_tiles_kernel(const __grid_constant__ Src src, const uint2* list,
                                                            const std::uint32_t* count, int all_tiles) {
    wait_for_previous();
    __shared__ __align__(16) std::uint8_t in2[2][kBlurInH][kInStride];  // rows y0-4 .., columns x0-16 ..
    __shared__ __align__(16) float rows[kBlurTileH + 6][kBlurTileW];
    __shared__ BlurTile info[3];
    __shared__ std::size_t row_at[kBlurInH];
    __shared__ int col_at[kInStride];
    const int tid = threadIdx.x;
    const int n = list ? static_cast<int>(*count) : all_tiles;
    const int grid = gridDim.x;
    const auto tile_at = [&](int i) { return list ? list[i] : make_uint2(0u, static_cast<unsigned>(i)); };
    if (static_cast<int>(blockIdx.x) >= n) return;
    if (tid == 0) blur_tile_at(src, tile_at(blockIdx.x), &info[0]);
    if (tid == 32 && static_cast<int>(blockIdx.x) + grid < n) blur_tile_at(src, tile_at(blockIdx.x + grid), &info[1]);
    __syncthreads();
    // tiles of aligned images are copied asynchronously, the next one while this one is blurred
    if (info[0].aligned) blur_stage_async(info[0], in2[0]);
    const auto entry_at = [&](int i) { return i < n ? tile_at(i) : make_uint2(0u, 0u); };
    uint2 ahead = entry_at(blockIdx.x + 2 * grid);
    int buf = 0, slot = 0;
    for (int i = blockIdx.x; i < n; i += grid, buf ^= 1) {
        std::uint8_t (*in)[kInStride] = in2[buf];
        const BlurTile& t = info[slot];
        const int next = slot == 2 ? 0 : slot + 1, after = next == 2 ? 0 : next + 1;
        if (!t.aligned) {  // unaligned image: reflected byte loads
            if (tid < kBlurInH) row_at[tid] = static_cast<std::size_t>(reflect101(t.y0 - 4 + tid, t.height)) * t.pitch;
            else if (tid < kBlurInH + kInStride) col_at[tid - kBlurInH] = reflect101(t.x0 - 16 + (tid - kBlurInH), t.width);
            __syncthreads();
            for (int k = tid; k < kBlurInH * (kInStride / 4); k += kBlurThreads) {
                const int r = k / (kInStride / 4), b = 4 * (k - r * (kInStride / 4));
                const std::uint8_t* row = t.image + row_at[r];
                *reinterpret_cast<std::uint32_t*>(&in[r][b]) =
                    static_cast<std::uint32_t>(row[col_at[b]]) | (static_cast<std::uint32_t>(row[col_at[b + 1]]) << 8) |
                    (static_cast<std::uint32_t>(row[col_at[b + 2]]) << 16) |
                    (static_cast<std::uint32_t>(row[col_at[b + 3]]) << 24);
            }
        }
        cp_async_wait_all();
        __syncthreads();  // also: everyone is done with the tile before
        if (t.aligned && blur_needs_columns(t.x0, t.width)) {
            blur_fix_columns(t.x0, t.width, in);
            __syncthreads();
        }
        if (i + grid < n && info[next].aligned) blur_stage_async(info[next], in2[buf ^ 1]);
        const int out_rows = min(kBlurTileH, t.height - t.y0);
        // rows pass: image rows y0-3 .., two rows x 8 outputs per item
        static_assert((kBlurTileH + 6) % 2 == 0 && (kBlurTileH + 6) / 2 * (kBlurTileW / 8) <= kBlurThreads,
                      "rows pass takes row pairs, one item per thread");
        if (tid < (out_rows + 7) / 2 * (kBlurTileW / 8)) {
            const int rr = 2 * (tid / (kBlurTileW / 8)), q = tid % (kBlurTileW / 8);
            const auto* ra = reinterpret_cast<const std::uint32_t*>(&in[rr + 1][0]) + 2 * q + 3;  // bytes 8q+12 .. 8q+27
            const auto* rb = reinterpret_cast<const std::uint32_t*>(&in[rr + 2][0]) + 2 * q + 3;
            const uint2 a12 = *reinterpret_cast<const uint2*>(ra + 1), b12 = *reinterpret_cast<const uint2*>(rb + 1);
            const std::uint32_t wa[4] = {ra[0], a12.x, a12.y, ra[3]}, wb[4] = {rb[0], b12.x, b12.y, rb[3]};
            // output 8q+k reads halo columns 8q+k+1 .. 8q+k+7, tap t on column
            // 8q+k+1+t; lane x holds row rr, lane y row rr + 1. The columns
            // stream in once and every output adds its taps in order (0 + a
            // nonnegative product is the product).
            float2 out[8], before;
#pragma unroll
            for (int m = 1; m <= 14; ++m) {
                const float2 xm = byte_pair(wa[m >> 2], wb[m >> 2], m & 3);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int tap = m - 1 - k;
                    if (tap == 1) out[k] = first_taps<kPacked>(before, xm);
                    else if (tap > 1 && tap < 7) out[k] = next_tap<kPacked>(out[k], tap, xm);
                }
                before = xm;
            }
            auto* o = reinterpret_cast<float4*>(&rows[rr][0]) + blur_quad(2 * q);
            auto* o1 = reinterpret_cast<float4*>(&rows[rr][0]) + blur_quad(2 * q + 1);
            constexpr int kNextRow = kBlurTileW / 4;
            o[0] = make_float4(out[0].x, out[1].x, out[2].x, out[3].x);
            o1[0] = make_float4(out[4].x, out[5].x, out[6].x, out[7].x);
            o[kNextRow] = make_float4(out[0].y, out[1].y, out[2].y, out[3].y);
            o1[kNextRow] = make_float4(out[4].y, out[5].y, out[6].y, out[7].y);
        }
        __syncthreads();
        // columns pass: a thread has rows 4p .. 4p+3 and columns 4q .. 4q+3
        static_assert(kBlurTileH / 4 * (kBlurTileW / 4) == 256, "columns pass: one 4x4 block per thread");
        const int row = 4 * (tid / (kBlurTileW / 4)), col = 4 * (tid % (kBlurTileW / 4));
        if (tid >= 256) {
            if (tid == kBlurThreads - 1 && i + 2 * grid < n) {
                blur_tile_at(src, ahead, &info[after]);
                ahead = entry_at(i + 3 * grid);
            }
        } else if (row < out_rows) {
            const auto* quads = reinterpret_cast<const float4*>(&rows[row][0]) + blur_quad(col / 4);
            float2 lo[4], hi[4], bl, bh;
#pragma unroll
            for (int r = 0; r < 10; ++r) {
                const float4 v = quads[r * (kBlurTileW / 4)];
                const float2 vl = make_float2(v.x, v.y), vh = make_float2(v.z, v.w);
#pragma unroll
                for (int o = 0; o < 4; ++o) {
                    const int tap = r - o;
                    if (tap == 1) {
                        lo[o] = first_taps<kPacked>(bl, vl);
                        hi[o] = first_taps<kPacked>(bh, vh);
                    } else if (tap > 1 && tap < 7) {
                        lo[o] = next_tap<kPacked>(lo[o], tap, vl);
                        hi[o] = next_tap<kPacked>(hi[o], tap, vh);
                    }
                }
                bl = vl;
                bh = vh;
            }
            std::uint8_t* dst = t.blurred + static_cast<std::size_t>(row) * t.blur_pitch + col;
            const int nx = t.whole ? 4 : t.width - t.x0 - col;
#pragma unroll
            for (int o = 0; o < 4; ++o, dst += t.blur_pitch) {
                const std::uint32_t packed = pack_bytes(round_pair(lo[o]), round_pair(hi[o]));
                if (t.whole || (nx >= 4 && row + o < out_rows && (reinterpret_cast<std::uintptr_t>(dst) & 3) == 0)) {
                    *reinterpret_cast<std::uint32_t*>(dst) = packed;
                } else if (row + o < out_rows) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (k < nx) dst[k] = static_cast<std::uint8_t>(packed >> (8 * k));
                }
            }
        }
        slot = next;
    }
}

// ---------------------------------------------------------- S3 describe

// Global (not __constant__): each thread reads a different pair, which the
// constant cache would serialise.
__device__ const int4 kOrbPattern[256] = {
#include "orb_pattern_31.inc"
};

// Half-widths of the rows of the radius-15 orientation disc, v = 0..15:
// 15 15 15 15 14 14 14 13 13 12 11 10 9 8 6 3 (one byte per row).
__device__ __forceinline__ int disc_half_width(int v) {
    constexpr unsigned long long lo = 0x0d0e0e0e0f0f0f0full;  // rows 0..7, row 0 in the low byte
    constexpr unsigned long long hi = 0x030608090a0b0c0dull;  // rows 8..15, row 8 in the low byte
    return v < 8 ? static_cast<int>((lo >> (8 * v)) & 0xff)
                 : static_cast<int>((hi >> (8 * (v - 8))) & 0xff);
}

// Weights of the orientation disc for 4-byte loads: the disc's 31 rows are
// read as 9 aligned words each (279 (row, word) slots, slot = 9 row + word),
// the first word starting a = (x - 15) & 3 bytes left of column x - 15. Byte
// k of word w is column u = 4w + k - a - 15 of row v = row - 15; inside the
// disc its weights are u (for m10) and v (for m01) as signed bytes, outside 0.
constexpr int kDiscSlots = 288;  // 9 rounds of 32 lanes over the 279 slots
struct alignas(16) DiscTable {
    uint2 w[4][kDiscSlots];  // [a][slot]: weights for m10, for m01
};
constexpr DiscTable disc_table() {
    constexpr int half[16] = {15, 15, 15, 15, 14, 14, 14, 13, 13, 12, 11, 10, 9, 8, 6, 3};
    DiscTable t{};
    for (int a = 0; a < 4; ++a)
        for (int slot = 0; slot < 279; ++slot) {
            const int v = slot / 9 - 15, word = slot % 9;
            unsigned int wu = 0, wv = 0;
            for (int k = 0; k < 4; ++k) {
                const int u = 4 * word + k - a - 15;
                if ((u < 0 ? -u : u) <= half[v < 0 ? -v : v]) {
                    wu |= (static_cast<unsigned int>(u) & 0xffu) << (8 * k);
                    wv |= (static_cast<unsigned int>(v) & 0xffu) << (8 * k);
                }
            }
            t.w[a][slot].x = wu;
            t.w[a][slot].y = wv;
        }
    return t;
}
__device__ const DiscTable kDiscTable = disc_table();

// acc + sum of the four unsigned bytes of `bytes` times the four signed bytes of `w`
__device__ __forceinline__ int dot4_us(std::uint32_t bytes, std::uint32_t w, int acc) {
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(bytes), "r"(w), "r"(acc));
    return d;
}

// cv::fastAtan2 in degrees [0, 360): odd polynomial of the smaller/larger
// magnitude ratio, every step rounded in float32.
__device__ __forceinline__ float fast_atan2_deg(float y, float x) {
    const float ax = fabsf(x), ay = fabsf(y);
    const bool wide = ax >= ay;
    const float eps = 0x1p-52f;
    const float t = wide ? __fdiv_rn(ay, __fadd_rn(ax, eps)) : __fdiv_rn(ax, __fadd_rn(ay, eps));
    const float t2 = __fmul_rn(t, t);
    float p = __fadd_rn(__fmul_rn(-0x1.4515b2p+1f, t2), 0x1.1d3f7ep+3f);
    p = __fadd_rn(__fmul_rn(p, t2), -0x1.2aaddcp+4f);
    p = __fadd_rn(__fmul_rn(p, t2), 0x1.ca44dep+5f);
    p = __fmul_rn(p, t);
    float a = wide ? p : __fsub_rn(90.0f, p);
    if (x < 0) a = __fsub_rn(180.0f, a);
    if (y < 0) a = __fsub_rn(360.0f, a);
    return a;
}

// The blurred byte at the pattern point rotated by (a, b) = (cos, sin),
// rounded half-to-even by adding 1.5 * 2^23 (as in round_pair): the float's
// bits are kRoundBits + the integer, and `bias`, -kRoundBits * (stride + 1)
// modulo 2^32, takes the offset out of row * stride + column.
constexpr std::uint32_t kRoundBits = 0x4B400000u;
__device__ __forceinline__ int rotated_sample(const std::uint8_t* centre, std::uint32_t stride, std::uint32_t bias,
                                              float fx, float fy, float a, float b) {
    const float cx = __fadd_rn(__fsub_rn(__fmul_rn(fx, a), __fmul_rn(fy, b)), 12582912.0f);
    const float cy = __fadd_rn(__fadd_rn(__fmul_rn(fx, b), __fmul_rn(fy, a)), 12582912.0f);
    return centre[static_cast<int>(__float_as_uint(cy) * stride + __float_as_uint(cx) + bias)];
}

// A warp describes up to keys / kDescWarps keypoints (the block stages the pattern
// and the disc weights once): first the intensity-centroid moments over the
// radius-15 disc of the unblurred image of each (kept on lane r for the r-th),
// then all their angles at once, one per lane (float fastAtan2, cos/sin
// evaluated in double then rounded to float), then, two keypoints per pass over
// the pattern, lane l packs pattern pairs 8l..8l+7 of the blurred image into
// descriptor byte l. An angle takes about 130 instructions, a quarter of a
// keypoint's when each is computed alone; a pattern entry is 4 of the shared
// memory wavefronts that bound the kernel.
// 5 blocks per SM (48 registers): at 8 the two-keypoint pass spills (194 us for
// 64 pairs of 512x512, K = 2000), at 6 and 4 it takes 172 and 178; one keypoint
// at a time from moments to samples took 192, this 166.
template <class Src>
__global__ __launch_bounds__(kDescWarps * 32, kDescCtasPerSm) void describe_kernel(const __grid_constant__ Src src, int keys) {
    __shared__ float4 pat[8][32];  // pat[k][l] = pair 8l + k as floats (x0, y0, x1, y1)
    __shared__ DiscTable disc;
    DescribeJob j;
    int local;
    if (!src.find(blockIdx.x, kDescKind, &j, &local)) {
        wait_for_previous();
        return;
    }
    // word loads of the disc need 4-byte aligned rows (block-uniform)
    const bool words = ((reinterpret_cast<std::uintptr_t>(j.image) | static_cast<std::uintptr_t>(j.pitch)) & 3) == 0;
    const auto stage = [&] {  // depends on the job and on constants alone
        const int p = threadIdx.x;  // 256 threads, one pattern pair each
        const int4 q = kOrbPattern[p];
        pat[p & 7][p >> 3] = make_float4(static_cast<float>(q.x), static_cast<float>(q.y), static_cast<float>(q.z),
                                         static_cast<float>(q.w));
        if (words)
            for (int e = threadIdx.x; e < static_cast<int>(sizeof(DiscTable) / 16); e += kDescWarps * 32)
                reinterpret_cast<uint4*>(&disc)[e] = __ldg(reinterpret_cast<const uint4*>(&kDiscTable) + e);
    };
    // a chained launch stages beside the launch before it, a batch's block once it
    // knows that it has keypoints (32 pairs, K = 20000, 2100 there: 183 -> 161 us; 64
    // pairs at 512x512, K = 2000, 1460 there: 165 -> 166)
    constexpr bool kChained = !std::is_same_v<Src, JobTable<DescribeJob>>;
    if constexpr (kChained) stage();
    wait_for_previous();
    // The grid covers the capacity; blocks past the keypoint count leave now.
    const int count = min(*j.count, j.capacity);
    int base = 0;  // first output row of this layer
    if (j.level_counts) {
        if (local == 0 && threadIdx.x == 0) atomicAdd(j.out_count, count);
        for (int m = 0; m < j.level; ++m) base += j.level_counts[m];
    }
    // keypoints per block: `keys` follows from the capacities; where fewer are there,
    // as few as keep the launch in one wave if every job has this one's, with blocks
    // enough for all. 1279x717, K = 60000, some 4000 there: S3 40 us by `keys`, 15 so;
    // this kernel, 800x600: 4 pairs, K = 8000, 2100 there 43 and 32 us; 32 pairs at 8
    // layers, K = 1000, 350 there 51 and 50 (54 where the chip is only to be filled).
    int per = keys;
    if (keys > kDescWarps && count < j.capacity) {
        const int blocks = (j.capacity + keys - 1) / keys;
        per = kDescWarps;
        const int most = 148 * kDescCtasPerSm / src.count();
        while (per < keys && (per * blocks < count || per * most < count)) per *= 2;
    }
    if (local * per >= count) return;
    if constexpr (!kChained) stage();
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int pitch = j.pitch, blur_pitch = j.blur_pitch;
    const int first = local * per + (threadIdx.x >> 5);  // the warp's r-th keypoint is first + r * kDescWarps
    const int rounds = min(per / kDescWarps, (count - first + kDescWarps - 1) / kDescWarps);
    if (rounds <= 0) return;
    // keypoint r on lane r: position (x = -1: too near the edge), moments, then cos and sin
    int x = -1, y = 0;
    if (lane < rounds) {
        const int index = first + lane * kDescWarps;
        const float fx = j.x[index], fy = j.y[index];
        x = __float2int_rn(fx);
        y = __float2int_rn(fy);
        if (j.level_counts) {
            j.out_x[base + index] = __fmul_rn(fx, j.scale);
            j.out_y[base + index] = __fmul_rn(fy, j.scale);
            if (j.out_response) j.out_response[base + index] = j.response[index];
        }
        if (x < kEdge || x >= j.width - kEdge || y < kEdge || y >= j.height - kEdge) x = -1;
    }
    int m10 = 0, m01 = 0;
    for (int r = 0; r < rounds; ++r) {
        const int cx = __shfl_sync(0xffffffffu, x, r), cy = __shfl_sync(0xffffffffu, y, r);
        if (cx < 0) continue;
        // Moments as exact integer sums over the disc. With aligned rows each
        // lane takes slots lane, lane + 32, ... of the disc's words (four
        // pixels per load, weighted by two byte dot products); otherwise lane
        // l owns column u = l - 15 and walks the 31 rows.
        int s10 = 0, s01 = 0;
        if (words) {
            const int xs = cx - 15, a = xs & 3;
            const std::uint8_t* top = j.image + static_cast<std::size_t>(cy - 15) * pitch + (xs - a);
#pragma unroll
            for (int k = 0; k < kDiscSlots / 32; ++k) {
                const int slot = 32 * k + lane;
                if (slot < 279) {
                    const int row = (slot * 57) >> 9, word = slot - 9 * row;  // slot / 9 for slot < 288
                    const std::uint32_t d =
                        __ldg(reinterpret_cast<const unsigned int*>(top + static_cast<std::size_t>(row) * pitch + 4 * word));
                    const uint2 w = disc.w[a][slot];
                    s10 = dot4_us(d, w.x, s10);
                    s01 = dot4_us(d, w.y, s01);
                }
            }
        } else {
            const int u = lane - 15, au = u < 0 ? -u : u;
            const std::uint8_t* centre = j.image + static_cast<std::size_t>(cy) * pitch + cx;
#pragma unroll
            for (int v = -15; v <= 15; ++v) {
                const int av = v < 0 ? -v : v;
                if (lane < 31 && au <= disc_half_width(av)) {
                    const int val = centre[v * pitch + u];
                    s10 += u * val;
                    s01 += v * val;
                }
            }
        }
        s10 = __reduce_add_sync(0xffffffffu, s10);
        s01 = __reduce_add_sync(0xffffffffu, s01);
        if (lane == r) {
            m10 = s10;
            m01 = s01;
        }
    }
    float a = 0.0f, b = 0.0f;
    if (lane < rounds) {
        const float angle = __fmul_rn(fast_atan2_deg(static_cast<float>(m01), static_cast<float>(m10)), 0x1.1df46ap-6f);
        // one sincos for both: it equals cos() and sin() bit for bit on every
        // float in [0, 6.2832] (all the angles this can produce; checked
        // exhaustively by tests/test_gpu_sincos.py)
        double sd, cd;
        sincos(static_cast<double>(angle), &sd, &cd);
        a = static_cast<float>(cd);
        b = static_cast<float>(sd);
    }
    const std::uint32_t bias = 0u - kRoundBits * (static_cast<std::uint32_t>(blur_pitch) + 1u);
    const auto centre_of = [&](int r, float& ca, float& cb) {  // the blurred centre; a null edge keypoint
        const int cx = __shfl_sync(0xffffffffu, x, r), cy = __shfl_sync(0xffffffffu, y, r);
        ca = __shfl_sync(0xffffffffu, a, r);
        cb = __shfl_sync(0xffffffffu, b, r);
        return cx < 0 ? nullptr : j.blurred + static_cast<std::size_t>(cy) * blur_pitch + cx;
    };
    const auto write = [&](int r, int value) {
        j.out[static_cast<std::size_t>(base + first + r * kDescWarps) * j.row_stride + lane] = static_cast<std::uint8_t>(value);
    };
    for (int r = 0; r < rounds; r += 2) {
        float a0, b0, a1 = 0.0f, b1 = 0.0f;
        const std::uint8_t* const c0 = centre_of(r, a0, b0);
        const std::uint8_t* const c1 = r + 1 < rounds ? centre_of(r + 1, a1, b1) : nullptr;
        int v0 = 0, v1 = 0;
        if (c0 && c1) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float4 q = pat[k][lane];
                v0 |= (rotated_sample(c0, blur_pitch, bias, q.x, q.y, a0, b0) <
                       rotated_sample(c0, blur_pitch, bias, q.z, q.w, a0, b0)) << k;
                v1 |= (rotated_sample(c1, blur_pitch, bias, q.x, q.y, a1, b1) <
                       rotated_sample(c1, blur_pitch, bias, q.z, q.w, a1, b1)) << k;
            }
        } else if (c0 || c1) {
            const std::uint8_t* const c = c0 ? c0 : c1;
            const float ca = c0 ? a0 : a1, cb = c0 ? b0 : b1;
            int v = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float4 q = pat[k][lane];
                v |= (rotated_sample(c, blur_pitch, bias, q.x, q.y, ca, cb) <
                      rotated_sample(c, blur_pitch, bias, q.z, q.w, ca, cb)) << k;
            }
            (c0 ? v0 : v1) = v;
        }
        write(r, v0);
        if (r + 1 < rounds) write(r + 1, v1);
    }
}

}  // namespace stitch::b200::s2s3
