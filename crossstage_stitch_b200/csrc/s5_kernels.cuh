// S5 kernels: batched MSAC homography (B -> A) with counter-based sampling,
// sm_100a. This translation unit must be compiled with -fmad=false: every
// double product and sum below is rounded on its own, exactly as in the
// reference's solver evaluated without contraction, so results are
// reproducible bit for bit against the CPU oracle.
//
// Reference semantics (file:line in the reference tree):
//   solver math ............ src/s5/s5_math.hpp:98-263
//   prepare / reuse checks .. src/s5/s5.cu:35-83
//   hypothesis generation ... src/s5/s5.cu:85-99
//   MSAC score: 128 lanes, lane l sums terms l, l+128, ... in order, then a
//   halving tree ............ src/s5/s5.cu:101-122
//   winner: valid, then lower loss, then lower hypothesis index
//                             src/s5/s5.cu:124-132
//   finish: serial re-score, refinement accepted on a strictly lower loss,
//   inlier mask r^2 <= tau^2, telemetry, H = D_A^-1 H_s D_B
//                             src/s5/s5.cu:139-212
//
// Layout of the work: a block of the search owns 8 * HPW consecutive
// hypotheses. Their models (fitted here by eight lanes each, or one per thread
// by fit_kernel) are first bounded from below and above in FP32, all of them over
// all matches; the few whose lower bound does not exceed the smallest loss
// known to the pair are then scored exactly, by 128 threads that play the
// reference's 128 virtual lanes, so that the per-lane sums and the reduction
// tree are the reference's, operation for operation.
#pragma once

#include <cfloat>

#include "common.cuh"

namespace stitch::b200::s5k {

struct Pt {
    double ax, ay, bx, by;
};

struct Model {
    double h[9];
    double loss;
    int hypothesis;
    int valid;
};

// Persistent per-pair search state at offset 0 of the S5 workspace.
struct State {
    Model best;  // raw winner over hypotheses [0, evaluated)
    HomographyResult result;
    const float* ax;
    const float* ay;
    const float* bx;
    const float* by;
    const std::int32_t* idx_a;
    const std::int32_t* idx_b;
    const int* count_a;
    const int* count_b;
    const int* count_m;
    int na, nb, nm;
    int cap_a, cap_b, cap_m;
    int evaluated;
    int batch_size;
    double threshold;
    std::uint64_t seed, generation;
    ScaleInfo scale_a, scale_b;
    int status;
    // bits of the smallest upper bound of a loss of this search (a model's
    // FP32 upper bound, its exact loss, or the previous winner's), +inf when
    // none: a pruning bound shared by every block of the pair (nonnegative
    // doubles order like their bits)
    unsigned long long bound;
    float coord_max[4];  // largest |ax|, |ay|, |bx|, |by| of the matches
};

constexpr unsigned long long kInfBits = 0x7ff0000000000000ull;  // +inf

constexpr int kSearchThreads = 256;
constexpr int kSearchWarps = kSearchThreads / 32;
constexpr int kMaxSearchBlocks = 2 * kSmCount;
// matched points staged in shared memory per search block: the batched form
// keeps several blocks per SM, the per-pair form has one or two
constexpr int kStagePoints = 2048;
constexpr int kStagePointsFused = 8192;
constexpr int kPrepareThreads = 1024;
constexpr int kFinishThreads = 256;

// Inputs of one pair, as the caller passed them.
struct PairIO {
    Keypoints a, b;
    Matches m;
    ScaleInfo sa, sb;
    ::stitch::s5::Config c;
    State* state;
    Model* block_best;  // [kMaxSearchBlocks]
    int search_blocks;  // blocks the search launch used for this pair
    int hpw;            // hypotheses per warp
    std::uint8_t* mask;
    double inverse_a[9];  // D_A^-1 (host)
    double d_b[9];        // D_B
    HomographyResult* result_out;  // optional second copy of the result (batched form)
};

template <class Job> struct OneJob {
    Job job;
    __device__ bool find(int block, Job* j, int* local) const {
        *j = job;
        *local = block;
        return true;
    }
};

template <class Job> struct JobTable {
    const Job* jobs;
    const int* prefix;
    int n;
    // optional block -> (job << 16 | block within the job) map: one load
    // instead of a binary search over the prefix
    const std::uint32_t* map = nullptr;
    int map_blocks = 0;
    __device__ bool find(int block, Job* j, int* local) const {
        if (map) {
            if (block >= map_blocks) return false;
            const std::uint32_t e = __ldg(map + block);
            *j = jobs[e >> 16];
            *local = static_cast<int>(e & 0xffffu);
            return true;
        }
        if (block >= prefix[n]) return false;
        int lo = 0, hi = n - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (prefix[mid] <= block) lo = mid; else hi = mid - 1;
        }
        *j = jobs[lo];
        *local = block - prefix[lo];
        return true;
    }
};

// ------------------------------------------------------------ solver math

__device__ __forceinline__ bool fin(double x) { return x == x && x <= DBL_MAX && x >= -DBL_MAX; }

__device__ __forceinline__ void mat3_mul(const double* a, const double* b, double* out) {
    double t[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            t[3 * i + j] = a[3 * i] * b[j] + a[3 * i + 1] * b[j + 3] + a[3 * i + 2] * b[j + 6];
#pragma unroll
    for (int i = 0; i < 9; ++i) out[i] = t[i];
}

// Divide by the largest magnitude; entries finite and |det| > 1e-15.
__device__ __forceinline__ bool h_normalize(double* h) {
    double scale = 0.0;
    for (int i = 0; i < 9; ++i) {
        if (!fin(h[i])) return false;
        if (fabs(h[i]) > scale) scale = fabs(h[i]);
    }
    if (!(scale > 0.0)) return false;
    for (int i = 0; i < 9; ++i) h[i] /= scale;
    const double det = h[0] * (h[4] * h[8] - h[5] * h[7]) - h[1] * (h[3] * h[8] - h[5] * h[6]) +
                       h[2] * (h[3] * h[7] - h[4] * h[6]);
    return fin(det) && fabs(det) > 1e-15;
}

// Squared forward reprojection error of B -> A; DBL_MAX when the projective
// denominator is not finite or too close to zero.
__device__ __forceinline__ double residual2(const double* h, const Pt& p) {
    const double z = h[6] * p.bx + h[7] * p.by + h[8];
    if (!fin(z) || fabs(z) < 1e-15) return DBL_MAX;
    const double dx = (h[0] * p.bx + h[1] * p.by + h[2]) / z - p.ax;
    const double dy = (h[3] * p.bx + h[4] * p.by + h[5]) / z - p.ay;
    const double r = dx * dx + dy * dy;
    return fin(r) ? r : DBL_MAX;
}

// SplitMix64 finaliser on a counter (public-domain algorithm, S. Vigna).
__device__ __forceinline__ std::uint64_t splitmix64(std::uint64_t v) {
    v += 0x9e3779b97f4a7c15ULL;
    v = (v ^ (v >> 30)) * 0xbf58476d1ce4e5b9ULL;
    v = (v ^ (v >> 27)) * 0x94d049bb133111ebULL;
    return v ^ (v >> 31);
}

// Four distinct indices in [0, n): draw k = counter seed ^ (4h + k) mod
// (n - k), stepped past the earlier draws in ascending order.
__device__ __forceinline__ int sample_draw(int n, std::uint64_t seed, int h, int k) {
    return static_cast<int>(splitmix64(seed ^ (static_cast<std::uint64_t>(h) * 4 + k)) %
                            static_cast<std::uint64_t>(n - k));
}

__device__ __forceinline__ void distinct_draws(int* s) {
#pragma unroll
    for (int k = 1; k < 4; ++k) {
        int v = s[k];
        // earlier draws in ascending order
        int lo[3] = {s[0], s[1], s[2]};
        if (k >= 2 && lo[0] > lo[1]) { const int t = lo[0]; lo[0] = lo[1]; lo[1] = t; }
        if (k >= 3) {
            if (lo[1] > lo[2]) { const int t = lo[1]; lo[1] = lo[2]; lo[2] = t; }
            if (lo[0] > lo[1]) { const int t = lo[0]; lo[0] = lo[1]; lo[1] = t; }
        }
#pragma unroll
        for (int i = 0; i < 3; ++i)
            if (i < k && v >= lo[i]) ++v;
        s[k] = v;
    }
}

// No three of the four points (xy of one image) nearly collinear.
__device__ __forceinline__ bool nondegenerate(const double (&p)[4][2]) {
    double scale = 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < i; ++j) {
            const double dx = p[i][0] - p[j][0], dy = p[i][1] - p[j][1];
            const double d = dx * dx + dy * dy;
            if (d > scale) scale = d;
        }
    bool ok = scale > 0.0 && fin(scale);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = i + 1; j < 4; ++j)
#pragma unroll
            for (int k = j + 1; k < 4; ++k) {
                const double x1 = p[j][0] - p[i][0], y1 = p[j][1] - p[i][1];
                const double x2 = p[k][0] - p[i][0], y2 = p[k][1] - p[i][1];
                ok = ok && !(fabs(x1 * y2 - y1 * x2) <= 1e-8 * scale);
            }
    return ok;
}

// Gauss-Jordan step of column C on the 8x9 system of fit4_regs: every index is
// a compile-time constant, and the pivot row swap is a predicated select per
// entry, so the system stays in registers.
template <int C> __device__ __forceinline__ void eliminate(double (&m)[8][9], double max_entry, bool& solvable) {
    constexpr auto idle = [](int r) { return C < 3 && r >= 3 && r < 6; };
    int piv = C;
    double best = fabs(m[C][C]), pv = m[C][C];
#pragma unroll
    for (int r = C + 1; r < 8; ++r)
        if (!idle(r) && fabs(m[r][C]) > best) { best = fabs(m[r][C]); piv = r; pv = m[r][C]; }
    solvable = solvable && fin(pv) && !(fabs(pv) <= 1e-12 * max_entry);
#pragma unroll
    for (int r = C + 1; r < 8; ++r)
#pragma unroll
        for (int jx = C; jx < 9; ++jx)
            if (!idle(r)) {
                const double a = m[C][jx], b = m[r][jx];
                m[C][jx] = r == piv ? b : a;
                m[r][jx] = r == piv ? a : b;
            }
#pragma unroll
    for (int jx = C + 1; jx < 9; ++jx) m[C][jx] /= pv;
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int jx = C + 1; jx < 9; ++jx)
            if (r != C && !idle(r)) m[r][jx] -= m[r][C] * m[C][jx];
}

// Minimal 4-point model on one thread: the normalised normal equations of the
// design rows {x, y, 1, 0, 0, 0, -u x, -u y, u} and {0, 0, 0, x, y, 1, -v x,
// -v y, v}, Gauss-Jordan with partial pivoting, h33 = 1, denormalisation and
// scaling, every value by the reference's operations in its order. Work whose
// result is known beforehand is left out:
// - products with a structural 0 add +-0 to a sum started at +0.0, the matrix
//   is symmetric (products commute) and its (0..2) and (3..5) blocks are equal,
//   so 27 sums and a count stand for the 72 entries;
// - rows 3..5 hold +0.0 in columns 0..2: they are never the pivot there (a
//   pivot of 0 is rejected) and subtracting 0 times a row changes nothing;
// - the pivot column itself is not read again.
// FP64 operations per model about 2700 -> 1450; fit_kernel of 64 pairs x 2000
// hypotheses 63 -> 55 us, and 46 us at three blocks per SM (168 registers).
__device__ __forceinline__ bool fit4_regs(const Pt* p, double* out) {
    double cax = 0, cay = 0, cbx = 0, cby = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) { cax += p[i].ax; cay += p[i].ay; cbx += p[i].bx; cby += p[i].by; }
    cax /= 4; cay /= 4; cbx /= 4; cby /= 4;
    double va = 0.0, vb = 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        va += (p[i].ax - cax) * (p[i].ax - cax) + (p[i].ay - cay) * (p[i].ay - cay);
        vb += (p[i].bx - cbx) * (p[i].bx - cbx) + (p[i].by - cby) * (p[i].by - cby);
    }
    if (!(va > 0.0) || !(vb > 0.0) || !fin(va) || !fin(vb)) return false;
    const double sa = sqrt(2.0 * 4 / va);
    const double sb = sqrt(2.0 * 4 / vb);
    double xx = 0, xy = 0, x1 = 0, yy = 0, y1 = 0;    // x, y block
    double xu[3] = {}, yu[3] = {}, ou[3] = {};        // x, y, 1 times -ux, -uy, u
    double xv[3] = {}, yv[3] = {}, ov[3] = {};        // and -vx, -vy, v
    double s66 = 0, s67 = 0, s68 = 0, s77 = 0, s78 = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double x = (p[i].bx - cbx) * sb, y = (p[i].by - cby) * sb;
        const double u = (p[i].ax - cax) * sa, v = (p[i].ay - cay) * sa;
        const double du[3] = {-u * x, -u * y, u}, dv[3] = {-v * x, -v * y, v};
        xx += x * x; xy += x * y; x1 += x; yy += y * y; y1 += y;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            xu[c] += x * du[c]; yu[c] += y * du[c]; ou[c] += du[c];
            xv[c] += x * dv[c]; yv[c] += y * dv[c]; ov[c] += dv[c];
        }
        s66 += du[0] * du[0] + dv[0] * dv[0];
        s67 += du[0] * du[1] + dv[0] * dv[1];
        s68 += du[0] * du[2] + dv[0] * dv[2];
        s77 += du[1] * du[1] + dv[1] * dv[1];
        s78 += du[1] * du[2] + dv[1] * dv[2];
    }
    double m[8][9];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < 9; ++c) m[r][c] = 0.0;
    m[0][0] = m[3][3] = xx;
    m[0][1] = m[1][0] = m[3][4] = m[4][3] = xy;
    m[0][2] = m[2][0] = m[3][5] = m[5][3] = x1;
    m[1][1] = m[4][4] = yy;
    m[1][2] = m[2][1] = m[4][5] = m[5][4] = y1;
    m[2][2] = m[5][5] = 4.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        m[0][6 + c] = xu[c]; m[1][6 + c] = yu[c]; m[2][6 + c] = ou[c];
        m[3][6 + c] = xv[c]; m[4][6 + c] = yv[c]; m[5][6 + c] = ov[c];
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        m[6 + c][0] = xu[c]; m[6 + c][1] = yu[c]; m[6 + c][2] = ou[c];
        m[6 + c][3] = xv[c]; m[6 + c][4] = yv[c]; m[6 + c][5] = ov[c];
    }
    m[6][6] = s66;
    m[6][7] = m[7][6] = s67;
    m[6][8] = s68;
    m[7][7] = s77;
    m[7][8] = s78;
    double max_entry = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        if (fabs(m[i][i]) > max_entry) max_entry = fabs(m[i][i]);
    // A failed pivot makes the model invalid; the steps after it still run
    // and their values are discarded.
    bool solvable = true;
    eliminate<0>(m, max_entry, solvable);
    eliminate<1>(m, max_entry, solvable);
    eliminate<2>(m, max_entry, solvable);
    eliminate<3>(m, max_entry, solvable);
    eliminate<4>(m, max_entry, solvable);
    eliminate<5>(m, max_entry, solvable);
    eliminate<6>(m, max_entry, solvable);
    eliminate<7>(m, max_entry, solvable);
    if (!solvable) return false;
    double h[9];
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = m[i][8];
    h[8] = 1.0;
    const double den_a[9] = {1.0 / sa, 0, cax, 0, 1.0 / sa, cay, 0, 0, 1};
    const double nrm_b[9] = {sb, 0, -sb * cbx, 0, sb, -sb * cby, 0, 0, 1};
    double tmp[9];
    mat3_mul(den_a, h, tmp);
    mat3_mul(tmp, nrm_b, out);
    return h_normalize(out);
}

__device__ __forceinline__ bool valid_domain(const double* h, int width, int height) {
    const double z[4] = {h[8], h[6] * (width - 1) + h[8], h[7] * (height - 1) + h[8],
                         h[6] * (width - 1) + h[7] * (height - 1) + h[8]};
    for (int i = 0; i < 4; ++i)
        if (!fin(z[i]) || fabs(z[i]) < 1e-15 || (z[i] > 0.0) != (z[0] > 0.0)) return false;
    return true;
}

__device__ __forceinline__ bool better(const Model& a, const Model& b) {
    return a.valid && (!b.valid || a.loss < b.loss || (a.loss == b.loss && a.hypothesis < b.hypothesis));
}

__device__ __forceinline__ Pt gather(const PairIO& j, int i) {
    const int ia = j.m.idx_a[i], ib = j.m.idx_b[i];
    return Pt{static_cast<double>(j.a.x[ia]), static_cast<double>(j.a.y[ia]), static_cast<double>(j.b.x[ib]),
              static_cast<double>(j.b.y[ib])};
}

__device__ __forceinline__ double octet(double v, int src) { return __shfl_sync(0xffffffffu, v, src, 8); }

// Hypothesis h by eight lanes (every lane of the warp calls, each eight with
// their own h): the sample, the degeneracy test, the 4-point fit and the
// domain test. The fit solves the normalised normal equations of the design
// rows {x, y, 1, 0, 0, 0, -u x, -u y, u} and {0, 0, 0, x, y, 1, -v x, -v y, v}
// by Gauss-Jordan with partial pivoting, h33 = 1, then denormalises and
// scales, as fit4_regs does. Lane r owns row r of the 8x9 system; every entry goes through the
// reference's operations in its order (products with a structural 0 only add
// +-0 to a sum started at +0.0 and are left out). True, with the model on all
// eight lanes, when the hypothesis is usable.
//
// For the per-pair call, whose hypotheses leave most of the chip idle: a
// thread per hypothesis (fit4_regs) takes 18,000 cycles, most of them its 45
// divisions, each a branchy sequence of about 125 cycles, one after the other;
// here a pivot row's divisions run side by side. Per-pair search at 512x512,
// 2000 hypotheses: 25 -> 15 us. It issues more instructions per hypothesis,
// so the batched form, which fills the chip, keeps fit4_regs (64 pairs x 2000
// hypotheses: 132 us with eight lanes).
__device__ __forceinline__ bool fit_octet(const PairIO& j, int nm, int h, int bw, int bh, double* out) {
    const int k8 = threadIdx.x & 7;
    // the sample: lane k < 4 draws and gathers point k
    int idx[4];
    {
        const int mine = sample_draw(nm, j.c.seed, h, k8 & 3);
#pragma unroll
        for (int k = 0; k < 4; ++k) idx[k] = __shfl_sync(0xffffffffu, mine, k, 8);
        distinct_draws(idx);
    }
    Pt p[4];
    {
        int i = idx[0];
#pragma unroll
        for (int k = 1; k < 4; ++k) i = (k8 & 3) == k ? idx[k] : i;
        const int ia = j.m.idx_a[i], ib = j.m.idx_b[i];
        const float ax = j.a.x[ia], ay = j.a.y[ia], bx = j.b.x[ib], by = j.b.y[ib];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            p[k] = Pt{__shfl_sync(0xffffffffu, ax, k, 8), __shfl_sync(0xffffffffu, ay, k, 8),
                      __shfl_sync(0xffffffffu, bx, k, 8), __shfl_sync(0xffffffffu, by, k, 8)};
    }
    // image A on the even lanes, B on the odd ones: degeneracy, centroid, scale
    double q[4][2];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        q[k][0] = k8 & 1 ? p[k].bx : p[k].ax;
        q[k][1] = k8 & 1 ? p[k].by : p[k].ay;
    }
    bool ok = nondegenerate(q);
    double cx = 0, cy = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) { cx += q[k][0]; cy += q[k][1]; }
    cx /= 4; cy /= 4;
    double var = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) var += (q[k][0] - cx) * (q[k][0] - cx) + (q[k][1] - cy) * (q[k][1] - cy);
    ok = ok && var > 0.0 && fin(var);
    const double scale = sqrt(2.0 * 4 / var);
    const double inv = 1.0 / scale;
    const double cax = octet(cx, 0), cay = octet(cy, 0), sa = octet(scale, 0), isa = octet(inv, 0);
    const double cbx = octet(cx, 1), cby = octet(cy, 1), sb = octet(scale, 1);
    {
        const unsigned int votes = __ballot_sync(0xffffffffu, ok) >> (threadIdx.x & 24);
        ok = (votes & 3u) == 3u;
    }
    // row k8 of the normal equations
    double m[9];
#pragma unroll
    for (int c = 0; c < 9; ++c) m[c] = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double x = (p[k].bx - cbx) * sb, y = (p[k].by - cby) * sb;
        const double u = (p[k].ax - cax) * sa, v = (p[k].ay - cay) * sa;
        const double ux = -u * x, uy = -u * y, vx = -v * x, vy = -v * y;
        const double r0 = k8 == 0 ? x : k8 == 1 ? y : k8 == 2 ? 1.0 : k8 == 6 ? ux : k8 == 7 ? uy : 0.0;
        const double r1 = k8 == 3 ? x : k8 == 4 ? y : k8 == 5 ? 1.0 : k8 == 6 ? vx : k8 == 7 ? vy : 0.0;
        m[0] += r0 * x;
        m[1] += r0 * y;
        m[2] += r0;
        m[3] += r1 * x;
        m[4] += r1 * y;
        m[5] += r1;
        m[6] += r0 * ux + r1 * vx;
        m[7] += r0 * uy + r1 * vy;
        m[8] += r0 * u + r1 * v;
    }
    double max_entry = fabs(m[0]);
#pragma unroll
    for (int c = 1; c < 8; ++c) max_entry = k8 == c ? fabs(m[c]) : max_entry;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        const double v = __shfl_xor_sync(0xffffffffu, max_entry, o);
        if (v > max_entry) max_entry = v;
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        // pivot: the first of the largest entries at or below the diagonal. (A
        // NaN may be picked or passed over; its row stays NaN until it is the
        // pivot row, so the system is rejected either way.)
        double best = k8 >= c ? fabs(m[c]) : -1.0;
        int piv = k8;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const double v = __shfl_xor_sync(0xffffffffu, best, o);
            const int r = __shfl_xor_sync(0xffffffffu, piv, o);
            if (v > best || (v == best && r < piv)) { best = v; piv = r; }
        }
        piv = max(__shfl_sync(0xffffffffu, piv, 0, 8), c);  // below c only when NaN entries alone are left
        const double pv = octet(m[c], piv);
        ok = ok && fin(pv) && !(fabs(pv) <= 1e-12 * max_entry);
        // the pivot row divided by the pivot: column c + 1 + k on lane k
        double num = 1.0;
#pragma unroll
        for (int jx = c + 1; jx < 9; ++jx) {
            const double v = octet(m[jx], piv);
            num = k8 == jx - c - 1 ? v : num;
        }
        const double quo = num / pv;
        // row c moves to the pivot row's place
        const double fc = octet(m[c], c);
        const double f = k8 == piv ? fc : m[c];
#pragma unroll
        for (int jx = c + 1; jx < 9; ++jx) {
            const double old = octet(m[jx], c);
            const double v = octet(quo, jx - c - 1);
            const double e = k8 == piv ? old : m[jx];
            m[jx] = k8 == c ? v : e - f * v;
        }
    }
    double n[9];
#pragma unroll
    for (int i = 0; i < 8; ++i) n[i] = octet(m[8], i);
    n[8] = 1.0;
    const double den_a[9] = {isa, 0, cax, 0, isa, cay, 0, 0, 1};
    const double nrm_b[9] = {sb, 0, -sb * cbx, 0, sb, -sb * cby, 0, 0, 1};
    double tmp[9];
    mat3_mul(den_a, n, tmp);
    mat3_mul(tmp, nrm_b, n);
    // scaled to the largest magnitude: entry k on lane k, entry 8 on every lane
    double top = 0.0;
    bool finite = true;
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        finite = finite && fin(n[i]);
        if (fabs(n[i]) > top) top = fabs(n[i]);
    }
    double e = n[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) e = k8 == i ? n[i] : e;
    e /= top;
    out[8] = n[8] / top;
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = octet(e, i);
    const double det = out[0] * (out[4] * out[8] - out[5] * out[7]) - out[1] * (out[3] * out[8] - out[5] * out[6]) +
                       out[2] * (out[3] * out[7] - out[4] * out[6]);
    return ok && finite && top > 0.0 && fin(det) && fabs(det) > 1e-15 && valid_domain(out, bw, bh);
}

__device__ __forceinline__ bool same_scale(const ScaleInfo& a, const ScaleInfo& b) {
    if (a.orig_w != b.orig_w || a.orig_h != b.orig_h || a.work_w != b.work_w || a.work_h != b.work_h ||
        a.sx != b.sx || a.sy != b.sy)
        return false;
    for (int i = 0; i < 9; ++i)
        if (a.D[i] != b.D[i]) return false;
    return true;
}

// --------------------------------------------------------------- prepare

// Restart or validate an extension, then check counts, indices and
// coordinates of every match. One block per pair.
template <class Src>
__global__ __launch_bounds__(kPrepareThreads) void prepare_kernel(const __grid_constant__ Src src) {
    wait_for_previous();
    __shared__ int go, bad;
    __shared__ unsigned int top[4];
    PairIO j;
    int local;
    if (!src.find(blockIdx.x, &j, &local)) return;
    State* s = j.state;
    if (threadIdx.x == 0) {
        const int na = *j.a.d_count, nb = *j.b.d_count, nm = *j.m.d_count;
        const auto& c = j.c;
        if (c.previous_hypotheses == 0) {
            s->best = Model{};
            s->ax = j.a.x; s->ay = j.a.y; s->bx = j.b.x; s->by = j.b.y;
            s->idx_a = j.m.idx_a; s->idx_b = j.m.idx_b;
            s->count_a = j.a.d_count; s->count_b = j.b.d_count; s->count_m = j.m.d_count;
            s->na = na; s->nb = nb; s->nm = nm;
            s->cap_a = j.a.capacity; s->cap_b = j.b.capacity; s->cap_m = j.m.capacity;
            s->evaluated = 0; s->batch_size = c.batch_size; s->threshold = c.threshold;
            s->seed = c.seed; s->generation = c.generation;
            s->scale_a = j.sa; s->scale_b = j.sb;
            s->status = static_cast<int>(Status::OK);
        } else if (s->evaluated != c.previous_hypotheses || s->generation != c.generation ||
                   s->seed != c.seed || s->threshold != c.threshold || s->batch_size != c.batch_size ||
                   s->ax != j.a.x || s->ay != j.a.y || s->bx != j.b.x || s->by != j.b.y ||
                   s->idx_a != j.m.idx_a || s->idx_b != j.m.idx_b || s->count_a != j.a.d_count ||
                   s->count_b != j.b.d_count || s->count_m != j.m.d_count || s->cap_a != j.a.capacity ||
                   s->cap_b != j.b.capacity || s->cap_m != j.m.capacity || s->na != na || s->nb != nb ||
                   s->nm != nm || !same_scale(s->scale_a, j.sa) || !same_scale(s->scale_b, j.sb)) {
            s->status = static_cast<int>(Status::INVALID_ARGUMENT);
        }
        s->bound = s->best.valid && fin(s->best.loss) ? static_cast<unsigned long long>(__double_as_longlong(s->best.loss))
                                                      : kInfBits;
        int g = s->status == static_cast<int>(Status::OK);
        if (g && (na < 0 || na > j.a.capacity || nb < 0 || nb > j.b.capacity || nm < 0 || nm > j.m.capacity)) {
            s->status = static_cast<int>(Status::INVALID_ARGUMENT);
            g = 0;
        }
        go = g;
        bad = 0;
    }
    if (threadIdx.x < 4) top[threadIdx.x] = 0;
    __syncthreads();
    if (!go) return;
    const int na = s->na, nb = s->nb, nm = s->nm;
    unsigned int mx[4] = {0, 0, 0, 0};  // |x| of a float orders like its bits
#pragma unroll 4
    for (int i = threadIdx.x; i < nm; i += kPrepareThreads) {
        const int ia = j.m.idx_a[i], ib = j.m.idx_b[i];
        if (ia < 0 || ia >= na || ib < 0 || ib >= nb) { bad = 1; continue; }
        const float q[4] = {j.a.x[ia], j.a.y[ia], j.b.x[ib], j.b.y[ib]};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (!fin(q[c])) bad = 1;
            mx[c] = max(mx[c], __float_as_uint(fabsf(q[c])));
        }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const unsigned int w = __reduce_max_sync(0xffffffffu, mx[c]);
        if ((threadIdx.x & 31) == 0) atomicMax(&top[c], w);
    }
    __syncthreads();
    if (threadIdx.x < 4) s->coord_max[threadIdx.x] = __uint_as_float(top[threadIdx.x]);
    if (threadIdx.x == 0) {
        if (bad) s->status = static_cast<int>(Status::INVALID_ARGUMENT);
        else if (nm < 4) s->status = static_cast<int>(Status::NOT_ENOUGH_POINTS);
    }
}

// ---------------------------------------------------------------- search

struct SearchJob {
    PairIO io;
    int first, count;  // hypotheses [first, first + count)
    Model* prefit;     // models of these hypotheses from fit_kernel, or null (fit in the search)
};

constexpr int kFitThreads = 128;

// One thread per hypothesis h in [first, first + count): the counter-based
// sample, the degeneracy test, the 4-point fit and the domain test into
// prefit[h - first] (valid = 0 for a rejected sample). A thread owns the
// whole 8x9 system, so this kernel runs with all the registers it needs,
// apart from the scoring.
template <class Src>
__global__ __launch_bounds__(kFitThreads, 3) void fit_kernel(const __grid_constant__ Src src) {
    wait_for_previous();
    SearchJob sj;
    int block;
    if (!src.find(blockIdx.x, &sj, &block)) return;
    const PairIO& j = sj.io;
    const State* s = j.state;
    const int h = sj.first + block * kFitThreads + threadIdx.x;
    if (h >= sj.first + sj.count) return;
    Model m{};
    m.hypothesis = h;
    m.valid = 0;
    if (s->status == static_cast<int>(Status::OK)) {
        int idx[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) idx[k] = sample_draw(s->nm, j.c.seed, h, k);
        distinct_draws(idx);
        Pt f[4];
        double qa[4][2], qb[4][2];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            f[k] = gather(j, idx[k]);
            qa[k][0] = f[k].ax; qa[k][1] = f[k].ay;
            qb[k][0] = f[k].bx; qb[k][1] = f[k].by;
        }
        m.valid = nondegenerate(qa) && nondegenerate(qb) && fit4_regs(f, m.h) &&
                  valid_domain(m.h, s->scale_b.work_w, s->scale_b.work_h);
    }
    sj.prefit[h - sj.first] = m;
}

// FP32 bounds of a model's loss L = sum of min(r^2, tau^2), r = |H b - a|.
// With u = 2^-24, the coordinate bounds Ax, Ay, Bx, By of the pair and the
// FP32 evaluation of X, Y, Z (two FMAs on rounded entries each), 1/Z (one
// approximate reciprocal, for which the PTX ISA states one unit in the last place
// over the full range: a relative error of 2u) and d = X (1/Z) - ax (one FMA):
//   |Z' - Z| <= EZ = 4u (|h6| Bx + |h7| By + |h8|) + 2e-15, likewise EX, EY,
//   e = |r' - r| <= c0 + c1 |1/Z'|, W = 4 tau + Ax + Ay,
//   c0 = 2.2u W + 4u tau,  c1 = 1.5 (W EZ + EX + EY),
// for points with both |d'| <= 2 tau and c0 + c1 |1/Z'| <= tau / 2. There
// min(r, tau)^2 changes by at most 2 tau e. Where c0 + c1 |1/Z'| > tau / 2 the
// bound used is 2 tau * tau / 2, which no change of min(r, tau)^2 exceeds; and
// with it <= tau / 2, |d'| > 2 tau implies that both r and r' exceed tau, so
// the term is tau^2 either way. (The 2e-15 covers |Z| < 1e-15, which the exact
// residual calls unreachable: then c1 |1/Z'| > tau / 2.) So
//   |L - L'| <= 2 tau (c0 n + c1 sum min(|1/Z'|, cap)) + 6u tau^2 n,
//   cap = (tau / 2 - c0) / c1,
// with 6u tau^2 for the rounding of each squared term, plus the FP32
// summation's relative error. Used only where no FP32 operation can overflow.
struct Bounds {
    double c0, c1;
    float cap;
};

__device__ __forceinline__ bool bounds_apply(const State* s, int nm, double tau) {
    const float* c = s->coord_max;
    return tau >= 1e-6 && tau <= 1e6 && nm <= (1 << 20) && fmaxf(fmaxf(c[0], c[1]), fmaxf(c[2], c[3])) <= 1048576.0f;
}

__device__ __forceinline__ Bounds model_bounds(const double* h, const State* s, double tau) {
    constexpr double u = 1.0 / 16777216.0;
    const double w = 4.0 * tau + s->coord_max[0] + s->coord_max[1];
    const double bx = s->coord_max[2], by = s->coord_max[3];
    const double ex = 4.0 * u * (fabs(h[0]) * bx + fabs(h[1]) * by + fabs(h[2])) + 1e-30;
    const double ey = 4.0 * u * (fabs(h[3]) * bx + fabs(h[4]) * by + fabs(h[5])) + 1e-30;
    const double ez = 4.0 * u * (fabs(h[6]) * bx + fabs(h[7]) * by + fabs(h[8])) + 2e-15;
    Bounds b;
    b.c0 = 1.05 * (2.2 * u * w + 4.0 * u * tau);
    b.c1 = 1.05 * 1.5 * (w * ez + ex + ey);
    const double cap = (0.5 * tau - b.c0) / b.c1;
    b.cap = cap > 0.0 ? static_cast<float>(fmin(cap, 1e30)) : 0.0f;
    return b;
}

__device__ __forceinline__ float approx_rcp(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Two FP32 operations per instruction (each rounded as the scalar one).
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2(float lo, float hi) {
    F2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ void f2_split(F2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
    F2 v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
    return v;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
    F2 v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
    F2 v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}

// Matches in shared memory, two by two: {bx0, bx1, by0, by1, -ax0, -ax1, -ay0,
// -ay1}, the operands of the packed FP32 bounds.
__device__ __forceinline__ void put_match(float* pts, int i, float ax, float ay, float bx, float by) {
    float* q = pts + 8 * (i >> 1) + (i & 1);
    q[0] = bx;
    q[2] = by;
    q[4] = -ax;
    q[6] = -ay;
}

__device__ __forceinline__ Pt get_match(const float* pts, int i) {
    const float* q = pts + 8 * (i >> 1) + (i & 1);
    return Pt{-q[4], -q[6], q[0], q[2]};
}

// Block b of a pair takes the groups b, b + blocks, ... of kGroup consecutive
// hypotheses; its best model goes to block_best[b].
// Why bounds first: with about 90 % inliers nearly every model used to be
// scored in FP64 over a fifth to all of the matches before it could be
// dropped, two FP64 divisions per match (36 issue slots each). The FP32 bounds
// take 10 instructions per match (two matches per FMA), read a match once for
// 32 models (a broadcast), and are within about 0.1 % of the loss, so that only the models
// that close to the best are left for FP64: usually one per block.
// Of 64 pairs x 2000 models 155 are scored in FP64 at 512x512; the batched
// search without the fit went 188 -> 64 us, the per-pair search 52 -> 15 us
// (2000 hypotheses, 310 matches) and 331 -> 95 us (8000, 8000).
// Layout: 256 / kGroup threads share a model, each over every (256 / kGroup)th
// pair of matches. kPrefit: the models come from fit_kernel (batched form);
// else the block fits them here (per-pair form, whose workspace has no room
// for them).
template <class Src, bool kPrefit, int kGroup>
__global__ __launch_bounds__(kSearchThreads, kPrefit ? 4 : 2) void search_kernel(const __grid_constant__ Src src) {
    wait_for_previous();
    constexpr int kSlices = kSearchThreads / kGroup;
    constexpr int kStage = kPrefit ? kStagePoints : kStagePointsFused;
    extern __shared__ float4 pts4[];
    float* const pts = reinterpret_cast<float*>(pts4);
    __shared__ double mh[kGroup][9], low[kGroup];  // models and the lower bounds of their losses
    __shared__ float part[kSlices][2][kGroup], caps[kGroup];
    __shared__ double red[2][128];
    __shared__ Model best;
    __shared__ int chosen[2];
    SearchJob sj;
    int block;
    if (!src.find(blockIdx.x, &sj, &block)) return;
    const PairIO& j = sj.io;
    State* s = j.state;
    const int t = threadIdx.x, lane = t & 31;
    if (t == 0) best.valid = 0;
    const bool ok = s->status == static_cast<int>(Status::OK);
    const int nm = ok ? s->nm : 0;
    const double tau = j.c.threshold, thr2 = tau * tau;
    const bool bounded = ok && bounds_apply(s, nm, tau);
    const auto stage = [&](int base) {
        const int n = min(kStage, nm - base);
#pragma unroll 4
        for (int i = t; i < n; i += kSearchThreads) {
            const int ia = j.m.idx_a[base + i], ib = j.m.idx_b[base + i];
            put_match(pts, i, j.a.x[ia], j.a.y[ia], j.b.x[ib], j.b.y[ib]);
        }
    };
    if (ok) stage(0);
    const int groups = ok ? (sj.count + kGroup - 1) / kGroup : 0;
    for (int group = block; group < groups; group += j.search_blocks) {
        const int h0 = sj.first + group * kGroup;
        // 1. models
        int valid = 0;
        if (kPrefit) {
            if (t < kGroup && h0 + t < sj.first + sj.count) {
                const Model& m = sj.prefit[h0 + t - sj.first];
                valid = m.valid;
                if (valid)
#pragma unroll
                    for (int e = 0; e < 9; ++e) mh[t][e] = m.h[e];
            }
        } else {
            for (int g = t >> 3; g - (lane >> 3) < kGroup; g += kSearchThreads / 8) {  // warp-uniform
                const int hyp = min(h0 + g, sj.first + sj.count - 1);
                double h[9];
                const bool fit = fit_octet(j, nm, hyp, s->scale_b.work_w, s->scale_b.work_h, h);
                if (g < kGroup) {
                    if ((t & 7) == 0) {
#pragma unroll
                        for (int e = 0; e < 9; ++e) mh[g][e] = h[e];
                        low[g] = fit && h0 + g < sj.first + sj.count ? 1.0 : 0.0;
                    }
                }
            }
            __syncthreads();
            if (t < kGroup) valid = low[t] != 0.0;
        }
        Bounds bd{};
        if (t < kGroup) {
            if (valid) {
                double h[9];
#pragma unroll
                for (int e = 0; e < 9; ++e) h[e] = mh[t][e];
                bd = model_bounds(h, s, tau);
            } else {
#pragma unroll
                for (int e = 0; e < 9; ++e) mh[t][e] = 0.0;
            }
            caps[t] = bd.cap;
        }
        __syncthreads();
        // 2. FP32 bounds
        double lo = 0.0;
        if (bounded) {
            const int m = t % kGroup, slice = t / kGroup;
            float h[9];
#pragma unroll
            for (int e = 0; e < 9; ++e) h[e] = static_cast<float>(mh[m][e]);
            const float cap = caps[m], top = static_cast<float>(thr2);
            F2 hh[9];
#pragma unroll
            for (int e = 0; e < 9; ++e) hh[e] = f2(h[e], h[e]);
            F2 sums = f2(0.0f, 0.0f), invs = sums;
            float sum = 0.0f, inv = 0.0f;
            for (int base = 0; base < nm; base += kStage) {
                if (nm > kStage) {
                    __syncthreads();
                    stage(base);
                    __syncthreads();
                }
                const int n = min(kStage, nm - base);
                const ulonglong2* const two = reinterpret_cast<const ulonglong2*>(pts);
#pragma unroll 4
                for (int i = slice; i < n / 2; i += kSlices) {
                    const ulonglong2 b = two[2 * i], a = two[2 * i + 1];
                    const F2 z = f2_fma(hh[6], b.x, f2_fma(hh[7], b.y, hh[8]));
                    const F2 x = f2_fma(hh[0], b.x, f2_fma(hh[1], b.y, hh[2]));
                    const F2 y = f2_fma(hh[3], b.x, f2_fma(hh[4], b.y, hh[5]));
                    float z0, z1;
                    f2_split(z, z0, z1);
                    const float r0 = approx_rcp(z0), r1 = approx_rcp(z1);
                    const F2 r = f2(r0, r1);
                    const F2 dx = f2_fma(x, r, a.x), dy = f2_fma(y, r, a.y);
                    float d0, d1;
                    f2_split(f2_fma(dx, dx, f2_mul(dy, dy)), d0, d1);
                    // a NaN counts as top, within its error
                    sums = f2_add(sums, f2(fminf(d0, top), fminf(d1, top)));
                    invs = f2_add(invs, f2(fminf(fabsf(r0), cap), fminf(fabsf(r1), cap)));
                }
                if ((n & 1) && slice == 0) {
                    const Pt q = get_match(pts, n - 1);
                    const float bx = static_cast<float>(q.bx), by = static_cast<float>(q.by);
                    const float r = approx_rcp(__fmaf_rn(h[6], bx, __fmaf_rn(h[7], by, h[8])));
                    const float dx = __fmaf_rn(__fmaf_rn(h[0], bx, __fmaf_rn(h[1], by, h[2])), r, -static_cast<float>(q.ax));
                    const float dy = __fmaf_rn(__fmaf_rn(h[3], bx, __fmaf_rn(h[4], by, h[5])), r, -static_cast<float>(q.ay));
                    sum += fminf(__fmaf_rn(dx, dx, dy * dy), top);
                    inv += fminf(fabsf(r), cap);
                }
            }
            {
                float lo0, hi0;
                f2_split(sums, lo0, hi0);
                sum += lo0 + hi0;
                f2_split(invs, lo0, hi0);
                inv += lo0 + hi0;
            }
            part[slice][0][m] = sum;
            part[slice][1][m] = inv;
            __syncthreads();
            if (t < kGroup) {
                double total = 0.0, reach = 0.0;
#pragma unroll
                for (int v = 0; v < kSlices; ++v) {
                    total += part[v][0][t];
                    reach += part[v][1][t];
                }
                const double rel = 1.2e-7 * (nm / kSlices + 16);  // FP32 summation of nonnegative terms
                const double err = 1.01 * (2.0 * tau * (bd.c0 * nm + bd.c1 * reach * (1.0 + rel)) + 3.6e-7 * thr2 * nm);
                lo = total * (1.0 - rel) - err;
                double hi = valid ? total * (1.0 + rel) + err : DBL_MAX;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    if (kGroup < 32 && o >= kGroup) continue;
                    const double v = __shfl_xor_sync(kGroup < 32 ? (1u << kGroup) - 1u : 0xffffffffu, hi, o);
                    hi = v < hi ? v : hi;
                }
                if ((t & 31) == 0 && hi < DBL_MAX)
                    atomicMin(&s->bound, static_cast<unsigned long long>(__double_as_longlong(hi)));
            }
        }
        if (t < kGroup) low[t] = valid ? lo : __longlong_as_double(static_cast<long long>(kInfBits));
        __syncthreads();
        // 3. exact losses of the models that may still win, the two lowest
        // bounds at a time. A model whose lower bound exceeds another valid
        // model's loss or upper bound loses to it (ties need equal losses).
        for (;;) {
            if (t < 32) {
                const double bound = __longlong_as_double(
                    static_cast<long long>(*reinterpret_cast<volatile unsigned long long*>(&s->bound)));
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    double v = DBL_MAX;
                    int at = -1;
                    for (int m = lane; m < kGroup; m += 32)
                        if (low[m] <= bound && low[m] < v) { v = low[m]; at = m; }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        const double w = __shfl_xor_sync(0xffffffffu, v, o);
                        const int x = __shfl_xor_sync(0xffffffffu, at, o);
                        if (x >= 0 && (at < 0 || w < v || (w == v && x < at))) { v = w; at = x; }
                    }
                    __syncwarp();
                    if (lane == 0) {
                        chosen[half] = at;
                        if (at >= 0) low[at] = __longlong_as_double(static_cast<long long>(kInfBits));
                    }
                    __syncwarp();
                }
            }
            __syncthreads();
            if (chosen[0] < 0) break;
            const int half = t >> 7, v = t & 127, m = chosen[half];
            if (m >= 0) {
                double h[9];
#pragma unroll
                for (int e = 0; e < 9; ++e) h[e] = mh[m][e];
                double acc = 0.0;
#pragma unroll 2
                for (int i = v; i < nm; i += 128) {
                    const double r = residual2(h, nm <= kStage ? get_match(pts, i) : gather(j, i));
                    acc += r < thr2 ? r : thr2;
                }
                red[half][v] = acc;
            }
            __syncthreads();
            if (v < 32 && m >= 0) {  // strides 64 and 32 of the tree, then 16 ... 1
                double a = (red[half][v] + red[half][v + 64]) + (red[half][v + 32] + red[half][v + 96]);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
                if (v == 0) red[half][0] = a;
            }
            __syncthreads();
            if (t == 0) {
                for (int k = 0; k < 2 && chosen[k] >= 0; ++k) {
                    Model cand;
                    cand.loss = red[k][0];
                    cand.hypothesis = h0 + chosen[k];
                    cand.valid = fin(cand.loss);
                    if (!better(cand, best)) continue;
                    for (int e = 0; e < 9; ++e) best.h[e] = mh[chosen[k]][e];
                    best.loss = cand.loss;
                    best.hypothesis = cand.hypothesis;
                    best.valid = 1;
                    atomicMin(&s->bound, static_cast<unsigned long long>(__double_as_longlong(cand.loss)));
                }
            }
        }
    }
    __syncthreads();
    if (t == 0) j.block_best[block] = best;
}

// ---------------------------------------------------------------- finish

// The finish kernel is bound by its serial FP64 sums: the reference adds
// every loss, centroid, spread and normal-matrix sum in index order on one
// thread, and bit-identical sums need that order. What is left to choose is
// how few such passes run one after another and what a pass waits for:
// - the points are gathered once into shared memory (kFinishStage of them);
// - the producer warps compute a chunk of terms while the lanes of warp 0, one per
//   sum, add the chunk before it, read two doubles at a time and a group of
//   eight ahead of the adds (chain_sums);
// - the sums that need the same pass share it: a model's loss, its inlier
//   residual sum and its inliers' centroid (6 lanes), the two spreads, and
//   the 28 distinct sums of the 72 normal-matrix entries;
// - the refit passes run over the list of kept points only: a dropped point
//   adds +0.0, which leaves a sum started at +0.0 bit for bit unchanged.
// Per-pair finish at 512x512, 310 matches: 49 -> 27 us; 8000 matches,
// half of them inliers: 641 -> 156 us (seven passes over all points before).
// Chunks are as long as shared memory allows (a chunk costs a barrier and the
// latency of its first loads, about 200 cycles, against 8 cycles per add).
constexpr int kFinishStage = 8192;  // matched points held in shared memory
constexpr int kFinishProducers = kFinishThreads - 32;
constexpr int kEvalChunk = 448;     // points per chunk of the loss and spread passes
constexpr int kMatrixChunk = 112;   // and of the normal-matrix pass
constexpr int kEvalSums = 6;        // loss, inlier residuals, centroid of the inliers
constexpr int kMatrixSums = 28;
// a sum's terms of a chunk: one row, padded by 16 bytes so that the rows of
// eight lanes reading 16 bytes each lie in different banks
__host__ __device__ constexpr int kTermRow(int chunk) { return chunk + 2; }
constexpr int kTermWords = kMatrixSums * kTermRow(kMatrixChunk);
static_assert(kEvalSums * kTermRow(kEvalChunk) <= kTermWords, "term buffer");

// Bytes of dynamic shared memory for a match capacity: two chunks of terms,
// the points, the kept list and two sets of keep flags.
__host__ __device__ inline int finish_smem_bytes(int match_capacity) {
    const int n = match_capacity < 1 ? 1 : (match_capacity < kFinishStage ? match_capacity : kFinishStage);
    return 2 * kTermWords * static_cast<int>(sizeof(double)) +
           (n + 7) / 8 * 8 * static_cast<int>(sizeof(float4) + sizeof(std::uint16_t) + 2);
}

struct FinishShared {
    float4* pts;
    std::uint16_t* list;
    std::uint8_t* keep[2];  // inliers of the current model and of the candidate
    double (*terms)[kTermWords];  // two chunks
};

// kSums sums over i < n of the terms produce(i, part, out) writes at out[c *
// kTermRow(kChunk)], c < kSums: sum c in index order on lane c of warp 0
// (acc, carried in and out), with the terms computed one chunk ahead by the
// other warps. The last chunk is filled up to a multiple of 16 with +0.0.
// Every thread of the block calls it; it ends with a barrier. A point's terms
// are computed in kParts parts by as many threads.
template <int kChunk, int kSums, int kParts, class F>
__device__ __forceinline__ void chain_sums(int n, double (*terms)[kTermWords], double& acc, F produce) {
    static_assert(kChunk % 16 == 0 && kChunk * kParts % kFinishProducers == 0, "producers");
    const int t = threadIdx.x;
    const int steps = (n + kChunk - 1) / kChunk;
#pragma unroll 1
    for (int step = 0; step <= steps; ++step) {
        if (t >= 32) {
            if (step < steps) {
#pragma unroll 1
                for (int w = t - 32; w < kChunk * kParts; w += kFinishProducers) {
                    const int x = w % kChunk, part = w / kChunk;
                    const int i = step * kChunk + x;
                    double* out = terms[step & 1] + x;
                    if (i < n) {
                        produce(i, part, out);
                    } else if (part == 0 && i < (n + 15) / 16 * 16) {
#pragma unroll 1
                        for (int c = 0; c < kSums; ++c) out[c * kTermRow(kChunk)] = 0.0;
                    }
                }
            }
        } else if (t < kSums && step > 0) {
            const int left = min(kChunk, n - (step - 1) * kChunk);
            const double2* row = reinterpret_cast<const double2*>(terms[(step - 1) & 1] + t * kTermRow(kChunk));
            double a = acc;
            double2 q0 = row[0], q1 = row[1], q2 = row[2], q3 = row[3];
#pragma unroll 1
            for (int i = 0; i < left; i += 16) {  // reads up to 8 terms past the last 16, without adding them
                const double2* r = row + i / 2;
                const double2 p0 = r[4], p1 = r[5], p2 = r[6], p3 = r[7];
                a += q0.x; a += q0.y; a += q1.x; a += q1.y;
                a += q2.x; a += q2.y; a += q3.x; a += q3.y;
                q0 = r[8]; q1 = r[9]; q2 = r[10]; q3 = r[11];
                a += p0.x; a += p0.y; a += p1.x; a += p1.y;
                a += p2.x; a += p2.y; a += p3.x; a += p3.y;
            }
            acc = a;
        }
        __syncthreads();
    }
}

__device__ __forceinline__ Pt finish_point(const PairIO& j, const FinishShared& sh, int i) {
    if (i < kFinishStage) {
        const float4 q = sh.pts[i];
        return Pt{q.x, q.y, q.z, q.w};
    }
    return gather(j, i);
}

// Serial loss, inlier residual sum and inlier centroid sums of model h, into
// sums[kEvalSums], and its inlier count into *kept; the inliers' flags go to
// keep, or to j.mask when there are more points than shared memory holds.
__device__ __forceinline__ void evaluate(const PairIO& j, const FinishShared& sh, int nm, double thr2,
                                         const double* hs, double* sums, int* kept, std::uint8_t* keep) {
    double h[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) h[e] = hs[e];
    constexpr int kRow = kTermRow(kEvalChunk);
    const bool staged = nm <= kFinishStage;
    double acc = 0.0;
    int mine = 0;
    if (threadIdx.x == 0) *kept = 0;
    chain_sums<kEvalChunk, kEvalSums, 1>(nm, sh.terms, acc, [&](int i, int, double* out) {
        const Pt p = finish_point(j, sh, i);
        const double r = residual2(h, p);
        const bool in = r <= thr2;
        mine += in;
        if (staged) keep[i] = in;
        else j.mask[i] = in;
        out[0] = r < thr2 ? r : thr2;
        out[kRow] = in ? r : 0.0;
        out[2 * kRow] = in ? p.ax : 0.0;
        out[3 * kRow] = in ? p.ay : 0.0;
        out[4 * kRow] = in ? p.bx : 0.0;
        out[5 * kRow] = in ? p.by : 0.0;
    });
    if (threadIdx.x < kEvalSums) sums[threadIdx.x] = acc;
    if (mine) atomicAdd(kept, mine);
    __syncthreads();
}

// The kept points' indices, in order, into sh.list (block-wide scan).
__device__ __forceinline__ void list_kept(const FinishShared& sh, const std::uint8_t* keep, int nm) {
    __shared__ int warp_total[kFinishThreads / 32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int seg = (nm + kFinishThreads - 1) / kFinishThreads;
    const int lo = min(nm, t * seg), hi = min(nm, lo + seg);
    int n = 0;
    for (int i = lo; i < hi; ++i) n += keep[i];
    int run = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += v;
    }
    if (lane == 31) warp_total[warp] = run;
    __syncthreads();
    int at = run - n;
    for (int w = 0; w < warp; ++w) at += warp_total[w];
    for (int i = lo; i < hi; ++i)
        if (keep[i]) sh.list[at++] = static_cast<std::uint16_t>(i);
    __syncthreads();
}

// 3x3 matrices with entry e (row-major) on lane e, lanes 9 and up a copy of
// entry 8: mat3_mul and h_normalize, each entry by the same operations.
__device__ __forceinline__ double warp_mat3(double a, double b) {
    const int lane = threadIdx.x & 31, e = lane < 9 ? lane : 8, r = 3 * (e / 3), c = e % 3;
    const double a0 = __shfl_sync(0xffffffffu, a, r), a1 = __shfl_sync(0xffffffffu, a, r + 1),
                 a2 = __shfl_sync(0xffffffffu, a, r + 2);
    const double b0 = __shfl_sync(0xffffffffu, b, c), b1 = __shfl_sync(0xffffffffu, b, c + 3),
                 b2 = __shfl_sync(0xffffffffu, b, c + 6);
    return a0 * b0 + a1 * b1 + a2 * b2;
}

// The nine entries, on every lane.
__device__ __forceinline__ void warp_spread(double x, double* out) {
#pragma unroll
    for (int i = 0; i < 9; ++i) out[i] = __shfl_sync(0xffffffffu, x, i);
}

__device__ __forceinline__ bool warp_normalize(double& x) {
    double scale = fabs(x);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        const double v = __shfl_xor_sync(0xffffffffu, scale, o);
        if (v > scale) scale = v;
    }
    scale = __shfl_sync(0xffffffffu, scale, 0);  // the largest of lanes 0..15: every entry
    if (!__all_sync(0xffffffffu, fin(x)) || !(scale > 0.0)) return false;
    x /= scale;
    double h[9];
    warp_spread(x, h);
    const double det = h[0] * (h[4] * h[8] - h[5] * h[7]) - h[1] * (h[3] * h[8] - h[5] * h[6]) +
                       h[2] * (h[3] * h[7] - h[4] * h[6]);
    return fin(det) && fabs(det) > 1e-15;
}

// fit4_regs' Gauss-Jordan by one warp on M in shared memory (destroyed): each
// entry takes the serial solver's operations, the lanes split the independent
// ones, and columns left of the pivot, which are not read again, are left
// alone. Same validity and model on every lane. The loop over the columns
// stays a loop: the code runs once per launch, and unrolled its instruction
// fetches took longer than the arithmetic.
__device__ inline bool warp_solve(double (*M)[9], double cax, double cay, double cbx, double cby, double sa,
                                  double sb, double* out) {
    const int lane = threadIdx.x & 31, row = lane & 7, col = lane < 9 ? lane : 8;
    double max_entry = fabs(M[row][row]);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        const double v = __shfl_xor_sync(0xffffffffu, max_entry, o);
        if (v > max_entry) max_entry = v;
    }
    bool solvable = true;
#pragma unroll 1
    for (int c = 0; c < 8; ++c) {
        // the first of the largest entries at or below the diagonal. (A NaN
        // may be picked or passed over here; its row stays NaN until it is the
        // pivot row, so the system is rejected either way.)
        double pv = M[row][c];
        double best = row >= c ? fabs(pv) : -1.0;
        int piv = row;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const double v = __shfl_xor_sync(0xffffffffu, best, o), w = __shfl_xor_sync(0xffffffffu, pv, o);
            const int r = __shfl_xor_sync(0xffffffffu, piv, o);
            if (v > best || (v == best && r < piv)) { best = v; pv = w; piv = r; }
        }
        piv = __shfl_sync(0xffffffffu, piv, 0);
        pv = __shfl_sync(0xffffffffu, pv, 0);
        if (piv < c) {  // only NaN entries are left
            piv = c;
            pv = M[c][c];
        }
        solvable = solvable && fin(pv) && !(fabs(pv) <= 1e-12 * max_entry);
        const double a = M[c][col], b = M[piv][col];
        const double scaled = b / pv;
        __syncwarp();
        if (lane >= c && lane < 9) {
            M[piv][lane] = a;
            M[c][lane] = scaled;
        }
        __syncwarp();
#pragma unroll
        for (int s = 0; s < 3; ++s) {
            const int e = lane + 32 * s, r = e / 9, jx = e % 9;
            if (e < 72 && r != c && jx > c) M[r][jx] -= M[r][c] * M[c][jx];
        }
        __syncwarp();
    }
    double x = col < 8 ? M[col][8] : 1.0;  // entry `col` of the normalised model
    const double isa = 1.0 / sa;
    const double den_a = col == 0 || col == 4 ? isa : col == 2 ? cax : col == 5 ? cay : col == 8 ? 1.0 : 0.0;
    const double nrm_b = col == 0 || col == 4 ? sb : col == 2 ? -sb * cbx : col == 5 ? -sb * cby : col == 8 ? 1.0 : 0.0;
    x = warp_mat3(warp_mat3(den_a, x), nrm_b);
    const bool ok = warp_normalize(x);
    warp_spread(x, out);
    return solvable && ok;
}

// Least-squares refit over the kept points (sums and keep: evaluate()'s, of
// the model that kept them), into out (shared memory); false, on every
// thread, when there is no model or its domain test fails. The few divisions
// and square roots run side by side on the lanes of a warp: one after the
// other, on one thread, they took as long as a pass over 300 points.
__device__ inline bool block_fit(const PairIO& j, const FinishShared& sh, const std::uint8_t* keep, int nm, int kept,
                                 const double* sums, int bw, int bh, double* out) {
    __shared__ double centre[4], spread[2], scale[2], total[kMatrixSums];
    __shared__ double m[8][9];
    __shared__ int ok;
    const int t = threadIdx.x;
    if (kept < 4) return false;
    const bool listed = nm <= kFinishStage;
    const int items = listed ? kept : nm;
    if (t < 4) centre[t] = sums[2 + t] / kept;
    if (listed) list_kept(sh, keep, nm);
    else __syncthreads();
    const double cax = centre[0], cay = centre[1], cbx = centre[2], cby = centre[3];
    const auto point = [&](int i, Pt& p) {  // whether item i is kept
        if (listed) {
            const float4 q = sh.pts[sh.list[i]];
            p = Pt{q.x, q.y, q.z, q.w};
            return true;
        }
        p = gather(j, i);
        return j.mask[i] != 0;
    };
    // spreads
    {
        constexpr int kRow = kTermRow(kEvalChunk);
        double acc = 0.0;
        chain_sums<kEvalChunk, 2, 1>(items, sh.terms, acc, [&](int i, int, double* o) {
            Pt p;
            const bool k = point(i, p);
            o[0] = k ? (p.ax - cax) * (p.ax - cax) + (p.ay - cay) * (p.ay - cay) : 0.0;
            o[kRow] = k ? (p.bx - cbx) * (p.bx - cbx) + (p.by - cby) * (p.by - cby) : 0.0;
        });
        if (t < 2) {
            spread[t] = acc;
            scale[t] = sqrt(2.0 * kept / acc);
        }
        __syncthreads();
    }
    const double va = spread[0], vb = spread[1];
    if (!(va > 0.0) || !(vb > 0.0) || !fin(va) || !fin(vb)) return false;
    const double sa = scale[0], sb = scale[1];
    // normal matrix of the design rows {x, y, 1, 0, 0, 0, -ux, -uy, u} and
    // {0, 0, 0, x, y, 1, -vx, -vy, v}. A product with a structural 0 adds
    // +-0, a no-op; the blocks (0..2, 0..2) and (3..5, 3..5) are equal, the
    // matrix is symmetric (products commute) and the entry of the two 1s is
    // the count. What is left are kMatrixSums sums, in two parts: the x, y
    // block with the u rows (14 sums), and the v rows with rows 6 and 7 (14).
    {
        constexpr int kRow = kTermRow(kMatrixChunk);
        double acc = 0.0;
        chain_sums<kMatrixChunk, kMatrixSums, 2>(items, sh.terms, acc, [&](int i, int part, double* o) {
            Pt p;
            const bool k = point(i, p);
            const double x = (p.bx - cbx) * sb, y = (p.by - cby) * sb;
            const double u = (p.ax - cax) * sa, v = (p.ay - cay) * sa;
            const double w = part == 0 ? u : v;
            const double wx = -w * x, wy = -w * y;
            double* q = o + (part == 0 ? 10 : 19) * kRow;
            q[0] = k ? x * wx : 0.0;
            q[kRow] = k ? x * wy : 0.0;
            q[2 * kRow] = k ? x * w : 0.0;
            q[3 * kRow] = k ? y * wx : 0.0;
            q[4 * kRow] = k ? y * wy : 0.0;
            q[5 * kRow] = k ? y * w : 0.0;
            q[6 * kRow] = k ? wx : 0.0;
            q[7 * kRow] = k ? wy : 0.0;
            q[8 * kRow] = k ? w : 0.0;
            if (part == 0) {
                o[0] = k ? x * x : 0.0;
                o[kRow] = k ? x * y : 0.0;
                o[2 * kRow] = k ? x : 0.0;
                o[3 * kRow] = k ? y * y : 0.0;
                o[4 * kRow] = k ? y : 0.0;
            } else {
                const double ux = -u * x, uy = -u * y;
                o[5 * kRow] = k ? ux * ux + wx * wx : 0.0;
                o[6 * kRow] = k ? ux * uy + wx * wy : 0.0;
                o[7 * kRow] = k ? ux * u + wx * v : 0.0;
                o[8 * kRow] = k ? uy * uy + wy * wy : 0.0;
                o[9 * kRow] = k ? uy * u + wy * v : 0.0;
            }
        });
        if (t < kMatrixSums) total[t] = acc;
        __syncthreads();
    }
    if (t < 72) {
        // sum of each entry: kMatrixSums is 0, kMatrixSums + 1 the count
        constexpr unsigned char kZ = kMatrixSums, kN = kMatrixSums + 1;
        constexpr unsigned char kSum[72] = {0,  1,  2,  kZ, kZ, kZ, 10, 11, 12,   // x
                                            1,  3,  4,  kZ, kZ, kZ, 13, 14, 15,   // y
                                            2,  4,  kN, kZ, kZ, kZ, 16, 17, 18,   // 1
                                            kZ, kZ, kZ, 0,  1,  2,  19, 20, 21,   // x
                                            kZ, kZ, kZ, 1,  3,  4,  22, 23, 24,   // y
                                            kZ, kZ, kZ, 2,  4,  kN, 25, 26, 27,   // 1
                                            10, 13, 16, 19, 22, 25, 5,  6,  7,    // -ux, -vx
                                            11, 14, 17, 20, 23, 26, 6,  8,  9};   // -uy, -vy
        const int e = kSum[t];
        m[t / 9][t % 9] = e == kZ ? 0.0 : e == kN ? static_cast<double>(kept) : total[e];
    }
    __syncthreads();
    if (t < 32) {
        double h[9];
        const bool solved = warp_solve(m, cax, cay, cbx, cby, sa, sb, h) && valid_domain(h, bw, bh);
        if (t == 0) {
            ok = solved;
#pragma unroll
            for (int i = 0; i < 9; ++i) out[i] = h[i];
        }
    }
    __syncthreads();
    return ok;
}

// One block per pair: fold the search blocks' winners into the saved raw
// winner, refine, and build the mask and the result.
template <class Src>
__global__ __launch_bounds__(kFinishThreads, 1) void finish_kernel(const __grid_constant__ Src src) {
    wait_for_previous();
    extern __shared__ float4 finish_smem[];  // terms, points, kept list, keep flags
    __shared__ double model[2][9], loss;  // current model and candidate; loss of the current one
    __shared__ HomographyResult res;
    __shared__ double sums[2][kEvalSums];
    __shared__ int keep_mask, kept[2];
    __shared__ double mins[4][kFinishThreads / 32];
    PairIO j;
    int local;
    if (!src.find(blockIdx.x, &j, &local)) return;
    State* s = j.state;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const double nanv = __longlong_as_double(0x7ff8000000000000ll);
    const int status0 = s->status;
    const bool go = status0 == static_cast<int>(Status::OK);
    const int cap = min(j.m.capacity, kFinishStage);
    FinishShared sh;
    const int room = (max(cap, 1) + 7) / 8 * 8;
    sh.terms = reinterpret_cast<double (*)[kTermWords]>(finish_smem);
    sh.pts = finish_smem + 2 * kTermWords * sizeof(double) / sizeof(float4);
    sh.list = reinterpret_cast<std::uint16_t*>(sh.pts + room);
    sh.keep[0] = reinterpret_cast<std::uint8_t*>(sh.list + room);
    sh.keep[1] = sh.keep[0] + room;
    if (warp == 0) {
        // 1. raw winner: the best block result, if it beats the saved one
        Model b;  // only loss, hypothesis and valid are used
        b.loss = 0.0;
        b.hypothesis = 0;
        b.valid = 0;
        int at = -1;
#pragma unroll 4
        for (int i = lane; i < j.search_blocks; i += 32) {
            Model c;
            c.loss = j.block_best[i].loss;
            c.hypothesis = j.block_best[i].hypothesis;
            c.valid = j.block_best[i].valid;
            if (better(c, b)) { b.loss = c.loss; b.hypothesis = c.hypothesis; b.valid = c.valid; at = i; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            Model c;
            c.loss = __shfl_xor_sync(0xffffffffu, b.loss, o);
            c.hypothesis = __shfl_xor_sync(0xffffffffu, b.hypothesis, o);
            c.valid = __shfl_xor_sync(0xffffffffu, b.valid, o);
            const int other = __shfl_xor_sync(0xffffffffu, at, o);
            if (better(c, b)) { b.loss = c.loss; b.hypothesis = c.hypothesis; b.valid = c.valid; at = other; }
        }
        at = __shfl_sync(0xffffffffu, at, 0);
        const bool take = go && at >= 0 && better(b, s->best);
        const bool any = take || s->best.valid;
        const double x = lane < 9 ? (take ? j.block_best[at].h[lane] : s->best.h[lane]) : 0.0;
        __syncwarp();
        if (take && lane < 9) s->best.h[lane] = x;
        if (take && lane == 0) {
            s->best.loss = b.loss;
            s->best.hypothesis = b.hypothesis;
            s->best.valid = b.valid;
        }
        static_assert(sizeof(HomographyResult) % 8 == 0 && sizeof(HomographyResult) / 8 <= 32, "result words");
        if (lane < sizeof(HomographyResult) / 8) reinterpret_cast<std::uint64_t*>(&res)[lane] = 0;  // padding too
        __syncwarp();
        if (lane < 9) {
            model[0][lane] = x;
            res.H[lane] = res.H_s[lane] = nanv;
        }
        if (lane == 0) {
            res.num_matches = (s->nm >= 0 && s->nm <= j.m.capacity) ? s->nm : 0;
            res.reproj_residual = nanv;
            res.status = go && !any ? Status::DEGENERATE : static_cast<Status>(status0);
        }
    } else if (go) {
        const int staged = min(s->nm, kFinishStage);
#pragma unroll 4
        for (int i = t - 32; i < staged; i += kFinishThreads - 32) {
            const int ia = j.m.idx_a[i], ib = j.m.idx_b[i];
            sh.pts[i] = make_float4(j.a.x[ia], j.a.y[ia], j.b.x[ib], j.b.y[ib]);
        }
    }
    __syncthreads();
    bool fill = true;  // whether the mask is still to be cleared
    if (res.status == Status::OK) {
        const int nm = s->nm;
        const double thr2 = j.c.threshold * j.c.threshold;
        const int bw = s->scale_b.work_w, bh = s->scale_b.work_h;
        // One loop, so that the code of a pass is fetched once: the raw model,
        // then each refit, accepted on a strictly lower serial loss.
        int cur = 0, trial = 0;
#pragma unroll 1
        for (int step = 0;; ++step) {
            evaluate(j, sh, nm, thr2, model[trial], sums[trial], &kept[trial], sh.keep[trial]);
            const double now = sums[trial][0];
            const bool take = step == 0 || (fin(now) && now < loss);
            __syncthreads();
            if (!take) break;
            cur = trial;
            if (t == 0) loss = now;
            if (step >= j.c.refinement_steps) break;
            trial = cur ^ 1;
            if (!block_fit(j, sh, sh.keep[cur], nm, kept[cur], sums[cur], bw, bh, model[trial])) break;
        }
        // mask and inlier extent of the final model, and the result
        double mnx = DBL_MAX, mny = DBL_MAX, mxx = -DBL_MAX, mxy = -DBL_MAX;
        if (nm <= kFinishStage) {
            for (int i = t; i < nm; i += kFinishThreads)
                if (sh.keep[cur][i]) {
                    const float4 q = sh.pts[i];
                    mnx = fmin(mnx, static_cast<double>(q.x)); mxx = fmax(mxx, static_cast<double>(q.x));
                    mny = fmin(mny, static_cast<double>(q.y)); mxy = fmax(mxy, static_cast<double>(q.y));
                }
        } else {
            double h[9];
            for (int e = 0; e < 9; ++e) h[e] = model[cur][e];
            for (int i = t; i < nm; i += kFinishThreads) {
                const Pt q = gather(j, i);
                const bool in = residual2(h, q) <= thr2;
                j.mask[i] = in;
                if (in) {
                    mnx = fmin(mnx, q.ax); mxx = fmax(mxx, q.ax);
                    mny = fmin(mny, q.ay); mxy = fmax(mxy, q.ay);
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mnx = fmin(mnx, __shfl_xor_sync(0xffffffffu, mnx, o));
            mny = fmin(mny, __shfl_xor_sync(0xffffffffu, mny, o));
            mxx = fmax(mxx, __shfl_xor_sync(0xffffffffu, mxx, o));
            mxy = fmax(mxy, __shfl_xor_sync(0xffffffffu, mxy, o));
        }
        if (lane == 0) {
            mins[0][warp] = mnx; mins[1][warp] = mny; mins[2][warp] = mxx; mins[3][warp] = mxy;
        }
        __syncthreads();
        if (warp == 0) {  // one lane per entry of the matrices
            const int inliers = kept[cur], e = lane < 9 ? lane : 8;
            double a = DBL_MAX, bb = DBL_MAX, c = -DBL_MAX, d = -DBL_MAX;
            for (int w = 0; w < kFinishThreads / 32; ++w) {
                a = fmin(a, mins[0][w]); bb = fmin(bb, mins[1][w]);
                c = fmax(c, mins[2][w]); d = fmax(d, mins[3][w]);
            }
            const double hs = model[cur][e];
            double ia = j.inverse_a[0], db = j.d_b[0];  // selects: a run-time index would put the job in local memory
#pragma unroll
            for (int i = 1; i < 9; ++i) {
                ia = e == i ? j.inverse_a[i] : ia;
                db = e == i ? j.d_b[i] : db;
            }
            double H = warp_mat3(warp_mat3(ia, hs), db);
            bool ok = warp_normalize(H);
            double hh[9];
            warp_spread(H, hh);
            ok = ok && valid_domain(hh, s->scale_b.orig_w, s->scale_b.orig_h) && inliers >= 4;
            // four divisions, one per lane
            const double w = fmax(1.0, static_cast<double>(s->scale_a.work_w - 1));
            const double ht = fmax(1.0, static_cast<double>(s->scale_a.work_h - 1));
            const double num = lane == 0 ? static_cast<double>(inliers) : lane == 1 ? sums[cur][1] : lane == 2 ? c - a : d - bb;
            const double den = lane == 0 ? nm : lane == 1 ? inliers : lane == 2 ? w : ht;
            const double q = num / den;
            const double cover_x = __shfl_sync(0xffffffffu, q, 2), cover_y = __shfl_sync(0xffffffffu, q, 3);
            if (ok && lane < 9) {
                res.H[lane] = H;
                res.H_s[lane] = hs;
            }
            if (ok && lane == 0) {
                res.num_inliers = inliers;
                res.inlier_ratio = q;
                res.inlier_coverage = fmin(1.0, cover_x) * fmin(1.0, cover_y);
            }
            if (ok && lane == 1) res.reproj_residual = sqrt(q);
            if (lane == 0) {
                if (!ok) res.status = Status::DEGENERATE;
                keep_mask = ok;
            }
        }
        __syncthreads();
        if (keep_mask) {
            fill = false;
            if (nm <= kFinishStage)
                for (int i = t; i < j.m.capacity; i += kFinishThreads) j.mask[i] = i < nm ? sh.keep[cur][i] : 0;
            else
                for (int i = nm + t; i < j.m.capacity; i += kFinishThreads) j.mask[i] = 0;
        }
    }
    if (fill)
        for (int i = t; i < j.m.capacity; i += kFinishThreads) j.mask[i] = 0;
    if (t == 0) {
        s->evaluated = j.c.hypotheses;
        s->result = res;
        if (j.result_out) *j.result_out = res;
    }
}

}  // namespace stitch::b200::s5k
