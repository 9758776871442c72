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
// Layout of the work: a warp owns HPW consecutive hypotheses; lanes
// 0..HPW-1 each draw one sample and test it for degeneracy, then the whole
// warp fits each usable sample (the 8x9 system in shared memory, entries split
// over the lanes) and scores it. Lane l of the warp plays the reference's
// virtual lanes l, l+32, l+64 and l+96, so both the per-lane sums and the
// reduction tree are the reference's, operation for operation.
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
    // bits of the smallest loss of a fully scored model of this search (or
    // of the previous winner), +inf when none: a pruning bound shared by
    // every warp of the pair (nonnegative doubles order like their bits)
    unsigned long long bound;
};

constexpr unsigned long long kInfBits = 0x7ff0000000000000ull;  // +inf

constexpr int kSearchThreads = 256;
constexpr int kSearchWarps = kSearchThreads / 32;
constexpr int kMaxSearchBlocks = 2 * kSmCount;
constexpr int kStagePoints = 4096;  // matched points staged in shared memory per search block
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
__device__ __forceinline__ void sample_four(int n, std::uint64_t seed, int h, int* s) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        int v = static_cast<int>(splitmix64(seed ^ (static_cast<std::uint64_t>(h) * 4 + k)) %
                                 static_cast<std::uint64_t>(n - k));
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

__device__ __forceinline__ double coord(const Pt& p, int image, int axis) {
    return image ? (axis ? p.by : p.bx) : (axis ? p.ay : p.ax);
}

// No three of the four points (in either image) nearly collinear.
__device__ __forceinline__ bool nondegenerate(const Pt* p) {
#pragma unroll
    for (int image = 0; image < 2; ++image) {
        double scale = 0.0;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < i; ++j) {
                const double dx = coord(p[i], image, 0) - coord(p[j], image, 0);
                const double dy = coord(p[i], image, 1) - coord(p[j], image, 1);
                const double d = dx * dx + dy * dy;
                if (d > scale) scale = d;
            }
        if (!(scale > 0.0) || !fin(scale)) return false;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = i + 1; j < 4; ++j)
#pragma unroll
                for (int k = j + 1; k < 4; ++k) {
                    const double x1 = coord(p[j], image, 0) - coord(p[i], image, 0);
                    const double y1 = coord(p[j], image, 1) - coord(p[i], image, 1);
                    const double x2 = coord(p[k], image, 0) - coord(p[i], image, 0);
                    const double y2 = coord(p[k], image, 1) - coord(p[i], image, 1);
                    if (fabs(x1 * y2 - y1 * x2) <= 1e-8 * scale) return false;
                }
    }
    return true;
}

// Minimal 4-point model on one thread: the normalised normal equations of the
// design rows {x, y, 1, 0, 0, 0, -u x, -u y, u} and {0, 0, 0, x, y, 1, -v x,
// -v y, v}, Gauss-Jordan with partial pivoting, h33 = 1, denormalisation and
// scaling. The 8x9 system stays in registers: every loop is unrolled and the
// pivot row swap is a predicated select per entry, so no entry is indexed at
// run time. Operations per entry are the reference's, in its order.
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
    double m[8][9];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < 9; ++c) m[r][c] = 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double x = (p[i].bx - cbx) * sb, y = (p[i].by - cby) * sb;
        const double u = (p[i].ax - cax) * sa, v = (p[i].ay - cay) * sa;
        const double r0[9] = {x, y, 1, 0, 0, 0, -u * x, -u * y, u};
        const double r1[9] = {0, 0, 0, x, y, 1, -v * x, -v * y, v};
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
            for (int c = 0; c < 9; ++c) m[r][c] += r0[r] * r0[c] + r1[r] * r1[c];
    }
    double max_entry = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        if (fabs(m[i][i]) > max_entry) max_entry = fabs(m[i][i]);
    // A failed pivot makes the model invalid; the loop still runs to the
    // end (an early exit would stop full unrolling) and the values computed
    // after a failure are discarded.
    bool solvable = true;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        int piv = c;
        double best = fabs(m[c][c]);
        double pv = m[c][c];
#pragma unroll
        for (int r = c + 1; r < 8; ++r)
            if (fabs(m[r][c]) > best) { best = fabs(m[r][c]); piv = r; pv = m[r][c]; }
        solvable = solvable && fin(pv) && !(fabs(pv) <= 1e-12 * max_entry);
        // (loops run over all columns with a compile-time skip of jx < c, a
        // form that keeps every entry in a register after unrolling)
#pragma unroll
        for (int r = c + 1; r < 8; ++r) {
            const bool sw = r == piv;
#pragma unroll
            for (int jx = 0; jx < 9; ++jx) {
                if (jx < c) continue;
                const double a = m[c][jx], b = m[r][jx];
                m[c][jx] = sw ? b : a;
                m[r][jx] = sw ? a : b;
            }
        }
        const double div = m[c][c];
#pragma unroll
        for (int jx = 0; jx < 9; ++jx)
            if (jx >= c) m[c][jx] /= div;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            if (r == c) continue;
            const double f = m[r][c];
#pragma unroll
            for (int jx = 0; jx < 9; ++jx)
                if (jx >= c) m[r][jx] -= f * m[c][jx];
        }
    }
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

// Match i of the pair: from the staged float4 copy when it is staged.
__device__ __forceinline__ Pt point_at(const PairIO& j, const float4* pts, int i) {
    if (i < kStagePoints) {
        const float4 q = pts[i];
        return Pt{q.x, q.y, q.z, q.w};
    }
    return gather(j, i);
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
__global__ __launch_bounds__(256) void prepare_kernel(const __grid_constant__ Src src) {
    __shared__ int go, bad;
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
    __syncthreads();
    if (!go) return;
    const int na = s->na, nb = s->nb, nm = s->nm;
    for (int i = threadIdx.x; i < nm; i += blockDim.x) {
        const int ia = j.m.idx_a[i], ib = j.m.idx_b[i];
        if (ia < 0 || ia >= na || ib < 0 || ib >= nb) { bad = 1; continue; }
        const Pt q = gather(j, i);
        if (!fin(q.ax) || !fin(q.ay) || !fin(q.bx) || !fin(q.by)) bad = 1;
    }
    __syncthreads();
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
// sample, the degeneracy test, the 4-point fit and the domain test, the same
// functions the search runs in place, into prefit[h - first] (valid = 0 for
// a rejected sample). A thread owns the whole 8x9 system, so this kernel
// runs with all the registers it needs, apart from the scoring.
template <class Src>
__global__ __launch_bounds__(kFitThreads) void fit_kernel(const __grid_constant__ Src src) {
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
        const int nm = s->nm;
        int idx[4] = {0, 0, 0, 0};
        sample_four(nm, j.c.seed, h, idx);
        Pt f[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) f[k] = gather(j, idx[k]);
        m.valid = nondegenerate(f) && fit4_regs(f, m.h) && valid_domain(m.h, s->scale_b.work_w, s->scale_b.work_h);
    }
    sj.prefit[h - sj.first] = m;
}

// Block b of a pair walks warp rounds b*8 + w, b*8 + w + 8*blocks, ...; a
// round is HPW consecutive hypotheses. The block's best model goes to
// block_best[b].
// Three blocks per SM: the register-resident 4-point fit then spills to
// L1-backed local memory, but it is a small share of the work, and the
// scoring loop gains the occupancy (1 block: 0.62 ms, 3 blocks: 0.43 ms for
// 64 pairs x 2000 hypotheses x ~530 matches).
constexpr int kPruneEvery = 128;  // points between the pruning checks of a model (multiple of 128)

// kPrefit: the models come from fit_kernel (sj.prefit) and the kernel only
// scores (batched form: 0.387 -> 0.367 ms per step with the fit kernel
// included; 4 and 5 blocks per SM spill in the scoring loop and are slower).
template <class Src, bool kPrefit>
__global__ __launch_bounds__(kSearchThreads, 3) void search_kernel(const __grid_constant__ Src src) {
    extern __shared__ float4 pts[];
    __shared__ Model warp_best[kSearchWarps];
    SearchJob sj;
    int block;
    if (!src.find(blockIdx.x, &sj, &block)) return;
    const PairIO& j = sj.io;
    const State* s = j.state;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // the warp's best model so far lives in shared memory, written by lane 0
    // (registers stay with the scoring loop)
    Model& best = warp_best[warp];
    if (lane == 0) best.valid = 0;
    __syncwarp();
    const bool ok = s->status == static_cast<int>(Status::OK);
    const int nm = ok ? s->nm : 0;
    const int staged = min(nm, kStagePoints);
    for (int i = threadIdx.x; i < staged; i += kSearchThreads) {
        const int ia = j.m.idx_a[i], ib = j.m.idx_b[i];
        pts[i] = make_float4(j.a.x[ia], j.a.y[ia], j.b.x[ib], j.b.y[ib]);
    }
    __syncthreads();
    if (ok) {
        const double thr2 = j.c.threshold * j.c.threshold;
        const int bw = s->scale_b.work_w, bh = s->scale_b.work_h;
        const std::uint64_t seed = j.c.seed;
        const int hpw = j.hpw;
        const int rounds = (sj.count + hpw - 1) / hpw;
        const int stride = j.search_blocks * kSearchWarps;
        for (int round = block * kSearchWarps + warp; round < rounds; round += stride) {
            const int h0 = sj.first + round * hpw;
            const int hend = min(sj.first + sj.count, h0 + hpw);
            // lanes 0..hpw-1 build one model each (system in registers)
            double hm[9];
            int valid = 0;
            if (kPrefit) {
                valid = lane < hend - h0 ? sj.prefit[h0 + lane - sj.first].valid : 0;
            } else if (lane < hend - h0) {
                int idx[4] = {0, 0, 0, 0};
                sample_four(nm, seed, h0 + lane, idx);
                Pt f[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (idx[k] < kStagePoints) {
                        const float4 q = pts[idx[k]];
                        f[k] = Pt{q.x, q.y, q.z, q.w};
                    } else {
                        f[k] = gather(j, idx[k]);
                    }
                }
                valid = nondegenerate(f) && fit4_regs(f, hm) && valid_domain(hm, bw, bh);
            }
            // then the whole warp scores the valid models one by one
            for (int k = 0; k < hend - h0; ++k) {
                if (!__shfl_sync(0xffffffffu, valid, k)) continue;
                double h[9];
                if (kPrefit) {
                    const Model& mk = sj.prefit[h0 + k - sj.first];  // the same address on every lane
#pragma unroll
                    for (int e = 0; e < 9; ++e) h[e] = mk.h[e];
                } else {
#pragma unroll
                    for (int e = 0; e < 9; ++e) h[e] = __shfl_sync(0xffffffffu, hm[e], k);
                }
                // Exact pruning against the smallest loss of a fully scored
                // model so far (this warp's best, or the pair's bound that
                // every warp publishes to): every term is >= 0 and a
                // correctly rounded sum of nonnegative values is nondecreasing
                // in each operand, so the tree sum of the partial accumulators
                // never exceeds the final loss. Once it is above that loss the
                // model cannot win (ties need equal losses).
                const double shared_bound =
                    __longlong_as_double(static_cast<long long>(*reinterpret_cast<volatile unsigned long long*>(&j.state->bound)));
                const double bound = best.valid && best.loss < shared_bound ? best.loss : shared_bound;
                const bool prune = bound <= DBL_MAX;
                // Lane l accumulates the points l, l+32, l+64, l+96 (virtual
                // lanes, slots 0..3) and every 128 after them in order: four
                // points per step, four independent FP64 chains. A point past
                // nm adds +0.0, which leaves a sum of nonnegative terms
                // (started at +0.0) bit for bit unchanged.
                double acc0 = 0.0, acc1 = 0.0, acc2 = 0.0, acc3 = 0.0;
                bool lost = false;
                for (int base = 0; base < nm; base += 128) {  // warp-uniform trip count
                    const int i0 = base + lane, i1 = i0 + 32, i2 = i0 + 64, i3 = i0 + 96;
                    if (base + 128 <= nm) {  // every slot of the step holds a point
                        const Pt p0 = point_at(j, pts, i0), p1 = point_at(j, pts, i1);
                        const Pt p2 = point_at(j, pts, i2), p3 = point_at(j, pts, i3);
                        const double r0 = residual2(h, p0), r1 = residual2(h, p1);
                        const double r2 = residual2(h, p2), r3 = residual2(h, p3);
                        acc0 += r0 < thr2 ? r0 : thr2;
                        acc1 += r1 < thr2 ? r1 : thr2;
                        acc2 += r2 < thr2 ? r2 : thr2;
                        acc3 += r3 < thr2 ? r3 : thr2;
                    } else {
                        // the last, partial step: a virtual lane past nm adds
                        // +0.0, a no-op on a sum of nonnegative terms, so the
                        // chains with no point left (warp-uniform) are skipped
                        const double r0 = residual2(h, point_at(j, pts, min(i0, nm - 1)));
                        acc0 += i0 < nm ? (r0 < thr2 ? r0 : thr2) : 0.0;
                        if (base + 32 < nm) {
                            const double r1 = residual2(h, point_at(j, pts, min(i1, nm - 1)));
                            acc1 += i1 < nm ? (r1 < thr2 ? r1 : thr2) : 0.0;
                        }
                        if (base + 64 < nm) {
                            const double r2 = residual2(h, point_at(j, pts, min(i2, nm - 1)));
                            acc2 += i2 < nm ? (r2 < thr2 ? r2 : thr2) : 0.0;
                        }
                        if (base + 96 < nm) {
                            const double r3 = residual2(h, point_at(j, pts, min(i3, nm - 1)));
                            acc3 += i3 < nm ? (r3 < thr2 ? r3 : thr2) : 0.0;
                        }
                    }
                    if (prune && (base & (kPruneEvery - 1)) == kPruneEvery - 128 && base + 128 < nm) {
                        double part = (acc0 + acc2) + (acc1 + acc3);
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
                        if (__shfl_sync(0xffffffffu, part > bound ? 1 : 0, 0)) {
                            lost = true;
                            break;
                        }
                    }
                }
                if (lost) continue;
                // virtual lanes l, l+32, l+64, l+96: strides 64 and 32 of the tree
                double v = (acc0 + acc2) + (acc1 + acc3);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
                if (lane == 0) {
                    Model cand;
#pragma unroll
                    for (int e = 0; e < 9; ++e) cand.h[e] = h[e];
                    cand.loss = v;
                    cand.hypothesis = h0 + k;
                    cand.valid = fin(v);
                    if (better(cand, best)) best = cand;
                    if (cand.valid) atomicMin(&j.state->bound, static_cast<unsigned long long>(__double_as_longlong(v)));
                }
                __syncwarp();
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        Model b = warp_best[0];
        for (int w = 1; w < kSearchWarps; ++w)
            if (better(warp_best[w], b)) b = warp_best[w];
        j.block_best[block] = b;
    }
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
