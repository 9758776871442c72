// Host-only check of the kernels that batch::Plan::build chooses for a batch:
// how the candidates are ordered and by what blocks, the rows of a resize tile. Built and run by tests/test_plan_choices.py on
// the CPU: build() with alloc_staging = false touches no device.
#include <cstdio>
#include <vector>

#include "batch.hpp"

using stitch::b200::batch::Plan;

namespace {

struct Shape {
    int pairs, w, h, k, levels;
};

bool build(const Shape& s, Plan* p) {
    static unsigned char fake[256];
    stitch_pair_desc d{};
    d.image_a = d.image_b = stitch_image_view{fake, s.w, s.h, (s.w + 15) / 16 * 16, 1};
    d.s2 = stitch_s2_config{20, s.k, 0.04f};
    d.s4.ratio_threshold = 0.8f;
    d.s5 = stitch_s5_config{500, 0, 64, 1, 3.0, 7, 1};
    d.pyramid = stitch_pyramid_config{s.levels, 1.2f};
    const std::vector<stitch_pair_desc> pairs(s.pairs, d);
    int bad = -1;
    return p->build(s.pairs, pairs.data(), &bad, false) == stitch::Status::OK;
}

int fail(const char* what, const Shape& s) {
    std::printf("%s: %d pairs of %dx%d, K = %d, %d levels\n", what, s.pairs, s.w, s.h, s.k, s.levels);
    return 1;
}

}  // namespace

int main() {
    // ranked whatever keys are there; by the keys that are there; sorted
    for (const Shape s : {Shape{1, 800, 600, 500, 1}, Shape{1, 800, 600, 8000, 1}, Shape{1, 800, 600, 8000, 8}, Shape{3, 800, 600, 2000, 8},
                          Shape{4, 800, 600, 1000, 1}, Shape{2, 800, 600, 8000, 1}}) {
        Plan p;
        if (!build(s, &p) || p.topk != Plan::kRanked) return fail("not ranked", s);
    }
    for (const Shape s : {Shape{3, 800, 600, 8000, 1}, Shape{8, 800, 600, 8000, 1}, Shape{16, 800, 600, 4000, 1}, Shape{4, 800, 600, 20000, 8},
                          Shape{6, 800, 600, 4000, 1}}) {
        Plan p;
        if (!build(s, &p) || p.topk != Plan::kByCounts) return fail("not decided by the keys", s);
    }
    for (const Shape s : {Shape{64, 512, 512, 2000, 8}, Shape{32, 800, 600, 2000, 1}, Shape{8, 800, 600, 8000, 8}}) {
        Plan p;
        if (!build(s, &p) || p.topk != Plan::kSorted) return fail("not sorted", s);
    }
    // sort blocks
    const struct {
        Shape s;
        int threads;
    } sorts[] = {{{32, 800, 600, 500, 1}, 512},  {{64, 800, 600, 256, 1}, 256},  {{8, 512, 512, 2000, 8}, 512},
                 {{64, 512, 512, 2000, 8}, 256}, {{64, 512, 512, 1000, 8}, 256}, {{32, 800, 600, 513, 1}, 1024}};
    for (const auto& c : sorts) {
        Plan p;
        if (!build(c.s, &p) || p.sort_threads != c.threads) return fail("other sort blocks", c.s);
    }
    // resize tiles: 128 rows from two waves of them on, 64 below; the tuning's value where it has one
    const struct {
        Shape s;
        int rows;
    } tiles[] = {{{2, 3700, 2159, 1000, 4}, 128}, {{2, 3700, 2100, 1000, 4}, 64}, {{64, 512, 512, 2000, 8}, 128}, {{8, 512, 512, 2000, 8}, 64}};
    for (const auto& c : tiles)
        for (const int tuned : {0, 32}) {
            Plan p;
            p.tuning.resize_tile_h = tuned;
            if (!build(c.s, &p) || p.resize_tile_h != (tuned ? tuned : c.rows)) return fail("other resize tiles", c.s);
        }
    std::printf("plan choices ok\n");
    return 0;
}
