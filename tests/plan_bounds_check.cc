// Evaluates the planner's box tests (3pcf_gb300/csrc/plan_bounds.h) on random
// boxes and prints a hash of every result's bits: compilations that contract
// products and sums differently have to print the same.
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include "../3pcf_gb300/csrc/plan_bounds.h"

using namespace tpcf;

static uint64_t state = 88172645463325252ull, hash = 1469598103934665603ull;

// (volatile: the inputs themselves leave nothing to contract)
static float uniform() {
    state ^= state << 13;
    state ^= state >> 7;
    state ^= state << 17;
    return (float)(state >> 40) / 16777216.0f;
}

static void add(float v) {
    uint32_t u;
    memcpy(&u, &v, 4);
    hash = (hash ^ u) * 1099511628211ull;
}

int main() {
    PlanParams pp{};
    pp.s_lo2 = 4.0f;
    pp.s_hi2 = 100.0f;
    pp.q_hi2 = 9.0f;
    for (int n = 0; n < 200000; n++) {
        float4 lo[3], hi[3];
        for (int t = 0; t < 3; t++) {
            volatile float a[6] = {uniform() * 40, uniform() * 40, uniform() * 40, uniform() * 9, uniform() * 9, uniform() * 9};
            lo[t] = make_float4(a[0], a[1], a[2], 0.f);
            hi[t] = make_float4(a[0] + a[3], a[1] + a[4], a[2] + a[5], 0.f);
        }
        const float2 ab = box_bounds2(lo[0], hi[0], lo[1], hi[1]), ac = box_bounds2(lo[0], hi[0], lo[2], hi[2]),
                     bc = box_bounds2(lo[1], hi[1], lo[2], hi[2]);
        for (const float2& b : {ab, ac, bc}) {
            add(b.x);
            add(b.y);
            add(near_share(b, 30.0f));
        }
        add(tri_possible(ab, ac, bc, pp) ? 1.f : 0.f);
        add(add_estimate(uniform() * 1000, 1 + (float)(n % 64), 1 + (float)(n % 61), 1 + (float)(n % 59), ab, ac, bc, 30.0f));
    }
    printf("%016llx\n", (unsigned long long)hash);
    return 0;
}
