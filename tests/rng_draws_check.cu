// Host check of every width of the transport kernels' generator and of its
// unchecked draws: RngW<16> (photon kernel), RngW<32> (electron kernel) and
// RngLocal (source kernel, precision split).  Look-aheads up to the widest that
// the window takes (W - 3 numbers), ensure(), get()/get2() within what they made
// present, checked draws, dropped windows, copies and restored copies, in random
// order: every number equals word n & 3 of block n >> 2 of the lazily computed
// Philox stream, and nothing made present is computed again.  Built and run by
// test_rng_draws.py.
#include <cstdio>
#include "egs_device.cuh"

namespace egsgpu {
static int g_fills = 0;   // blocks computed outside a look-ahead
static __host__ __device__ __noinline__ uint4 philox_block(uint32_t b, uint32_t s0, uint32_t s1, uint32_t k0,
                                                           uint32_t k1) {
#ifndef __CUDA_ARCH__
    ++g_fills;
#endif
    uint32_t o[4];
    philox10(b, s0, s1, 0u, k0, k1, o);
    return make_uint4(o[0], o[1], o[2], o[3]);
}
}  // namespace egsgpu

using namespace egsgpu;

static unsigned long long lcg = 0x9e3779b97f4a7c15ull;
static uint32_t pick(uint32_t m) {
    lcg = lcg * 6364136223846793005ull + 1442695040888963407ull;
    return (uint32_t)(lcg >> 33) % m;
}

// L: numbers of the widest look-ahead; own: get() relies on what is present (RngLocal's checks)
template <class R, int L, bool own>
static int check(const char *name, long long &unchecked) {
    for (int trial = 0; trial < 3000; ++trial) {
        const uint32_t seed = 1 + pick(1000), hist = pick(1u << 30);
        const uint64_t sid = ((uint64_t)pick(1u << 30) << 32) | pick(1u << 30);
        R r;
        r.init(seed, hist, sid, pick(64));
        R saved = r;
        int present = 0;   // numbers that the calls so far guarantee
        auto same = [&](float v, uint32_t n) {
            uint32_t o[4];
            philox10(n >> 2, (uint32_t)sid, (uint32_t)(sid >> 32), 0u, seed, hist, o);
            return v == ((float)(o[n & 3u] >> 9) + 0.5f) * (1.0f / 8388608.0f);
        };
        for (int op = 0; op < 300; ++op) {
            const uint32_t k = pick(16), n = r.n;
            const int before = g_fills;
            bool ok = true;
            int drawn = 0;
            if (k < 2) {
                const int want = 1 + pick(L);
                r.ahead(want);
                present = want > present ? want : present;
            } else if (k < 4) {
                const int want = 1 + pick(L);
                r.ensure(want);
                if (own) present = want > present ? want : present;
            } else if (k < 8 && present >= 1) {
                ok = same(r.get(), n);
                drawn = 1;
                ++unchecked;
            } else if (k < 11 && present >= 2) {
                const float2 v = r.get2();
                ok = same(v.x, n) && same(v.y, n + 1);
                drawn = 2;
                unchecked += 2;
            } else if (k < 12) {
                ok = same(r.u(), n);
                drawn = 1;
            } else if (k < 13) {
                const float2 v = r.u2();
                ok = same(v.x, n) && same(v.y, n + 1);
                drawn = 2;
            } else if (k == 13) {
                r.drop();
                present = 0;
            } else if (k == 14) {   // a copy continues the stream but holds no window
                R c = r;
                r = c;
                present = 0;
            } else if (pick(2)) {   // back to an earlier copy
                r = saved;
                present = 0;
            } else saved = r;
            if (!ok || (drawn && r.n != n + drawn)) { printf("%s: draw %u differs\n", name, n); return 1; }
            if (drawn && drawn <= present && g_fills != before) { printf("%s: draw %u computed a block\n", name, n); return 1; }
            present = present > drawn ? present - drawn : 0;
        }
    }
    return 0;
}

int main() {
    long long n16 = 0, n32 = 0, nl = 0;
    if (check<RngW<16>, 13, true>("RngW<16>", n16) || check<RngW<32>, 29, true>("RngW<32>", n32) ||
        check<RngLocal, 29, false>("RngLocal", nl)) return 1;
    printf("ok %lld %lld %lld\n", n16, n32, nl);
    return 0;
}
