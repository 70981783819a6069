// walk_to_end on the host: the walk's end by a cycle against the plain loop of
// iterations, over made-up walks.  The iteration is replaced (an explicit
// specialisation for method bits that no caller has) by a step along a chain of
// states that runs into a cycle; each state says which voxel it is in, whether
// its t_max are those formed from the voxel, and the t that a step into it
// sets.  walk_to_end must end every such walk as the plain loop does: same
// result, same iteration count.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

// what the header takes from the device
using std::max;
using std::min;
template <typename T>
static T __ldg(const T *p) { return *p; }
static int __float2int_rz(float x) { return (int)x; }
static int __float2int_rd(float x) { return (int)std::floor(x); }
static int __ffs(int v) { return __builtin_ffs(v); }
static int __ffsll(long long v) { return __builtin_ffsll(v); }
static unsigned __activemask() { return 1u; }
static uint32_t __shfl_sync(unsigned, uint32_t v, int) { return v; }
static int __all_sync(unsigned, int p) { return p; }
static uint32_t __float_as_uint(float f) {
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return u;
}
static unsigned long long atomicAdd(unsigned long long *p, unsigned long long v) { return *p += v; }

#include "vx_walk.cuh"

namespace {
struct Node {
    int32_t voxel;
    bool formed;      // t_max as formed from the voxel
    bool step;        // the move into it is a step, which sets t
    float t;
};
struct Chain {
    std::vector<Node> nodes;
    uint32_t tail;    // nodes[tail..] repeat
    uint32_t at;
};
Chain g_chain;

void enter(vx::Walk &k, const Node &n, bool trace) {
    k.s.vx = n.voxel;
    k.s.mx = (float)(n.voxel + 1) + (n.formed ? 0.0f : 0.25f);
    k.s.my = k.s.mz = 1.0f;
    k.la = 0;
    if (trace) k.t_cur = n.formed ? k.s.mx - 1.0f : n.t;
    else if (n.step) k.t_cur = n.t;
}
vx::Walk start(uint32_t cap, float tmax, bool trace) {
    vx::Walk k{};
    k.s.ix = k.s.iy = k.s.iz = 1.0f;
    k.s.stx = k.s.sty = k.s.stz = 1;
    k.s.pmx = k.s.pmy = k.s.pmz = -1;
    k.tmax = tmax;
    k.cap = cap;
    k.kind = trace ? vx::KIND_TRACE : vx::KIND_NO_WATER;
    g_chain.at = 0;
    enter(k, g_chain.nodes[0], trace);
    return k;
}
int move(vx::Walk &k, bool trace) {
    if (k.iters >= k.cap) return vx::WALK_CAP;
    ++k.iters;
    if (k.t_cur > k.tmax) return vx::WALK_END;
    if (++g_chain.at == g_chain.nodes.size()) g_chain.at = g_chain.tail;
    enter(k, g_chain.nodes[g_chain.at], trace);
    return vx::WALK_CONT;
}
constexpr uint32_t kTestFl = 1u << 20;
}  // namespace

namespace vx {
namespace {
template <>
int walk_step<kTestFl, false, (int)KIND_NO_WATER>(const DevWorld &, const Geo &,
                                                  const VxTraceParams &, Ro, Walk &k, Hit &,
                                                  uint64_t &) {
    return move(k, false);
}
template <>
int walk_step<kTestFl, false, (int)KIND_TRACE>(const DevWorld &, const Geo &, const VxTraceParams &,
                                               Ro, Walk &k, Hit &, uint64_t &) {
    return move(k, true);
}
}  // namespace
}  // namespace vx

namespace {
long g_walks = 0, g_bad = 0, g_short = 0;
template <int KIND>
void compare(uint32_t cap, float tmax) {
    const bool trace = KIND == (int)vx::KIND_TRACE;
    const vx::DevWorld w{};
    const vx::Geo g{};
    const VxTraceParams p{};
    vx::Hit h{};
    uint64_t bytes = 0;
    vx::Walk a = start(cap, tmax, trace);
    int ra;
    while ((ra = move(a, trace)) == vx::WALK_CONT) {
    }
    vx::Walk b = start(cap, tmax, trace);
    const int rb = vx::walk_to_end<kTestFl, false, KIND>(w, g, p, vx::Ro{0, 0, 0}, b, h, bytes);
    ++g_walks;
    if (ra == vx::WALK_END) ++g_short;
    if (a.iters != b.iters || (ra == vx::WALK_END) != (rb == vx::WALK_END) || b.cap != cap) {
        if (++g_bad <= 5)
            std::printf("kind %d cap %u tmax %g tail %u cycle %zu: plain %d at %u, got %d at %u\n",
                        KIND, cap, tmax, g_chain.tail, g_chain.nodes.size() - g_chain.tail, ra,
                        a.iters, rb, b.iters);
    }
}
void both(uint32_t cap, float tmax) {
    compare<(int)vx::KIND_NO_WATER>(cap, tmax);
    compare<(int)vx::KIND_TRACE>(cap, tmax);
}
}  // namespace

int main() {
    // a cycle of every length first entered at every iteration around the first
    // looks, whose last move is a step that sets a t of its own
    for (uint32_t tail = 170; tail < 260; ++tail)
        for (uint32_t len = 1; len <= 130; ++len)
            for (int past = 0; past < 2; ++past) {
                g_chain = Chain{{}, tail, 0};
                for (uint32_t i = 0; i < tail + len; ++i)
                    g_chain.nodes.push_back({(int32_t)i, true, false, 0.0f});
                // the cycle comes back into its first state by the step: the
                // state is entered without it once, from the tail
                Node back = g_chain.nodes[tail];
                back.step = true;
                back.t = past ? 2.0f : 0.5f;
                g_chain.nodes.push_back(back);
                g_chain.tail = tail + 1;
                if (len == 1) g_chain.nodes[tail + 1].step = true, g_chain.nodes[tail + 1].t = back.t;
                both(1024, 1.0f);
            }
    // random chains
    std::mt19937 rng(1);
    auto u = [&](uint32_t n) { return (uint32_t)(rng() % n); };
    for (int i = 0; i < 200000; ++i) {
        const uint32_t tail = u(400), lens[6] = {1, 2, 3, 1 + u(8), 60, 1 + u(200)},
                       len = lens[u(6)];
        g_chain = Chain{{}, tail, 0};
        const uint32_t formed = u(4), steps = u(4), late = u(3);
        for (uint32_t k = 0; k < tail + len; ++k)
            g_chain.nodes.push_back({(int32_t)k, u(4) >= formed, u(4) < steps,
                                     late == 0 && u(64) == 0 ? 2.0f : 0.5f});
        both(u(2) ? 1024 : 1 + u(1200), 1.0f);
    }
    std::printf("%ld walks, %ld ended by t, %ld differ\n", g_walks, g_short, g_bad);
    return g_bad == 0 ? 0 : 1;
}
