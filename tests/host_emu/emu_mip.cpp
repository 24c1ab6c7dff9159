// emu_mip.cpp - TEST INFRASTRUCTURE: the mip generator's tile loop (zap_b200/csrc/mip.cu, up to its first kernel) as one CTA on
// the host, its threads as coroutines under a scheduler that keeps one warp back (tests/test_mip_tiles_on_host.py).
//
// A thread runs until it meets a barrier. Of the threads that can go on, those of the slow warp go last, so all that the
// kernel's barriers allow to happen before that warp's next step has happened by then: a buffer that is written again
// too early is read after it was written, every time.
#include <cuda_runtime.h>
#include <ucontext.h>

#include <algorithm>
#include <vector>

using std::max;
using std::min;

namespace emu {
constexpr int kThreads = 256, kStack = 128 << 10;
enum State { kReady, kAtCta, kAtWarp, kDone };
struct Thread {
    ucontext_t ctx;
    State state;
    std::vector<char> stack;
};
std::vector<Thread> threads(kThreads);
ucontext_t scheduler;
int current = 0;
dim3 thread_idx(0), block_idx(0), grid_dim(1);

void wait(State s) {
    const int me = current;
    threads[me].state = s;
    swapcontext(&threads[me].ctx, &scheduler);
    thread_idx.x = (unsigned)me;
}
// frees the threads [lo, hi) when every one of them that still runs waits in state s; false if some do not
bool release(int lo, int hi, State s) {
    bool any = false;
    for (int k = lo; k < hi; k++) {
        if (threads[k].state == kDone) continue;
        if (threads[k].state != s) return false;
        any = true;
    }
    for (int k = lo; k < hi; k++) if (threads[k].state == s) threads[k].state = kReady;
    return any;
}
bool run(void (*body)(), int slow_warp) {  // false: the threads wait for one another for good
    for (int k = 0; k < kThreads; k++) {
        Thread &t = threads[k];
        t.stack.resize(kStack);
        getcontext(&t.ctx);
        t.ctx.uc_stack.ss_sp = t.stack.data();
        t.ctx.uc_stack.ss_size = kStack;
        t.ctx.uc_link = &scheduler;
        t.state = kReady;
        makecontext(&t.ctx, body, 0);
    }
    for (;;) {
        int next = -1, done = 0;
        for (int k = 0; k < kThreads; k++) {
            done += threads[k].state == kDone;
            if (threads[k].state == kReady && (next < 0 || (next >> 5) == slow_warp)) next = k;
        }
        if (done == kThreads) return true;
        if (next < 0 || (next >> 5) == slow_warp) {  // nothing else can go on: barriers that are met come first
            bool freed = false;
            for (int w = 0; w < kThreads; w += 32) freed = release(w, w + 32, kAtWarp) || freed;
            freed = release(0, kThreads, kAtCta) || freed;
            if (freed) continue;
            if (next < 0) return false;
        }
        current = next;
        thread_idx.x = (unsigned)next;
        swapcontext(&scheduler, &threads[next].ctx);
        if (threads[next].state == kReady) threads[next].state = kDone;  // came back through uc_link
    }
}
}  // namespace emu

#define threadIdx emu::thread_idx
#define blockIdx emu::block_idx
#define gridDim emu::grid_dim
#define __syncthreads() emu::wait(emu::kAtCta)
#define __syncwarp() emu::wait(emu::kAtWarp)
#define __ldg(p) (*(p))

#include EMU_MIP_SOURCE

using namespace ztc;

namespace {
const MipChain *g_chains;
const MipTile *g_tiles;
int g_ntiles;
MipScratch g_scratch[2];
void body() {
    mip_tiles_of_cta(g_ntiles, NoTables{}, g_scratch, [&](int k, const MipChain *&c, int &x, int &y) {
        c = g_chains + g_tiles[k].chain; x = g_tiles[k].x; y = g_tiles[k].y;
    });
}
}  // namespace

// The tiles of n chains (linear light), in the batch's order, all by one CTA whose warp `slow_warp` is kept back. Chain i:
// a w[i] x h[i] packed source at src[i], levels[i] levels to dst[6 i + level - 1]. 0 on success.
extern "C" int emu_mip_chains(int n, const uint8_t *const *src, const int *w, const int *h, const int *levels, uint8_t *const *dst, int slow_warp) {
    std::vector<MipChain> chains(n);
    std::vector<MipTile> tiles;
    for (int i = 0; i < n; i++) {
        MipChain &c = chains[i];
        c = MipChain{};
        c.src = src[i]; c.pitch = (size_t)w[i] * 4; c.w = w[i]; c.h = h[i]; c.levels = levels[i]; c.srgb = 0;
        c.dst_pitch = (size_t)std::max(1, w[i] / 2) * 4;
        for (int l = 0; l < levels[i]; l++) c.dst[l] = dst[6 * i + l];
        const int tx = (std::max(1, w[i] / 2) + 31) / 32, ty = (std::max(1, h[i] / 2) + 31) / 32;
        for (int t = 0; t < tx * ty; t++) tiles.push_back({i, t % tx, t / tx, 0});
    }
    g_chains = chains.data(); g_tiles = tiles.data(); g_ntiles = (int)tiles.size();
    return emu::run(body, slow_warp) ? 0 : -1;
}
