/* Host model of what unit_sync.cuh orders: a warp's barrier counted against its
 * votes, and tensor memory whose loads and stores take effect only when they
 * are waited for. Prints what was out of order; exits 0 if nothing was. */
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>

#define __device__
#define __host__
#define __forceinline__ inline
using std::fabs;
static size_t __cvta_generic_to_shared(const void* p) { return (size_t)p; }
static unsigned atomicOr(unsigned* p, unsigned v) { unsigned o = *p; *p |= v; return o; }

/* accesses to shared memory since the last barrier of the warp */
static int unordered = 0, wrong = 0;
static void access() { unordered = 1; }
static void __syncwarp() { unordered = 0; }
static void voted(const char* what)
{
    if (unordered) std::printf("%s: no barrier between the accesses before it and those after it\n", what), wrong++;
    unordered = 0;
}
static unsigned __reduce_or_sync(unsigned, unsigned v) { voted("vote"); return v; }
static int __any_sync(unsigned, bool f) { voted("any"); return f; }

#define WLDPC_TMEM_CUH   /* in place of tmem.cuh */
namespace wldpc {
struct Tmem {
    uint32_t column[512];
    bool in_flight[512];
    uint32_t coming[512];   /* value of a store that was not waited for */
    int loading = 0;
} tm;
static void store(uint32_t a, uint32_t v)
{
    if (tm.in_flight[a] && tm.coming[a] != v)
        std::printf("column %u: %u stored over a store of %u in flight\n", a, v, tm.coming[a]), wrong++;
    tm.in_flight[a] = true;
    tm.coming[a] = v;
}
static void tm_st8(const uint32_t* r, uint32_t a) { for (int i = 0; i < 8; i++) store(a + i, r[i]); }
static void tm_wait_st()
{
    for (int a = 0; a < 512; a++) {
        if (tm.in_flight[a]) tm.column[a] = tm.coming[a];
        tm.in_flight[a] = false;
    }
}
template <int D> void tm_ld(uint32_t* r, uint32_t a)
{
    for (int i = 0; i < D; i++) {
        if (tm.in_flight[a + i]) std::printf("column %u: loaded under a store in flight\n", a + i), wrong++;
        r[i] = tm.column[a + i];
    }
    tm.loading = D;
}
template <int D, int N> void tm_wait_ld(uint32_t (&)[N]) { tm.loading = 0; }
}  // namespace wldpc

#include "unit_sync.cuh"

using namespace wldpc;

static void votes()
{
    unsigned words[4] = {0, 0, 0, 0};
    UnitSync<1> unit{words, 0, 0};
    access();   /* a layer's last stores */
    unit.vote(1u);
    access();
    unit.any(true);
}

/* a unit that starts its next frames right after the last layer's stores */
template <int R> static void clear()
{
    constexpr int NBLK = num_blocks(R), last = layer_degree(R, kMb[R] - 1);
    uint32_t M[kMaxDeg] = {};
    for (int a = 0; a < 512; a++) tm.column[a] = 1000u + a;
    tm_ld<layer_degree(R, 0)>(M, 0);
    for (int a = NBLK - last; a < NBLK; a++) store(a, 7u);
    unit_clear_messages<R>(M, 0);
    tm_wait_ld<layer_degree(R, 0)>(M);
    tm_wait_st();
    for (int a = 0; a < NBLK; a++)
        if (tm.column[a]) std::printf("rate %d: message %d is %u\n", R, a, tm.column[a]), wrong++;
    for (int e = 0; e < layer_degree(R, 0); e++)
        if (M[e]) std::printf("rate %d: loaded message %d is %u\n", R, e, M[e]), wrong++;
    if (tm.column[NBLK] != 1000u + NBLK) std::printf("rate %d: a column past the messages was stored\n", R), wrong++;
}

int main(int argc, char** argv)
{
    if (argc == 2 && !std::strcmp(argv[1], "votes")) votes();
    else if (argc == 2 && !std::strcmp(argv[1], "clear")) clear<0>(), clear<1>(), clear<2>(), clear<3>(), clear<4>(), clear<5>();
    else return 2;
    return wrong ? 1 : 0;
}
