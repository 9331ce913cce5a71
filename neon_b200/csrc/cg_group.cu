// cg_group.cu -- Jacobi-PCG as one persistent launch per solve (conjugate_gradient::solve,
// linear_solver.cpp:67-109): iterations, dot products and stop tests run inside one cooperative
// kernel, one CTA per SM.
//
// What bounds the small and middle systems is not bandwidth but the chain of launches: three
// kernels per iteration (SpMV, x/r update, p update), two of them ending in a last-block
// reduction, took 17-20 us per iteration whatever the size below 20^3 hex8 cells (27 us at
// 37x29x32), and up to 31 iterations past convergence ran empty.  Here a group of CTAs owns a
// system.  A CTA keeps z of every row it reads (its halo), its rows' vectors and as much of its
// rows of K as fit in shared memory; the rest of K streams from L2 through rings of bulk copies that
// run ahead across the sums, since K does not change (41 bytes per cycle and SM; ordinary coalesced
// loads, four steps in flight per warp, reached 19).
//
// An iteration sums once over the group (after Chronopoulos and Gear, J. Comput. Appl. Math. 25, 1989):
// with w = K z, s = K p follows from s = w + beta s, and, K being symmetric,
// p.s = z.w + 2 beta z.s' + beta^2 p'.s' with the last step's s' and p', so that
//   1  z of the halo, the only vector that crosses between CTAs
//   2  w = K z and z.w; one sum of z.w, r.r, r.z and z.s'                 -> stop test, beta, alpha
//   3  p = z + beta p, s = w + beta s, x += alpha p, r -= alpha s, z = D^-1 r
// z.s' is summed, not taken as -beta p'.s' as in that paper.  That shorter form assumes z.r' = 0 and
// multiplies each error of p.s by beta^2: it holds while the recurrences run from their start, but a
// launch that carries on along a kept direction (a replaced residual, a solve cut into launches) breaks
// z.r' = 0, and ill-conditioned systems (near-incompressible, bulk / shear 1e4 and more) then stagnate.
// The textbook form sums twice (p.q, then r.r and r.z); what the second sum costs is latency, the same
// at every size: 6.0 -> 5.0 us per iteration at 12^3 hex8 cells, 6.6 -> 5.6 at 20^3, 10.6 -> 9.4 at
// 28^3, 11.6 -> 11.7 at 37x29x32 (two more vectors in shared memory leave less room for K), with the
// iteration counts and the errors of before (now 4.8, 5.4, 9.1 and 11.4: fewer exchanges in a sum).  The first iteration of a launch takes the textbook form
// (s = K p, p.s), because its p may carry on from an earlier launch.
// In the sum every member adds the same numbers in the same order: all take the same decision and a
// solve is bit-reproducible.  Members exchange partial sums and z as 16-byte {value, tag} pairs, written
// and read in one access: a reader waits for the tag it expects, so nothing needs a fence or a separate
// barrier.  A z is overwritten only after the sum that follows it, to which every reader contributes
// after its reads.  Sums go over m1 CTAs, then over m2 such groups (a push to each peer's own slots):
// 2.1 k cycles for up to 16 CTAs and 3.6 k for 144, where an arrival count with release and acquire took
// 3.8 k and 4.8 k, and polling all partials in one place 9.8 k (every SM then polls the same 37 lines).
//
// Co-residency comes from the cooperative launch; every wait has a limit, after which the CTA reports
// the launch as failed and returns, leaving its system's `done` at 0.  A CTA may have to wait for members
// that still work on earlier systems.  So that such a wait has a bound that no legitimate work reaches,
// a turn ends after kTurnIterations with its state stored, and the caller launches again (a launch
// reloads K, 20 to 60 us in at least 10 ms).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#include "cg_group.cuh"

namespace nb2 {

namespace {

constexpr int kGT = 512;             // threads of a CTA
constexpr int kGW = kGT / 32;
constexpr int kStages = 2;           // chunks in flight per warp
constexpr int kCopyLimit = 1 << 22;  // tries on one bulk copy (each suspends for a while)
constexpr int kSide = 16;            // most CTAs of one level of a sum
constexpr int kValues = 4;           // values of a sum
constexpr int kSlots = 2 * 2 * kSide * kValues;  // exchange slots of a CTA
constexpr int kPollLimit = 1 << 22;  // polls of one tag inside an iteration (seconds)
constexpr int kTurnIterations = 2048;  // a system's most iterations in one launch
// polls (0.4 us and more each) for each turn that other members may still have to finish: seconds,
// where 2048 iterations take up to 1 s for the largest parts
constexpr int kStartLimit = 1 << 23;

constexpr int kLpr = 4;              // lanes per row of a tile
constexpr int B = 3;                 // block size

template <typename V>
struct Step {
    static constexpr int VB = 32 * B * B * (int)sizeof(V);  // value bytes of a step
    static constexpr int CB = 32 * 2;                       // column bytes
    static constexpr int CS = 2;                            // steps of a ring chunk
    static constexpr int RB = CS * (VB + CB);               // bytes of a ring chunk
};

// Shared memory of a part: z and the row numbers of its halo and its tiles' first steps; then as many
// of the own rows' six vectors as leave room for the rings (the others stay in global memory); then
// K, or the rings and as many steps of K as fit behind them.
constexpr int kVectors = 6;  // w, r, s, p, x, D^-1
struct PartLayout {
    bool fits;
    int vectors;             // resident ones
    int vec, bytes;          // offset of the first, bytes of each
    int ring, k, room;       // offsets; steps of K that are resident
};

template <typename V, typename X>
__host__ __device__ inline PartLayout part_layout(int nh, int nt, int nd, int steps, int bytes) {
    constexpr int step = Step<V>::VB + Step<V>::CB, rings = kGW * kStages * Step<V>::RB;
    const long long p = ((long long)(sizeof(X) * B + 4) * nh + 4ll * (nt + 1) + 127) / 128 * 128;
    const long long one = ((long long)sizeof(X) * nd + 127) / 128 * 128;
    PartLayout L;
    L.fits = p + rings <= bytes;
    L.vectors = kVectors;
    while (L.vectors > 0 && p + L.vectors * one + rings > bytes) --L.vectors;
    L.vec = (int)p;
    L.bytes = (int)one;
    L.ring = (int)(p + L.vectors * one);
    const bool all = L.ring + (long long)steps * step <= bytes;
    L.k = all ? L.ring : L.ring + rings;
    L.room = all ? steps : (bytes - L.k) / step;
    return L;
}

template <typename V, typename X>
struct GroupArgs {
    const int *tile_row, *tile_end, *tile_off, *part_tile, *halo_ptr, *halo, *own0;
    const unsigned short* col;
    const V* val;
    const GroupTurn* turns;
    const int* turn_ptr;
    X *x, *r, *p, *w, *s;
    double* z;
    const X* inv;
    const float* dc;
    GroupScalars S;
    double* slots;   // per member [2 levels][2 parities][kSide][kValues]{value, tag}
    unsigned long long tag0;  // of this launch
    unsigned *failed, launch;  // *failed = launch: a wait of this launch ran out
    int start_limit;
    int smem_bytes;  // all of the dynamic shared memory
};

struct GroupShared {
    double red[2][kValues][kGW];  // by parity: one barrier per sum orders its reuse in a group of one
    double sum[kValues];
    unsigned long long bar[kGW][kStages];
    int failed;
    const unsigned* failed_launch;  // GroupArgs::failed, launch
    unsigned launch;
};

// {value, tag} in one 16-byte access
__device__ __forceinline__ void tag_store(double* a, double v, unsigned long long tag) {
    asm volatile(
        "{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::
            "l"(a),
        "l"(__double_as_longlong(v)), "l"(tag)
        : "memory");
}
__device__ __forceinline__ void tag_load(const double* a, double& v, unsigned long long& tag) {
    long long lo;
    asm volatile(
        "{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
        : "=l"(lo), "=l"(tag)
        : "l"(a)
        : "memory");
    v = __longlong_as_double(lo);
}

// whether a wait of this launch ran out somewhere; looked at now and then
__device__ __forceinline__ bool others_failed(int polls, const unsigned* failed, unsigned launch) {
    return (polls & 1023) == 1023 && *(const volatile unsigned*)failed == launch;
}

// One level of a sum, by one warp for two values: lane (h, j) = (lane / 16, lane % 16) sends its value
// h to member j's slots and waits for member j's; every lane returns the sum of value h over the n
// members.
__device__ __forceinline__ double level_sum(double* to, const double* from, double v, bool on,
                                            unsigned long long tag, int limit, GroupShared& sh) {
    if (on) tag_store(to, v, tag);
    double got = 0.0;
    unsigned long long t = tag;
    for (int k = 0;; ++k) {
        if (on) tag_load(from, got, t);
        if (__all_sync(0xffffffffu, t == tag)) break;
        if (__any_sync(0xffffffffu, k > limit || others_failed(k, sh.failed_launch, sh.launch))) {
            sh.failed = 1;
            break;
        }
    }
    double a = on ? got : 0.0;
#pragma unroll
    for (int o = kSide / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
}

// Sum of v over all threads of the group, the same bits in every CTA; warp 0 sends the first two
// values, warp 1 the others.  False when a wait ran out.
__device__ __forceinline__ bool group_sum(GroupShared& sh, double* slots, const GroupTurn& g,
                                          unsigned long long tag, int limit,
                                          double (&v)[kValues]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int par = (int)(tag & 1);
    double(&red)[4][kGW] = sh.red[par];
    static_assert(kGW == kSide && kValues == 4, "the lanes' shares of the four values");
    // a lane hands on what it does not keep: after two steps each quarter of the warp holds one value
    // (6 exchanges instead of 20; a system on one CTA waits for them in every iteration)
    const bool half = (lane & 16) != 0, quarter = (lane & 8) != 0;
    const double s0 = (half ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, half ? v[0] : v[2], 16);
    const double s1 = (half ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, half ? v[1] : v[3], 16);
    double t = (quarter ? s1 : s0) + __shfl_xor_sync(0xffffffffu, quarter ? s0 : s1, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((lane & 7) == 0) red[lane >> 3][warp] = t;
    __syncthreads();
    const int j = lane & 15;
    if (g.m1 == 1) {  // alone: every warp adds the warps' sums itself, a quarter for each value
        double a = red[lane >> 3][lane & 7] + red[lane >> 3][8 + (lane & 7)];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
#pragma unroll
        for (int k = 0; k < kValues; ++k) v[k] = __shfl_sync(0xffffffffu, a, 8 * k);
        return !sh.failed;
    }
    if (warp < 2) {
        const int h = 2 * warp + (lane >> 4);
        double a = red[h][j];
#pragma unroll
        for (int o = kGW / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        const int row = g.rank / g.m1, i = g.rank - row * g.m1;
        auto slot = [&](int member, int level, int from) {
            return slots + 2ll * (member * kSlots + ((level * 2 + par) * kSide + from) * kValues + h);
        };
        a = level_sum(slot(row * g.m1 + j, 0, i), slot(g.rank, 0, j), a, j < g.m1, tag, limit,
                      sh);
        if (g.m2 > 1)
            a = level_sum(slot(j * g.m1 + i, 1, row), slot(g.rank, 1, j), a, j < g.m2, tag, limit,
                          sh);
        if (j == 0) sh.sum[h] = a;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kValues; ++k) v[k] = sh.sum[k];
    return !sh.failed;
}

__device__ __forceinline__ unsigned smem_addr(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

// one lane's share of w = K z for one step: the entry's block times its column's z
template <typename V, typename X>
__device__ __forceinline__ void step_product(const V* v, int c, const X* p, X (&y)[B]) {
    X pn[B];
#pragma unroll
    for (int k = 0; k < B; ++k) pn[k] = p[B * c + k];
#pragma unroll
    for (int i = 0; i < B; ++i) {
        X t = (X)v[(i * B) * 32] * pn[0];
#pragma unroll
        for (int k = 1; k < B; ++k) t += (X)v[(i * B + k) * 32] * pn[k];
        y[i] += t;
    }
}

// A warp's stream of K: its steps [first, first + steps), again and again, in chunks of CS steps
// through kStages places in shared memory.  Lane 0 issues; chunk n (counted over the kernel's
// life) goes to place n % kStages in its (n / kStages)-th phase.
template <typename V>
struct Ring {
    using S = Step<V>;
    unsigned char* buf;  // [kStages][RB]
    unsigned long long* bar;
    const V* val;
    const unsigned short* col;
    int first, steps, chunks;
    unsigned issued, used;  // chunks
    int next;               // position in the stream of the next chunk to issue

    __device__ void issue() {
        const unsigned st = issued % kStages;
        const int s0 = next * S::CS, n = min(S::CS, steps - s0);
        const unsigned mb = smem_addr(bar + st);
        unsigned char* dst = buf + st * S::RB;
        const long long from = first + s0;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb),
                     "r"(n * (S::VB + S::CB))
                     : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
            "[%3];" ::"r"(smem_addr(dst)),
            "l"(val + from * (32 * B * B)), "r"(n * S::VB), "r"(mb)
            : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
            "[%3];" ::"r"(smem_addr(dst + S::CS * S::VB)),
            "l"(col + from * 32), "r"(n * S::CB), "r"(mb)
            : "memory");
        ++issued;
        next = next + 1 == chunks ? 0 : next + 1;
    }

    // the oldest chunk in flight has arrived; false when it did not within the limit
    __device__ bool wait() const {
        const unsigned mb = smem_addr(bar + used % kStages), phase = (used / kStages) & 1;
        for (int n = 0; n < kCopyLimit; ++n) {
            unsigned ok;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(ok)
                : "r"(mb), "r"(phase)
                : "memory");
            if (ok) return true;
        }
        return false;
    }
};

template <typename V, typename X>
__global__ void __launch_bounds__(kGT, 1) k_group_cg(GroupArgs<V, X> A) {
    using S = Step<V>;
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ GroupShared sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ri = lane / kLpr, sl = lane % kLpr;
    if (tid == 0) {
        sh.failed = 0;
        sh.failed_launch = A.failed;
        sh.launch = A.launch;
    }
    if (tid < kGW * kStages)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sh.bar[0][0] + tid))
                     : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    unsigned chunks_used = 0;
    for (int turn = A.turn_ptr[blockIdx.x]; turn < A.turn_ptr[blockIdx.x + 1]; ++turn) {
        const GroupTurn g = A.turns[turn];
        const int job = g.job;
        if (A.S.done[job]) continue;
        unsigned long long tag = A.tag0;  // counts the sums of this turn
        const bool alone = g.m1 == 1;
        double* slots = A.slots + 2ll * g.slot0;
        // this part's tiles, rows, unknowns and halo
        const int tb = A.part_tile[g.part], te = A.part_tile[g.part + 1];
        const int row0 = A.tile_row[tb], row1 = A.tile_end[te - 1];
        const long long d0 = (long long)B * row0;
        const int nd = B * (row1 - row0);
        const int h0 = A.halo_ptr[g.part], nh = A.halo_ptr[g.part + 1] - h0;
        const int own = A.own0[g.part], nown = row1 - row0, pown = B * own;
        const int off0 = A.tile_off[tb], nsteps = A.tile_off[te] - off0;
        const PartLayout lay = part_layout<V, X>(nh, te - tb, nd, nsteps, A.smem_bytes);
        if (!lay.fits) {  // the plan checked every part
            if (tid == 0) *(volatile unsigned*)A.failed = A.launch;
            break;
        }
        X* sp = reinterpret_cast<X*>(dyn);  // z of the halo (p in the first iteration)
        int* shalo = reinterpret_cast<int*>(sp + (size_t)B * nh);
        int* soff = shalo + nh;
        auto vector = [&](int k, X* global) {
            return k < lay.vectors ? reinterpret_cast<X*>(dyn + lay.vec + k * lay.bytes)
                                   : global + d0;
        };
        X *vw = vector(0, A.w), *vr = vector(1, A.r), *vs = vector(2, A.s), *vp = vector(3, A.p),
          *vx = vector(4, A.x);
        const X* vi = vector(5, const_cast<X*>(A.inv));
        unsigned char* kbuf = dyn + lay.k;
        int tr = tb;  // tiles [tb, tr) are resident
        while (tr < te && A.tile_off[tr + 1] - off0 <= lay.room) ++tr;
        const int rsteps = A.tile_off[tr] - off0;
        const V* sval = reinterpret_cast<const V*>(kbuf);
        const unsigned short* scol =
            reinterpret_cast<const unsigned short*>(kbuf + (size_t)rsteps * S::VB);
        // this warp's share of the streamed tiles, and the first chunks on their way
        const int ts0 = tr + (int)((long long)(te - tr) * warp / kGW);
        const int ts1 = tr + (int)((long long)(te - tr) * (warp + 1) / kGW);
        Ring<V> ring;
        ring.buf = dyn + lay.ring + warp * (kStages * S::RB);
        ring.bar = sh.bar[warp];
        ring.val = A.val;
        ring.col = A.col;
        ring.first = A.tile_off[ts0];
        ring.steps = A.tile_off[ts1] - ring.first;
        ring.chunks = (ring.steps + S::CS - 1) / S::CS;
        ring.issued = ring.used = chunks_used;
        ring.next = 0;
        const bool streams = ring.steps > 0;
        // the turn before read this memory with ordinary loads
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (streams && lane == 0)
            for (int k = 0; k < kStages; ++k) ring.issue();
        {
            const uint4* src = reinterpret_cast<const uint4*>(A.val + (long long)off0 * B * B * 32);
            uint4* dst = reinterpret_cast<uint4*>(kbuf);
            const int n16 = rsteps * (S::VB / 16);
            for (int i = tid; i < n16; i += kGT) dst[i] = src[i];
            const uint4* cs = reinterpret_cast<const uint4*>(A.col + (long long)off0 * 32);
            uint4* cd = dst + n16;
            for (int i = tid; i < rsteps * (S::CB / 16); i += kGT) cd[i] = cs[i];
        }
        for (int t = tb + tid; t <= te; t += kGT) soff[t - tb] = A.tile_off[t] - off0;
        double absnew = A.S.absnew[job], beta = A.S.beta[job], rr = A.S.rr[job];
        X bx = (X)beta;
        for (int i = tid; i < nh; i += kGT) {
            const int a = A.halo[h0 + i];
            shalo[i] = a;
            if (i < own || i >= own + nown)
#pragma unroll
                for (int k = 0; k < B; ++k) sp[B * i + k] = A.p[(long long)B * a + k];
        }
        for (int i = tid; i < nd; i += kGT) {
            const X r0 = A.r[d0 + i], iv = A.inv[d0 + i], z0 = iv * r0;
            if (!alone) tag_store(A.z + 2 * (d0 + i), (double)z0, tag + 1);
            sp[pown + i] = z0 + bx * A.p[d0 + i];
            if (lay.vectors > 1) vr[i] = r0;
            if (lay.vectors > 4) vx[i] = A.x[d0 + i];
            if (lay.vectors > 5) const_cast<X*>(vi)[i] = iv;
        }
        const double thr = A.S.thr[job], rrcap = A.S.rrcap[job];
        int iters = A.S.iters[job], status = 0;
        const int maxit = A.S.maxit[job], begun = iters;
        double v[kValues] = {0.0, 0.0, 0.0, 0.0}, pq = 0.0;
        bool first = true, paused = false;
        // the members may come from other systems: a longer wait until all are here
        int limit = A.start_limit;
        bool ok = true;
        __syncthreads();
        for (;;) {
            // 1: z of the halo (in the first iteration p, which may carry on from an earlier launch)
            ++tag;
            if (!alone) {
                constexpr int U = 6;  // loads in flight (4: +3% at 33^3, 8: +8% at 20^3)
                const int outer = B * nh - nd;
                for (int i0 = tid; i0 < outer; i0 += U * kGT) {
                    const double* at[U];
                    double zv[U];
                    unsigned long long t[U];
                    int to[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int o = i0 + u * kGT, i = o < pown ? o : o + nd, j = i / B;
                        t[u] = tag;
                        at[u] = nullptr;
                        to[u] = i;
                        if (o < outer) {
                            at[u] = A.z + 2 * ((long long)B * shalo[j] + (i - B * j));
                            tag_load(at[u], zv[u], t[u]);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        for (int k = 0; t[u] != tag; ++k) {
                            if (k > limit || others_failed(k, A.failed, A.launch)) {
                                sh.failed = 1;
                                break;
                            }
                            tag_load(at[u], zv[u], t[u]);
                        }
                        if (at[u]) sp[to[u]] = first ? (X)zv[u] + bx * sp[to[u]] : (X)zv[u];
                    }
                }
            }
            __syncthreads();
            // 2: w = K z and z.w
            v[0] = 0.0;
            auto diagonal = [&](int t) {
                const int a = row0 + (t - tb) * (32 / kLpr) + ri;
                return A.dc && a < row1 && sl < B ? (X)__ldg(A.dc + (long long)B * a + sl) : (X)0;
            };
            auto finish = [&](int t, X dci, X(&y)[B]) {
#pragma unroll
                for (int s = kLpr / 2; s > 0; s >>= 1)
#pragma unroll
                    for (int k = 0; k < B; ++k) y[k] += __shfl_xor_sync(0xffffffffu, y[k], s);
                const int a = row0 + (t - tb) * (32 / kLpr) + ri;
                if (a < row1 && sl < B) {
                    const long long i = (long long)B * a + sl;
                    X yi = y[0];
#pragma unroll
                    for (int k = 1; k < B; ++k) yi = sl == k ? y[k] : yi;
                    const X pi = sp[pown + (int)(i - d0)];
                    if (A.dc) yi += dci * pi;
                    vw[i - d0] = yi;
                    v[0] += (double)pi * (double)yi;
                }
            };
            for (int t = tb + warp; t < tr; t += kGW) {
                const int o = soff[t - tb], w = soff[t - tb + 1] - o;
                const X dci = diagonal(t);
                X y[B];
#pragma unroll
                for (int k = 0; k < B; ++k) y[k] = (X)0;
#pragma unroll 4
                for (int s = o; s < o + w; ++s)
                    step_product<V, X>(sval + (size_t)s * (B * B * 32) + lane,
                                          scol[s * 32 + lane], sp, y);
                finish(t, dci, y);
            }
            for (int t = ts0, s = 0; t < ts1; ++t) {  // s: position in the warp's stream
                const int w = soff[t - tb + 1] - soff[t - tb];
                const X dci = diagonal(t);
                X y[B];
#pragma unroll
                for (int k = 0; k < B; ++k) y[k] = (X)0;
                for (int e = s + w; s < e; ++s) {
                    const int in = s % S::CS;
                    if (in == 0 && !ring.wait()) sh.failed = 1;
                    const unsigned char* from = ring.buf + (ring.used % kStages) * S::RB;
                    step_product<V, X>(
                        reinterpret_cast<const V*>(from + in * S::VB) + lane,
                        reinterpret_cast<const unsigned short*>(from + S::CS * S::VB)[in * 32 + lane],
                        sp, y);
                    if (in == S::CS - 1 || s + 1 == ring.steps) {
                        __syncwarp();
                        ++ring.used;
                        if (lane == 0) ring.issue();
                    }
                }
                finish(t, dci, y);
            }
            ok = group_sum(sh, slots, g, tag, limit, v);
            limit = kPollLimit;
            if (!ok) break;
            if (first) {
                pq = v[0];
            } else {
                rr = v[1];
                if (!isfinite(rr)) {
                    status = NB2_E_NAN;
                    break;
                }
                if (rr < thr) break;
                if (rr > rrcap) {
                    status = NB2_E_CG_BREAKDOWN;
                    break;
                }
                beta = v[2] / absnew;
                absnew = v[2];
                if (++iters >= maxit) {
                    status = NB2_E_CG_MAXIT;
                    break;
                }
                if (iters - begun >= kTurnIterations) {
                    paused = true;
                    break;
                }
                pq = v[0] + beta * (2.0 * v[3] + beta * pq);
                bx = (X)beta;
            }
            // Eigen's CG carries on through p.Ap <= 0 (an indefinite tangent); only a
            // non-finite step size is a failure
            const double alpha = absnew / pq;
            if (!isfinite(alpha)) {
                status = NB2_E_NAN;
                break;
            }
            // 3: p, s = K p, x, r, z and the shares of r.r, r.z and z.s; z carries the tag of the
            // sum that follows it
            const X ax = (X)alpha;
            v[1] = v[2] = v[3] = 0.0;
            for (int i = tid; i < nd; i += kGT) {
                X pi = sp[pown + i], si = vw[i];
                if (!first) {
                    pi += bx * vp[i];
                    si += bx * vs[i];
                }
                vp[i] = pi;
                vs[i] = si;
                vx[i] += ax * pi;
                const X rn = vr[i] - ax * si, zi = vi[i] * rn;
                vr[i] = rn;
                sp[pown + i] = zi;
                if (!alone) tag_store(A.z + 2 * (d0 + i), (double)zi, tag + 1);
                v[1] += (double)rn * (double)rn;
                v[2] += (double)rn * (double)zi;
                v[3] += (double)zi * (double)si;
            }
            first = false;
        }
        // the copies still in flight (the rings run ahead)
        if (streams) {
            for (int k = 0; k < kStages; ++k) {
                ring.wait();
                ++ring.used;
            }
            chunks_used = ring.used;
        }
        if (!ok) {
            if (tid == 0) *(volatile unsigned*)A.failed = A.launch;
            break;
        }
        // leave the state where the other kernels expect it
        for (int i = tid; i < nd; i += kGT) {
            if (lay.vectors > 1) A.r[d0 + i] = vr[i];
            if (lay.vectors > 3) A.p[d0 + i] = first ? sp[pown + i] : vp[i];
            if (lay.vectors > 4) A.x[d0 + i] = vx[i];
        }
        if (g.rank == 0 && tid == 0) {
            A.S.absnew[job] = absnew;
            A.S.beta[job] = beta;
            A.S.rr[job] = rr;
            A.S.iters[job] = iters;
            A.S.status[job] = status;
            A.S.done[job] = !paused;
        }
        __syncthreads();  // shared memory is reused by the next turn
    }
}

template <typename V>
__global__ void k_sell_fill(int ntiles, const int* __restrict__ tile_row,
                            const int* __restrict__ tile_end, const int* __restrict__ tile_off,
                            const int* __restrict__ rp, const V* __restrict__ K,
                            const unsigned char* __restrict__ mask, V* __restrict__ val) {
    const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (t >= ntiles) return;
    const int lane = threadIdx.x & 31, a = tile_row[t] + lane / kLpr, sl = lane % kLpr;
    const bool ok = a < tile_end[t];
    const int b0 = ok ? rp[a] : 0, deg = ok ? rp[a + 1] - b0 : 0;
    const int o = tile_off[t], w = tile_off[t + 1] - o, bb = B * B;
    for (int i = 0; i < B; ++i) {
        const bool on = ok && !(mask && mask[(long long)B * a + i]);
        for (int s = 0; s < w; ++s) {
            const int k = kLpr * s + sl;
            const V* src = K + (long long)bb * (b0 + k) + i * B;
            V* dst = val + ((long long)(o + s) * bb + i * B) * 32 + lane;
            for (int e = 0; e < B; ++e) dst[e * 32] = on && k < deg ? src[e] : (V)0;
        }
    }
}

// The halo of each part, with a bitmap over the range of columns it reads in shared memory: the
// first call (halo null) counts, the second writes the sorted rows and the local columns.  Parts
// whose range does not fit report -1.
__global__ void k_sell_halo(const int* __restrict__ part_tile, const int* __restrict__ tile_row,
                            const int* __restrict__ tile_end, const int* __restrict__ tile_off,
                            const int* __restrict__ rp, const int* __restrict__ ci, int words,
                            int* __restrict__ count, const int* __restrict__ halo_ptr,
                            int* __restrict__ halo, int* __restrict__ own0,
                            unsigned short* __restrict__ col) {
    extern __shared__ unsigned bits[];  // [words] bitmap, [words + 1] ranks
    __shared__ int lo, hi;
    __shared__ int scan[32];
    const int part = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
    const int tb = part_tile[part], te = part_tile[part + 1];
    const int r0 = tile_row[tb], r1 = tile_end[te - 1];
    const int e0 = rp[r0], e1 = rp[r1];
    int mn = r0, mx = r1 - 1;
    for (int k = e0 + tid; k < e1; k += nt) {
        mn = min(mn, ci[k]);
        mx = max(mx, ci[k]);
    }
    if (tid == 0) {
        lo = r0;
        hi = r1 - 1;
    }
    __syncthreads();
    atomicMin(&lo, mn);
    atomicMax(&hi, mx);
    __syncthreads();
    const int base = lo & ~31, nw = (hi >> 5) - (base >> 5) + 1;
    if (nw > words) {
        if (tid == 0 && count) count[part] = -1;
        return;
    }
    int* rank = reinterpret_cast<int*>(bits) + words;
    for (int i = tid; i < nw; i += nt) bits[i] = 0u;
    __syncthreads();
    for (int k = e0 + tid; k < e1; k += nt)
        atomicOr(&bits[(ci[k] - base) >> 5], 1u << ((ci[k] - base) & 31));
    for (int a = r0 + tid; a < r1; a += nt) atomicOr(&bits[(a - base) >> 5], 1u << ((a - base) & 31));
    __syncthreads();
    // exclusive ranks of the words: each thread a run of them, then the runs
    const int per = (nw + nt - 1) / nt, w0 = min(tid * per, nw), w1 = min(w0 + per, nw);
    int mine = 0;
    for (int i = w0; i < w1; ++i) mine += __popc(bits[i]);
    int incl = mine;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if ((tid & 31) >= o) incl += v;
    }
    if ((tid & 31) == 31) scan[tid >> 5] = incl;
    __syncthreads();
    int before = incl - mine, total = 0;
    for (int i = 0; i < nt / 32; ++i) {
        if (i < (tid >> 5)) before += scan[i];
        total += scan[i];
    }
    for (int i = w0; i < w1; ++i) {
        rank[i] = before;
        before += __popc(bits[i]);
    }
    __syncthreads();
    if (!halo) {
        if (tid == 0) count[part] = total;
        return;
    }
    auto place = [&](int c) {
        const int w = (c - base) >> 5, b = (c - base) & 31;
        return rank[w] + __popc(bits[w] & ((1u << b) - 1u));
    };
    const int h0 = halo_ptr[part];
    for (int i = tid; i < nw; i += nt) {
        unsigned v = bits[i];
        int at = h0 + rank[i];
        while (v) {
            halo[at++] = base + 32 * i + __ffs(v) - 1;
            v &= v - 1;
        }
    }
    if (tid == 0) own0[part] = place(r0);
    const int lane = tid & 31, sl = lane % kLpr;
    for (int t = tb + (tid >> 5); t < te; t += nt >> 5) {
        const int a = tile_row[t] + lane / kLpr;
        const bool ok = a < tile_end[t];
        const int b0 = ok ? rp[a] : 0, deg = ok ? rp[a + 1] - b0 : 0;
        // padding points at the tile's first row, a valid place to read
        const unsigned short pad = (unsigned short)place(tile_row[t]);
        for (int s = tile_off[t], k = sl; s < tile_off[t + 1]; ++s, k += kLpr)
            col[(long long)s * 32 + lane] = k < deg ? (unsigned short)place(ci[b0 + k]) : pad;
    }
}

int device_sms(nb2_ctx* c) {
    if (c->sms == 0) {
        int sms = 0, coop = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device) !=
                cudaSuccess ||
            cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device) !=
                cudaSuccess ||
            cudaDeviceGetAttribute(&c->smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin,
                                   c->device) != cudaSuccess ||
            !coop) {
            cudaGetLastError();
            sms = -1;
        }
        c->sms = sms;
    }
    return c->sms;
}

// The largest m1 x m2 <= n with both at most kSide (one level up to kSide).
int group_shape(int n, int* m1) {
    if (n <= kSide) {
        *m1 = n;
        return n;
    }
    int best = 0;
    for (int a = 2; a <= kSide; ++a) {
        const int b = std::min(n / a, kSide);
        if (a * b > best) {
            best = a * b;
            *m1 = a;
        }
    }
    return best;
}

// Cycles of an iteration of a system of t tiles on n CTAs: the sums and the exchange, and the
// tiles, read from L2 at about 45 bytes per cycle and SM.
double iteration_cost(int t, int n, double tile_bytes) {
    return (n == 1 ? 600.0 : (n <= kSide ? 4200.0 : 6500.0)) + tile_bytes / 45.0 * t / n;
}

// The number of CTAs of each system.  A system of up to `alone` tiles is one CTA's work; any other gets
// all SMs when it is the only one.  In a batch the systems run side by side, each with the CTAs that let
// all end together (iterations grow like the cells along a side, the cube root of the tiles), as long as
// their K stays in L2; a larger batch takes several such sets in turn.
std::vector<int> group_sizes(const std::vector<int>& tiles, int alone, int ncta,
                             double tile_bytes) {
    constexpr double kL2 = 90e6;
    const size_t n = tiles.size();
    double total = 0.0;
    for (int t : tiles) total += t;
    const int sets = (int)std::max({1.0, std::ceil(total * tile_bytes / kL2),
                                    std::ceil(1.5 * n / ncta)});
    std::vector<double> side(n);
    for (size_t j = 0; j < n; ++j) side[j] = std::cbrt((double)std::max(tiles[j], 1));
    auto sizes = [&](double T) {
        std::vector<int> s(n, 1);
        for (size_t j = 0; j < n; ++j) {
            const int t = tiles[j];
            if (t <= alone) continue;
            int m = 2, m1;
            while (m < std::min(t, ncta) && side[j] * iteration_cost(t, m, tile_bytes) > T) ++m;
            s[j] = group_shape(m, &m1);
        }
        return s;
    };
    double lo = 0.0, hi = 1e12;
    for (int k = 0; k < 60; ++k) {
        const double mid = 0.5 * (lo + hi);
        long long sum = 0;
        for (int v : sizes(mid)) sum += v;
        (sum > (long long)sets * ncta ? lo : hi) = mid;
    }
    return sizes(hi);
}

// Tiles of the pattern (row pointers on the host) and the parts of each system.  False when
// padding would more than double the matrix.
bool sell_tiles(const int* rp, const std::vector<int>& offsets, int ncta, int value_bytes,
                SellPlan* P, std::vector<int>& row, std::vector<int>& end, std::vector<int>& off,
                std::vector<int>& part) {
    constexpr int rows = 32 / kLpr;
    long long steps = 0;
    std::vector<int> tiles;
    for (size_t j = 0; j + 1 < offsets.size(); ++j) {
        P->job_tile.push_back((int)row.size());
        for (int a = offsets[j]; a < offsets[j + 1]; a += rows) {
            const int e = std::min(a + rows, offsets[j + 1]);
            int deg = 0;
            for (int i = a; i < e; ++i) deg = std::max(deg, rp[i + 1] - rp[i]);
            row.push_back(a);
            end.push_back(e);
            off.push_back((int)steps);
            steps += (deg + kLpr - 1) / kLpr;
        }
        tiles.push_back((int)row.size() - P->job_tile.back());
    }
    const int total = (int)row.size();
    P->job_tile.push_back(total);
    off.push_back((int)steps);
    P->ntiles = total;
    P->steps = steps;
    const double tile_bytes = (32.0 * B * B * value_bytes + 64.0) * (double)steps / total;
    const std::vector<int> sizes = group_sizes(tiles, 96 / rows, ncta, tile_bytes);
    for (size_t j = 0; j < tiles.size(); ++j) {
        int m1;
        const int size = group_shape(sizes[j], &m1);
        P->job_m1.push_back(m1);
        P->job_part.push_back((int)part.size());
        for (int r = 0; r < size; ++r)
            part.push_back(P->job_tile[j] + (int)((long long)tiles[j] * r / size));
    }
    P->nparts = (int)part.size();
    P->job_part.push_back(P->nparts);
    part.push_back(total);
    const long long nnz = rp[offsets.back()];
    return steps < (1ll << 26) && 32 * steps <= 2 * nnz + 4096;
}

template <typename T>
bool dev_copy(nb2_ctx* c, T** d, const std::vector<T>& h) {
    return cudaMalloc((void**)d, sizeof(T) * std::max<size_t>(h.size(), 1)) == cudaSuccess &&
           cudaMemcpyAsync(*d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice,
                           c->stream) == cudaSuccess;
}

bool sell_halo(nb2_ctx* c, SellPlan* P, const std::vector<int>& part, const int* rp,
               const int* ci) {
    const int dynamic = c->smem_optin - 1024, words = dynamic / 8 - 1;
    int* count = nullptr;
    std::vector<int> h(P->nparts), ptr(1, 0);
    bool ok = cudaFuncSetAttribute(k_sell_halo, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   dynamic) == cudaSuccess &&
              cudaMalloc(&count, sizeof(int) * P->nparts) == cudaSuccess;
    auto launch = [&]() {
        k_sell_halo<<<P->nparts, 512, dynamic, c->stream>>>(
            P->part_tile, P->tile_row, P->tile_end, P->tile_off, rp, ci, words, count, P->halo_ptr,
            P->halo, P->own0, P->col);
        c->launches++;
        return cudaGetLastError() == cudaSuccess;
    };
    ok = ok && launch() &&
         cudaMemcpyAsync(h.data(), count, sizeof(int) * P->nparts, cudaMemcpyDeviceToHost,
                         c->stream) == cudaSuccess &&
         cudaStreamSynchronize(c->stream) == cudaSuccess;
    if (count) cudaFree(count);
    if (!ok) return false;
    for (int j = 0; j < P->nparts; ++j) {
        const int n = h[j];
        // (FP64 needs the most shared memory; 4 KB stand for the kernel's static arrays)
        if (n < 0 || n > 65535 ||
            !part_layout<double, double>(n, part[j + 1] - part[j], 0, 0, c->smem_optin - 4096).fits)
            return false;
        ptr.push_back(ptr.back() + n);
    }
    return dev_copy(c, &P->halo_ptr, ptr) &&
           cudaMalloc(&P->halo, sizeof(int) * std::max(ptr.back(), 1)) == cudaSuccess &&
           cudaMalloc(&P->own0, sizeof(int) * P->nparts) == cudaSuccess &&
           cudaMalloc(&P->col, sizeof(unsigned short) * 32 * std::max<long long>(P->steps, 1)) ==
               cudaSuccess &&
           launch() && cudaStreamSynchronize(c->stream) == cudaSuccess;
}

SellPlan* sell_build(nb2_ctx* c, const int* h_rp, const std::vector<int>& offsets,
                     int value_bytes, const int* rp, const int* ci) {
    const int sms = device_sms(c);
    if (sms <= 0) return nullptr;
    // z of a part's own rows alone must fit in shared memory
    if (offsets.size() == 2 && offsets[1] / sms > c->smem_optin / (8 * B + 4)) return nullptr;
    auto* P = new SellPlan();
    P->offsets = offsets;
    std::vector<int> row, end, off, part;
    const size_t unknowns = (size_t)offsets.back() * B;
    const bool ok = sell_tiles(h_rp, offsets, sms, value_bytes, P, row, end, off, part) &&
                    dev_copy(c, &P->tile_row, row) && dev_copy(c, &P->tile_end, end) &&
                    dev_copy(c, &P->tile_off, off) && dev_copy(c, &P->part_tile, part) &&
                    cudaMalloc(&P->z, 16 * unknowns) == cudaSuccess &&
                    cudaMemsetAsync(P->z, 0, 16 * unknowns, c->stream) == cudaSuccess &&
                    cudaMalloc(&P->s, 8 * unknowns) == cudaSuccess &&
                    cudaMalloc(&P->turn_ptr, sizeof(int) * (sms + 1)) == cudaSuccess &&
                    sell_halo(c, P, part, rp, ci);
    if (!ok) {
        cudaGetLastError();  // an allocation failure is not sticky: go without
        sell_release(P);
        return nullptr;
    }
    return P;
}

// Longest systems first, each on the window of CTAs that is free earliest; every CTA takes its
// turns in that one global order, so no two groups wait for each other.
void make_schedule(SellPlan* P, const std::vector<int>& active, int ncta) {
    std::vector<int> jobs;
    for (size_t j = 0; j + 1 < P->job_tile.size(); ++j)
        if (active.empty() || active[j]) jobs.push_back((int)j);
    auto tiles = [&](int j) { return P->job_tile[j + 1] - P->job_tile[j]; };
    std::stable_sort(jobs.begin(), jobs.end(), [&](int a, int b) { return tiles(a) > tiles(b); });
    std::vector<double> free_at(ncta, 0.0);
    std::vector<std::vector<GroupTurn>> lists(ncta);
    P->nslots = 0;
    for (int j : jobs) {
        const int size = P->job_part[j + 1] - P->job_part[j];
        int best = 0;
        double when = 1e300;
        for (int c0 = 0; c0 + size <= ncta; ++c0) {
            const double w = *std::max_element(free_at.begin() + c0, free_at.begin() + c0 + size);
            if (w < when) {
                when = w;
                best = c0;
            }
        }
        const int m1 = P->job_m1[j];
        const double cost =
            std::cbrt((double)tiles(j)) * iteration_cost(tiles(j), size, 9000.0);
        for (int r = 0; r < size; ++r) {
            lists[best + r].push_back(
                GroupTurn{j, P->job_part[j] + r, r, m1, size / m1, P->nslots});
            free_at[best + r] = when + cost;
        }
        P->nslots += size * kSlots;
    }
    P->h_turns.clear();
    P->h_turn_ptr.assign(1, 0);
    for (auto& l : lists) {
        P->h_turns.insert(P->h_turns.end(), l.begin(), l.end());
        P->h_turn_ptr.push_back((int)P->h_turns.size());
    }
}

template <typename V>
int fill(nb2_ctx* c, SellPlan* P, const int* rp, const V* K, const unsigned char* mask) {
    void*& v = P->val[sizeof(V) == 4];
    if (!v && cudaMalloc(&v, sizeof(V) * 32 * B * B * std::max<long long>(P->steps, 1)) !=
                  cudaSuccess) {
        cudaGetLastError();
        v = nullptr;
        return NB2_E_INPUT;
    }
    k_sell_fill<V><<<(P->ntiles + 7) / 8, 256, 0, c->stream>>>(
        P->ntiles, P->tile_row, P->tile_end, P->tile_off, rp, K, mask, (V*)v);
    c->launches++;
    NB2_CUDA(c, cudaGetLastError());
    return NB2_OK;
}

template <typename T>
int grow(nb2_ctx* c, T** d, int* cap, int need, size_t bytes) {
    if (need <= *cap) return NB2_OK;
    if (*d) cudaFree(*d);
    *d = nullptr;
    *cap = 0;
    NB2_CUDA(c, cudaMalloc((void**)d, bytes * need));
    *cap = need;
    return NB2_OK;
}

template <typename V, typename X>
int run(nb2_ctx* c, SellPlan* P, GroupScalars S, const std::vector<int>& active, X* x, X* r, X* p,
        X* q, const X* inv, const float* dc) {
    const int ncta = device_sms(c);
    auto kernel = k_group_cg<V, X>;
    cudaFuncAttributes fa;
    NB2_CUDA(c, cudaFuncGetAttributes(&fa, kernel));
    const int dynamic = (c->smem_optin - (int)fa.sharedSizeBytes) / 128 * 128;
    NB2_CUDA(c, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dynamic));
    make_schedule(P, active, ncta);
    const int nturns = (int)P->h_turns.size();
    if (nturns == 0) return NB2_OK;
    NB2_TRY(grow(c, &P->turns, &P->turns_cap, nturns, sizeof(GroupTurn)));
    if (P->nslots > P->slots_cap) {
        NB2_TRY(grow(c, &P->slots, &P->slots_cap, P->nslots, 16));
        NB2_CUDA(c, cudaMemsetAsync(P->slots, 0, 16ll * P->nslots, c->stream));
    }
    const size_t bytes = sizeof(GroupTurn) * nturns;
    if (P->sent_turns.size() != P->h_turns.size() || P->sent_turn_ptr != P->h_turn_ptr ||
        std::memcmp(P->sent_turns.data(), P->h_turns.data(), bytes) != 0) {
        P->sent_turns.clear();
        NB2_CUDA(c, cudaMemcpyAsync(P->turns, P->h_turns.data(), bytes,
                                    cudaMemcpyHostToDevice, c->stream));
        NB2_CUDA(c, cudaMemcpyAsync(P->turn_ptr, P->h_turn_ptr.data(), sizeof(int) * (ncta + 1),
                                    cudaMemcpyHostToDevice, c->stream));
        P->sent_turns = P->h_turns;
        P->sent_turn_ptr = P->h_turn_ptr;
    }
    GroupArgs<V, X> A;
    A.tile_row = P->tile_row;
    A.tile_end = P->tile_end;
    A.tile_off = P->tile_off;
    A.part_tile = P->part_tile;
    A.halo_ptr = P->halo_ptr;
    A.halo = P->halo;
    A.own0 = P->own0;
    A.col = P->col;
    A.val = (const V*)P->val[sizeof(V) == 4];
    A.turns = P->turns;
    A.turn_ptr = P->turn_ptr;
    A.x = x;
    A.r = r;
    A.z = P->z;
    A.p = p;
    A.w = q;
    A.s = (X*)P->s;
    A.inv = inv;
    A.dc = dc;
    A.S = S;
    A.slots = P->slots;
    A.failed = &c->cgs->group_failed;
    A.launch = ++c->group_launches;
    // no value of an earlier launch carries a tag of this one
    A.tag0 = ((unsigned long long)A.launch << 32) + 2;
    int turns = 1;  // of one CTA
    for (int i = 0; i < ncta; ++i)
        turns = std::max(turns, P->h_turn_ptr[i + 1] - P->h_turn_ptr[i]);
    A.start_limit = (int)std::min((long long)kStartLimit * turns, 1ll << 30);
    A.smem_bytes = dynamic;
    void* args[] = {&A};
    NB2_CUDA(c, cudaLaunchCooperativeKernel((const void*)kernel, dim3(ncta), dim3(kGT), args,
                                            (size_t)dynamic, c->stream));
    c->launches++;
    return NB2_OK;
}

}  // namespace

void sell_release(SellPlan* P) {
    if (!P) return;
    void* ptrs[] = {P->tile_row, P->tile_end, P->tile_off, P->part_tile, P->halo_ptr,
                    P->halo,     P->own0,     P->col,      P->val[0],    P->val[1],
                    P->z,        P->s,        P->slots,    P->turns,    P->turn_ptr};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    delete P;
}

int sell_plan(nb2_ctx* c, const std::vector<int>& offsets, int value_bytes, SellPlan** out) {
    if (c->sell_offsets != offsets) {
        sell_release(c->sell);
        c->sell = sell_build(c, c->h_brp.data(), offsets, value_bytes, c->brp, c->bcol);
        c->sell_offsets = offsets;
    }
    *out = c->sell;
    return NB2_OK;
}

template <typename V>
int sell_fill(nb2_ctx* c, SellPlan* P, const V* K, const unsigned char* mask) {
    return fill<V>(c, P, c->brp, K, mask);
}
template int sell_fill<double>(nb2_ctx*, SellPlan*, const double*, const unsigned char*);
template int sell_fill<float>(nb2_ctx*, SellPlan*, const float*, const unsigned char*);

template <typename V, typename X>
int group_cg(nb2_ctx* c, SellPlan* P, GroupScalars S, const std::vector<int>& active, X* x, X* r,
             X* p, X* q, const X* inv, const float* dc) {
    return run<V, X>(c, P, S, active, x, r, p, q, inv, dc);
}
bool group_failed(const nb2_ctx* c) { return c->h_cgs->group_failed == c->group_launches; }

template int group_cg<double, double>(nb2_ctx*, SellPlan*, GroupScalars, const std::vector<int>&,
                                      double*, double*, double*, double*, const double*,
                                      const float*);
template int group_cg<float, float>(nb2_ctx*, SellPlan*, GroupScalars, const std::vector<int>&,
                                    float*, float*, float*, float*, const float*, const float*);
template int group_cg<float, double>(nb2_ctx*, SellPlan*, GroupScalars, const std::vector<int>&,
                                     double*, double*, double*, double*, const double*,
                                     const float*);

}  // namespace nb2
