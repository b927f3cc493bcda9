// radiance_pass.cu — sm_103a kernels of the per-block radiance update.
//
// Restates shaders/radiance.comp (main :361-413, trace_ray :316-346, CastRay_fast :183-291) as two
// kernels per round of up to kChunkTasks tasks (a task = one 32-ray subgroup of one probe):
//
//   march_kernel     persistent warps take tasks from a queue in guided chunks (large early,
//                    single tasks at the end; through a shared-memory block per CTA when the
//                    launch has few tasks per warp).  A warp sets up a task's 32 rays in lock step
//                    (hash seeds, direction, origin, 1/direction), the rays its lanes were marching
//                    in a pool in shared memory meanwhile, and takes their first coarse step there
//                    (38% of the demo's rays end on it).  Its lanes march in a flat loop, up to three
//                    coarse steps per iteration; a lane whose ray ends writes its result (fraction,
//                    info; the set-up wrote its origin and direction) and takes a ray from the pool;
//                    when that is empty, the next task is set up, so lanes never wait for each other.
//   finalize_kernel  eight consecutive tasks per CTA of two warps: the rays read back, the hits
//                    packed 32 to a warp for the refine DDA, material, trilinear fetch of the
//                    previous radiance and shading; then one lane per task and channel for the
//                    xor-butterfly sum.  When R/32 divides 8 a probe's subgroups share a CTA and
//                    their means are summed in order (a lean instantiation when every probe of the
//                    launch does); otherwise through global scratch and a per-probe counter.
//                    Lookup and hit counters are summed per CTA.
//
// Several passes of one context (launch_passes): one march launch over all their tasks (the
// traversal does not read the radiance volume), then each pass's finalize in order, each launched
// as a programmatic dependent of the one before (its volume-free work runs in that one's tail).
// The pass start (next = prev, counters cleared) runs inside the launches, not as copies between
// them; a one-pass call right after another pass call starts its march in the previous
// finalize's tail.
//
// Exactness: see radiance_device.cuh.  Memory: both kernels test voxels through the compact
// world (uint8 ids + occupancy bits, L1-resident; staged in shared memory by the march of a launch
// over one world that fits); between the kernels each ray keeps 32 B (RayBuffer): 268 MB for a
// single pass's round of 2^18 tasks, up to 537 MB for several passes, 1.07 GB for a batch's round
// of 2^20.

#include "radiance_device.cuh"
#include "lumrad_devloop.h"
#include "lumrad_launch.h"

#include <type_traits>

namespace lumrad {
namespace {

// ---------------------------------------------------------------- march kernel
// A ray is regular when each reciprocal of its direction is at most 2^100 in magnitude (no zero
// component; only an exact cancellation in the set-up gives one, or one of a tiny magnitude) and
// its probe lies in the world (its origin then does).  Such a ray's march never meets a NaN or an infinity: its positions
// stay below 2^16 in magnitude, its block corners within 32 of them, and its fraction grows by at
// least 0.5 - 2^-8 per step.  Hence, for it:
//   (a) GLSL's min/max (y < x ? y : x) equal the hardware's min/max: they differ only on NaN and
//       on the sign of a zero, and the skip's 0.01 floor maps both zeros alike;
//   (b) every position it looks up lies in (-1, 16*size + 1): a step adds 0.5 to the fraction, and
//       the skip before it ends at the face of an air block it was in, up to the rounding of the
//       axis with the largest direction component (at least 0.57: an error below 0.02) and the
//       0.01 floor; a ray whose position is outside takes no further step.  So the lookup needs no
//       range test (solid_inside);
//   (c) the 2*max_dist+2 step bound is never reached: the fraction passes max_dist first;
//   (d) while the fraction before the skip is below `exit_fraction` no position is outside, so the
//       exact test is made only for the lanes past it.
// A warp whose rays are all regular marches with those forms; any other warp with the exact forms
// of the general case.  Both give the same bits for a regular ray.
__device__ __forceinline__ bool regular_ray(float ivx, float ivy, float ivz) {
    const float lim = 1.2676506002282294e30f;   // 2^100
    return fabsf(ivx) <= lim && fabsf(ivy) <= lim && fabsf(ivz) <= lim;
}

// A fraction below every one at which the position o + d*f of a regular ray is outside the world:
// per axis the distance to the face ahead less 2^-7 (the position's roundings: below 2^-8 at 2^15)
// over |d|, the least of them less 2^-20 of it (the quotient's roundings); at least 0.
__device__ __forceinline__ float exit_fraction(float3 o, float3 d, float rx, float ry, float rz, float wx, float wy, float wz) {
    const float ex = fmul(fsub(fabsf(fsub(d.x > 0.0f ? wx : 0.0f, o.x)), 0.0078125f), fabsf(rx));
    const float ey = fmul(fsub(fabsf(fsub(d.y > 0.0f ? wy : 0.0f, o.y)), 0.0078125f), fabsf(ry));
    const float ez = fmul(fsub(fabsf(fsub(d.z > 0.0f ? wz : 0.0f, o.z)), 0.0078125f), fabsf(rz));
    return fmaxf(fmul(fminf(ex, fminf(ey, ez)), 0.99999905f), 0.0f);
}

// STAGE: one CTA of kStageWarps warps per SM, with the launch's compact world (compact grid and
// occupancy masks, every world of the launch the same) copied into shared memory at the start;
// lookups are then 32-bit-addressed shared loads (fewer address instructions, lower latency than
// the L1-resident form: a pass over every probe of a 64x64x32 world, 256 rays, 1,979 -> 1,764 us once its
// 157 KB fit; 8% off the demo step's march).  Used where the world fits beside the rays' pools (52 KB of the 227 KB per CTA: a 64x64x16 world of 34 block types takes 87 KB, and compact
// worlds up to 174 KB fit); other launches (batches, servers, larger worlds, hit records) read the
// world from global memory through L1.
constexpr int kStageWarps = 32;
// Queue defaults (LaunchArgs guided_div / max_chunk = 0): the CTA queue's divisor and the chunk
// cap; the per-warp queue divides by kWarpQueueDiv
constexpr int kQueueDiv = 2;
constexpr int kQueueCap = 32;
static_assert(LUMRAD_MAX_CHUNK < (1 << 12) && kQueueCap <= LUMRAD_MAX_CHUNK, "a chunk's count fits 12 bits");
constexpr int kWarpQueueDiv = 1;
// launches with fewer tasks than this per warp claim through the CTA queue (march_kernel's CTAQ)
constexpr int kCtaQueueTasksPerWarp = 32;
// A warp's pool: the rays its lanes were marching when the next task was set up (the set-up needs
// their registers; the new task's rays that go on stay in the lanes that built them).  Idle lanes take
// from it, and when it is empty the next task is set up.  A ray: origin + index, direction + fraction,
// 1/direction + exit fraction, steps.  (Against a ring that the new task's rays all went through and a
// second place for the lanes': half the shared memory, 371 -> 339 M warp instructions for a run of 64
// worlds batched, 2,229 -> 2,189 us with its reads; the 64-ray demo frame 178 -> 170 us.)
struct RayPool {
    float4 o[kTaskRays], d[kTaskRays], i[kTaskRays];
    int steps[kTaskRays];
};
constexpr size_t kStagePoolBytes = (size_t)kStageWarps * sizeof(RayPool);

// Tasks are claimed in two levels.  A CTA takes guided blocks from the launch's queue word
// (remaining / (div * CTAs), clamped to [1, cap * warps per CTA]) into a shared-memory block word
// (start << 32 | length << 20 | next); its warps take guided chunks of that block (its remainder /
// warps per CTA, clamped to [1, cap]) with a shared-memory atomic, and the warp that finds it
// empty fetches the next block under a shared lock.  The global word sees one claim per CTA block
// instead of one per warp chunk (same-address atomics serialise), and warps balance at single
// tasks at the end of a launch.
// A CTA's first block is its own by index (first_block), without the queue: in a launch of at most a
// task per warp every task is, spread evenly over the CTAs.  (A 64-ray pass over 8x8x8 / 20x20x8 /
// 50x50x12 blocks: 16.5 / 20.6 / 71.8 us; with every block from the queue, 32 warps to a CTA before the
// next SM gets one, and every warp counted out by a global atomic 20.7 / 27.1 / 73.7.)
struct CtaQueue {
    unsigned long long blk;
    int lock, done, finished;
};

template <int WPC>
__device__ __forceinline__ long long first_block(const LaunchArgs& la, int n_round) {
    const long long ctas = gridDim.x;
    if (n_round <= ctas * WPC) return (n_round + ctas - 1) / ctas;
    const int div = la.guided_div > 0 ? la.guided_div : kQueueDiv;
    const int cap = la.max_chunk > 0 ? la.max_chunk : kQueueCap;
    return max(1LL, min(n_round / (div * ctas), min(4095LL, (long long)cap * WPC)));
}

// One claim from the CTA's block: start << 12 | count of a guided chunk (its remainder / WPC,
// clamped to [1, cap]; / (2 * WPC) measured 0.4% slower on a single pass, a CTA divisor of 3
// instead of 2 3% slower), or -2 when the block looked empty or ran out.
template <int WPC>
__device__ __forceinline__ long long claim_from_block(int cap, CtaQueue* q) {
    const unsigned long long b = *reinterpret_cast<volatile unsigned long long*>(&q->blk);
    const int next = (int)(b & 0xFFFFFull), len = (int)((b >> 20) & 0xFFFull);
    if (next >= len) return -2;
    const int k = max(1, min(cap, (len - next) / WPC));
    const unsigned long long o = atomicAdd(&q->blk, (unsigned long long)k);
    const int n2 = (int)(o & 0xFFFFFull), l2 = (int)((o >> 20) & 0xFFFull);
    return n2 < l2 ? ((long long)(o >> 32) + n2) << 12 | min(k, l2 - n2) : -2;
}

// The slow path (lane 0 of a warp that found the block empty): fetch the next block under the
// CTA's lock, or claim from a block another warp fetched meanwhile.  Returns a chunk as
// claim_from_block does, or -1 when the launch's tasks are exhausted.  Not inlined: the march loop
// keeps its registers (a call per block, not per chunk).
template <int WPC>
__device__ __noinline__ long long refill_block(const LaunchArgs& la, int n_round, CtaQueue* q) {
    const int div = la.guided_div > 0 ? la.guided_div : kQueueDiv;
    const int cap = la.max_chunk > 0 ? la.max_chunk : kQueueCap;
    const long long ctas = gridDim.x, base = first_block<WPC>(la, n_round) * ctas;
    for (int it = 0; it < (1 << 22); it++) {
        const long long c = claim_from_block<WPC>(cap, q);
        if (c != -2) return c;
        if (*reinterpret_cast<volatile int*>(&q->done)) return -1;
        if (atomicCAS(&q->lock, 0, 1) == 0) {
            const unsigned long long b = *reinterpret_cast<volatile unsigned long long*>(&q->blk);
            if ((b & 0xFFFFFull) < ((b >> 20) & 0xFFFull)) {   // another warp filled it since
                atomicExch(&q->lock, 0);
                continue;
            }
            const long long rem = (long long)n_round - base - (long long)*reinterpret_cast<volatile unsigned long long*>(la.queue);
            const long long cta_cap = min(4095LL, (long long)cap * WPC);
            const long long kk = rem / ((long long)div * ctas);
            const long long k = kk < 1 ? 1 : (kk > cta_cap ? cta_cap : kk);
            const unsigned long long start = atomicAdd(la.queue, (unsigned long long)k) + (unsigned long long)base;
            if ((long long)start >= (long long)n_round) {
                *reinterpret_cast<volatile int*>(&q->done) = 1;
                __threadfence_block();
                atomicExch(&q->lock, 0);
                return -1;
            }
            const long long len = min(k, (long long)n_round - (long long)start);
            const long long own = max(1LL, min((long long)cap, len / (long long)WPC));
            atomicExch(&q->blk, (start << 32) | ((unsigned long long)len << 20) | (unsigned long long)own);
            atomicExch(&q->lock, 0);
            return ((long long)start << 12) | own;
        }
        __nanosleep(64);
    }
    atomicOr(la.error, 1);   // the lock holder never finished (it waits for nothing: cannot happen)
    return -1;
}

// What bounds it: instruction issue (83% of the slots on the demo's 8-pass launch, every world
// lookup in shared memory).  Per 32-ray task that launch issues 890 warp instructions, of which the
// set-up with its first step is about 400 and an iteration (3 steps of about 45 and the hand-out)
// 200.  The launch: 436 -> 366 us, 452 -> 373 M warp instructions, with: lookups without range
// tests or conversions for regular rays (solid_inside), x and y in register pairs, the first step
// in the set-up, results and hand-outs once per three steps, and reciprocals and the square root
// without their checks for operands that cannot occur.  The set-up's x and y in register pairs too: the
// 8-pass step 694.2 -> 689.8 us, every probe of 64x64x32 1,756 -> 1,746 us, 64 worlds batched 2,214 -> 2,196
// us.  (A ray's second random vector is the first of the next lane's; taken from there by shuffles, lane
// 31's formed for eight tasks at a time, one hash less per ray: no faster, 1% slower on the batch.)
template <bool RECORD, bool STAGE = false, bool CTAQ = false>
__global__ void __launch_bounds__(STAGE ? kStageWarps * 32 : kWarps * 32, STAGE ? 1 : 4)
march_kernel(const __grid_constant__ LaunchArgs la) {
    if (CTAQ) grid_launch_dependents();   // its finalize (LaunchArgs::after_march)
    if (la.pass_mask) {   // several passes: mark each pass's probes (this call's mask: the previous
                          // call's last finalize clears the other)
        const long long stride = (long long)gridDim.x * blockDim.x;
        for (int i = 0; i < la.n_worlds; i++) {
            const WorldPass& w = la.worlds[i];
            for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < w.n_groups; g += stride) {
                const short4 q = w.req[g * w.size + w.shift];
                if (q.x < 0 || q.y < 0 || q.z < 0 || q.x >= w.X || q.y >= w.Y || q.z >= w.Z) continue;
                atomicOr(la.pass_mask + (q.x + (long long)w.X * (q.y + (long long)w.Y * q.z)), 1u << i);
            }
        }
    }
    RayPool* s_pool;
    const uint8_t* s_cg = nullptr;
    const uint16_t* s_rows = nullptr;
    if constexpr (STAGE) {
        extern __shared__ __align__(16) unsigned char s_dyn[];
        s_pool = reinterpret_cast<RayPool*>(s_dyn);
        unsigned char* wb = s_dyn + kStagePoolBytes;
        const WorldPass& w0 = la.worlds ? la.worlds[0] : la.single;
        const int cg_bytes = (w0.X + 1) * (w0.Y + 1) * (w0.Z + 1) * (w0.cgrid_wide ? 2 : 1);
        const int cg_pad = (cg_bytes + 15) & ~15;
        const int cb_bytes = w0.n_compact * 512;
        const uint8_t* gcg = reinterpret_cast<const uint8_t*>(w0.cgrid);
        for (int i = threadIdx.x; i < cg_bytes / 16; i += blockDim.x)
            reinterpret_cast<uint4*>(wb)[i] = __ldg(reinterpret_cast<const uint4*>(gcg) + i);
        for (int i = (cg_bytes & ~15) + (int)threadIdx.x; i < cg_bytes; i += blockDim.x) wb[i] = __ldg(gcg + i);
        for (int i = threadIdx.x; i < cb_bytes / 16; i += blockDim.x)
            reinterpret_cast<uint4*>(wb + cg_pad)[i] = __ldg(reinterpret_cast<const uint4*>(w0.cbits) + i);
        __syncthreads();
        s_cg = wb;
        s_rows = reinterpret_cast<const uint16_t*>(wb + cg_pad);
    } else {
        __shared__ RayPool a_pool[kWarps];
        s_pool = a_pool;
    }

    if (la.dev_count) grid_dependency_wait();   // a list from the kernels before (the world is in place by now)
    if (la.time_start && blockIdx.x == 0 && threadIdx.x == 0) {   // the pass's kernel-time start
        la.time_start[0] = globaltimer_ns();
        la.time_start[1] = 0;
    }
    int n_round = la.chunk_end - la.chunk_begin;
    if (la.dev_count) {   // a list built on the device: its own length bounds the round
        const long long real = (long long)(__ldcg(la.dev_count) / la.single.size) * (la.single.R >> 5);
        n_round = (int)max(0LL, min((long long)n_round, real - la.chunk_begin));
    }
    if (la.dev_total)     // a table built on the device: its task count bounds the round
        n_round = (int)max(0LL, min((long long)n_round, __ldcg(la.dev_total) - la.chunk_begin));
    constexpr int kWpc = STAGE ? kStageWarps : kWarps;
    __shared__ CtaQueue s_q;
    if (threadIdx.x == 0) {
        long long start = 0, len = 0;
        if (CTAQ) {
            const long long first = first_block<kWpc>(la, n_round);
            start = (long long)blockIdx.x * first;
            len = max(0LL, min(first, n_round - start));
            s_q.done = first * gridDim.x >= n_round;
        }
        s_q.blk = ((unsigned long long)start << 32) | ((unsigned long long)len << 20);
        s_q.lock = 0;
        s_q.finished = 0;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    RayPool& pool = s_pool[wib];
    const unsigned lt_mask = (1u << lane) - 1u;
    // current world (warp-uniform)
    const WorldPass* wp = &la.single;
    MarchView mv{0, 0, 0, 0, nullptr, nullptr};
    float wx = 0.0f, wy = 0.0f, wz = 0.0f, max_dist = 0.0f;
    unsigned kb = 0;
    int max_steps = 0;
    int w_begin = 0, w_end = 0;
    int taken = 0, pooled = 0;   // the pool's rays [taken, pooled) wait for a lane
    bool slow = false;           // a ray of the lanes or the pool is not regular
    int tb = 0, te = 0;          // grabbed task chunk [tb, te)
    bool exhausted = false;
    int pending = -1;            // grabbed task of another world, waiting for the lanes to drain

    // lane ray state
    int my = -1;                 // round-relative index of the lane's ray, -1 if idle
    f32x2 oxy = 0, dxy = 0, ivxy = 0, cxy = 0;   // x and y of origin, direction, 1/direction, corner
    float oz = 0, dz = 0, ivz = 0, cz = 0, frac = 0;
    int steps = 0;
    float fexit = 0.0f;          // exit_fraction over the axes; -1: the ray is not regular

    // Claims: CTAQ, through the CTA's block (claim_from_block, refill_block; launches with few tasks
    // per warp, such as a single pass: the warps balance at single tasks); else straight from the
    // launch's queue word in guided chunks of remaining / (div * warps), clamped to [1, cap]
    // (several passes, batches: large chunks, few claims).  Two instantiations: the CTA queue's code costs the
    // other form's march loop registers (2.5% on an 8-pass launch when only branched around).
    auto next_task = [&]() -> int {
        if (pending >= 0) return pending;
        if (tb >= te) {
            if (exhausted) return -1;
            long long c = 0;
            if (lane == 0) {
                const int cap = la.max_chunk > 0 ? la.max_chunk : kQueueCap;
                if (CTAQ) {
                    c = claim_from_block<kWpc>(cap, &s_q);
                    if (c == -2) c = refill_block<kWpc>(la, n_round, &s_q);
                } else {
                    const unsigned long long cur = *reinterpret_cast<volatile unsigned long long*>(la.queue);
                    const long long kk = ((long long)n_round - (long long)cur) /
                                         ((long long)(la.guided_div > 0 ? la.guided_div : kWarpQueueDiv) * la.total_warps);
                    const long long k = kk < 1 ? 1 : (kk > cap ? cap : kk);
                    const unsigned long long start = atomicAdd(la.queue, (unsigned long long)k);
                    c = (long long)start >= (long long)n_round ? -1 : (long long)(start << 12) | min(k, (long long)n_round - (long long)start);
                }
            }
            c = __shfl_sync(kFull, c, 0);
            if (c < 0) {
                exhausted = true;
                return -1;
            }
            tb = la.chunk_begin + (int)(c >> 12);
            te = tb + (int)(c & 0xFFF);
        }
        return tb;
    };
    auto corner = [&](float dx, float dy) {   // the far corner's offset in a block, less kBlockBias (exact)
        cxy = pack2(dx > 0.0f ? 16.0f - kBlockBias : -kBlockBias, dy > 0.0f ? 16.0f - kBlockBias : -kBlockBias);
        cz = dz > 0.0f ? 16.0f - kBlockBias : -kBlockBias;
    };
    // the pool's next rays to the lanes in `need`
    auto assign = [&](unsigned need) {
        const int slot = taken + __popc(need & lt_mask);
        if (((need >> lane) & 1u) && slot < pooled) {
            const float4 o4 = pool.o[slot], d4 = pool.d[slot], i4 = pool.i[slot];
            my = __float_as_int(o4.w);
            oxy = pack2(o4.x, o4.y); oz = o4.z;
            dxy = pack2(d4.x, d4.y); dz = d4.z;
            ivxy = pack2(i4.x, i4.y); ivz = i4.z;
            fexit = i4.w;
            corner(d4.x, d4.y);
            frac = d4.w;
            steps = pool.steps[slot];
        }
        taken = min(pooled, taken + __popc(need));
    };
    // ray i has ended, its last lookup at p
    auto end_ray = [&](int i, float px, float py, float pz, bool solid, uint32_t info) {
        if (RECORD) {
            int blk;
            const int v = voxel_value(*wp, f2i(px), f2i(py), f2i(pz), blk);
            if (solid) info |= (uint32_t)v << 16;
            la.ray_blk[i] = blk;
        }
        __stcg(la.rays.res + i, make_uint2(__float_as_uint(frac), info));
    };
    // One coarse step (CastRay_fast, radiance.comp:198-244) of the lane's regular ray, straight-line
    // (the empty-block skip, radiance.comp:215-226, is formed for every lane and selected where the
    // block is air); true if the ray may have ended: `solid`, or at p or frac (ray_ended).
    float f1 = 0.0f, px = 0.0f, py = 0.0f, pz = 0.0f;
    bool solid = false;
    auto step = [&](bool wide) -> bool {
        f1 = fadd(frac, 0.5f);
        const f32x2 pxy = add_product2(oxy, mul2(dxy, pack2(f1, f1)));
        unpack2(pxy, px, py);
        pz = fadd(oz, fmul(dz, f1));
        const float qx = fabsf(px), qy = fabsf(py), qz = fabsf(pz);
        const float bx = __fadd_rz(qx, kBlockBias), by = __fadd_rz(qy, kBlockBias), bz = __fadd_rz(qz, kBlockBias);
        const int cid = cell_id<STAGE>(STAGE ? s_cg : mv.cgrid, cell_inside(mv.X + 1, mv.Y + 1, kb, bx, by, bz), wide);
        solid = solid_inside<STAGE>(STAGE ? s_rows : reinterpret_cast<const uint16_t*>(mv.cbits), cid, qx, qy, qz);
        float tx, ty;
        // to the face ahead (b + c is exact)
        unpack2(sub_product2(mul2(add2(pack2(bx, by), cxy), ivxy), mul2(pxy, ivxy)), tx, ty);
        const float tz = fsub(fmul(fadd(bz, cz), ivz), fmul(pz, ivz));
        const float sk = fmaxf(fminf(tx, fminf(ty, tz)), 0.01f);
        frac = cid == 0 ? fadd(f1, sk) : f1;
        steps++;
        return solid || f1 >= fexit || frac >= max_dist;
    };
    auto ray_ended = [&]() -> bool {
        return solid || frac >= max_dist || px < 0.0f || py < 0.0f || pz < 0.0f || px >= wx || py >= wy || pz >= wz;
    };
    // (a hit in a block of id 0 has the skip in its fraction, and the refine starts past it: general)
    auto hit_info = [&]() -> uint32_t { return (uint32_t)steps | (frac == f1 ? kInfoRegular : 0u) | (solid ? kInfoHit : 0u); };
    auto more_tasks = [&]() { return pending < 0 && !(exhausted && tb >= te); };

    // The coarse march of the lanes' rays, up to three steps per iteration (two: 1-2% slower, four:
    // equal): a lane whose ray ends takes no further one, and the ended rays' results are written
    // and their lanes given new rays once per iteration.  Runs until the pool is empty while tasks
    // may remain, or no lane has a ray.  FAST: every lane's ray and the pool's are regular.
    auto march = [&](auto fast_tag, auto wide_tag) {
        constexpr bool FAST = decltype(fast_tag)::value;
        constexpr bool WIDE = decltype(wide_tag)::value;
        while (true) {
            bool fin = false;
            if constexpr (FAST) {
                if (my >= 0) {
                    fin = step(WIDE);
                    if (!fin) fin = step(WIDE);
                    if (!fin) fin = step(WIDE);
                }
                if (fin) {
                    fin = ray_ended();
                    if (fin) {
                        end_ray(my, px, py, pz, solid, hit_info());
                        my = -1;
                    }
                }
            } else {
                // the general form: GLSL's min and max, the step bound, range-tested lookups
                const uint8_t* cgp = STAGE ? s_cg : mv.cgrid;
                const uint16_t* rowp = STAGE ? s_rows : reinterpret_cast<const uint16_t*>(mv.cbits);
                float ox, oy, dx, dy, ivx, ivy, cx, cy;
                unpack2(oxy, ox, oy);
                unpack2(dxy, dx, dy);
                unpack2(ivxy, ivx, ivy);
                unpack2(cxy, cx, cy);
                for (int u = 0; u < 2 && my >= 0; u++) {
                    const float f = fadd(frac, 0.5f);
                    const float x = fadd(ox, fmul(dx, f)), y = fadd(oy, fmul(dy, f)), z = fadd(oz, fmul(dz, f));
                    int cid;
                    const bool hit = solid_at_p<WIDE, STAGE>(cgp, rowp, mv.X, mv.Y, mv.Z, f2i(x), f2i(y), f2i(z), cid);
                    // the block's low corner (ix/16)*16 with ix = trunc(x) is trunc(x/16)*16, exact
                    // in FP32 (a NaN x gives a NaN skip either way)
                    const float bx = fadd_exact_mul(fadd(cx, kBlockBias), truncf(fmul(x, 0.0625f)), 16.0f);
                    const float by = fadd_exact_mul(fadd(cy, kBlockBias), truncf(fmul(y, 0.0625f)), 16.0f);
                    const float bz = fadd_exact_mul(fadd(cz, kBlockBias), truncf(fmul(z, 0.0625f)), 16.0f);
                    const float tx = fadd(fmul(bx, ivx), fmul(-x, ivx));
                    const float ty = fadd(fmul(by, ivy), fmul(-y, ivy));
                    const float tz = fadd(fmul(bz, ivz), fmul(-z, ivz));
                    const float sk = gmax(gmin(tx, gmin(ty, tz)), 0.01f);
                    frac = cid == 0 ? fadd(f, sk) : f;
                    steps++;
                    const bool out = x < 0.0f || y < 0.0f || z < 0.0f || x >= wx || y >= wy || z >= wz || frac >= max_dist;
                    if (hit || out || steps >= max_steps) {
                        end_ray(my, x, y, z, hit,
                                (uint32_t)steps | (fexit >= 0.0f && frac == f ? kInfoRegular : 0u) |
                                    (hit ? kInfoHit : (out ? 0u : kInfoCapped)));
                        my = -1;
                        fin = true;
                    }
                }
            }
            const unsigned fm = __ballot_sync(kFull, fin);
            if (fm) {
                assign(fm);
                if (taken == pooled && (more_tasks() || !__any_sync(kFull, my >= 0))) break;
            }
        }
    };

    while (true) {
        // 1. the pool empty: set up tasks until one leaves rays
        const bool refill = taken == pooled && (pending >= 0 || more_tasks());
        bool left = !refill;
        if (refill) {   // the lanes' rays into the pool: the set-up needs the registers
            const unsigned pm = __ballot_sync(kFull, my >= 0);
            slow = __any_sync(kFull, my >= 0 && fexit < 0.0f);
            taken = 0;
            pooled = __popc(pm);
            if (my >= 0) {
                const int slot = __popc(pm & lt_mask);
                float x, y;
                unpack2(oxy, x, y);
                pool.o[slot] = make_float4(x, y, oz, __int_as_float(my));
                unpack2(dxy, x, y);
                pool.d[slot] = make_float4(x, y, dz, frac);
                unpack2(ivxy, x, y);
                pool.i[slot] = make_float4(x, y, ivz, fexit);
                pool.steps[slot] = steps;
                my = -1;
            }
        }
        while (!left) {
            const int t = next_task();
            if (t < 0) break;
            if (t < w_begin || t >= w_end) {
                const WorldPass* wq = la.worlds ? la.worlds + world_of(la, t) : &la.single;
                if (t >= (int)(wq->task_begin + wq->n_tasks)) {   // alignment gap between worlds
                    if (pending == t) pending = -1; else tb++;
                    continue;
                }
                // another world: drain this one first, unless it is another pass over the same
                // compact world with the same bound (passes of one context), whose rays march alike
                const bool alike = reinterpret_cast<const uint8_t*>(wq->cgrid) == mv.cgrid &&
                                   wq->max_dist == max_dist;
                if (!alike && pooled > 0) {
                    if (pending != t) tb++;
                    pending = t;
                    break;
                }
                wp = wq;
                mv = march_view(*wp);
                kb = cell_bias(mv.X + 1, mv.Y + 1);
                wx = fmul((float)mv.X, 16.0f); wy = fmul((float)mv.Y, 16.0f); wz = fmul((float)mv.Z, 16.0f);
                max_dist = wp->max_dist;
                max_steps = wp->max_steps;
                w_begin = (int)wp->task_begin;
                w_end = (int)(wp->task_begin + wp->n_tasks);
            }
            if (pending == t) pending = -1; else tb++;
            // lane i builds ray i of the task (subgroup k of workgroup g)
            const int t_local = t - w_begin;
            const int nsub = wp->R >> 5;
            const int g = div_nsub(t_local, nsub);
            const uint32_t inv = (uint32_t)t_local * kTaskRays + (uint32_t)lane;
            const float3 r1 = ray_random(*wp, inv), r2 = ray_random(*wp, inv + 1);
            const bool inside = setup_ray(*wp, g, (t_local - g * nsub) * kTaskRays + lane, r1, r2, oxy, oz, dxy, dz);
            float3 o, d;
            unpack2(oxy, o.x, o.y);
            unpack2(dxy, d.x, d.y);
            o.z = oz;
            d.z = dz;
            const int idx = (t - la.chunk_begin) * kTaskRays + lane;
            __stcg(la.rays.od + idx, make_float4(o.x, o.y, o.z, d.x));
            __stcg(la.rays.dd + idx, make_float2(d.y, d.z));
            float rx = rcp_normal(d.x), ry = rcp_normal(d.y), rz = rcp_normal(d.z);
            const bool regular = inside && regular_ray(rx, ry, rz);
            if (!regular) {
                rx = __frcp_rn(d.x);
                ry = __frcp_rn(d.y);
                rz = __frcp_rn(d.z);
            }
            // the rays' first step here, where all 32 lanes take it
            ivxy = pack2(rx, ry); ivz = rz;
            fexit = regular ? exit_fraction(o, d, rx, ry, rz, wx, wy, wz) : -1.0f;
            corner(d.x, d.y);
            frac = 0.0f;
            steps = 0;
            my = idx;
            const bool fast = __all_sync(kFull, regular);
            if (!fast) slow = true;
            else if (step(mv.wide) && ray_ended()) {
                end_ray(idx, px, py, pz, solid, hit_info());
                my = -1;
            }
            left = __any_sync(kFull, my >= 0);
        }
        __syncwarp();
        // 2. idle lanes take rays
        assign(__ballot_sync(kFull, my < 0));
        if (!__any_sync(kFull, my >= 0)) {
            // nothing in flight and nothing set up: no task was left (a task of another world
            // would have been set up above, the lanes being drained)
            if ((pending >= 0 || taken < pooled) && lane == 0) atomicOr(la.error, 1);
            break;
        }
        // 3. march
        if (mv.wide) {
            if (!slow) march(std::true_type{}, std::true_type{});
            else march(std::false_type{}, std::true_type{});
        } else {
            if (!slow) march(std::true_type{}, std::false_type{});
            else march(std::false_type{}, std::false_type{});
        }
    }


    // The pass's start (see LaunchArgs), after the marching: a launch dependent on the previous
    // pass's finalize marches in that launch's tail and waits here for it to end before touching
    // what that launch reads or writes (the volumes, the counters)
    if (la.copy_dst || la.clear_stats || la.count_dst) {
        grid_dependency_wait();
        const long long stride = (long long)gridDim.x * blockDim.x;
        const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
        if (la.copy_dst) {   // next starts as a copy of prev
            const long long n16 = la.copy_bytes >> 4;
            const uint4* s16 = reinterpret_cast<const uint4*>(la.copy_src);
            uint4* d16 = reinterpret_cast<uint4*>(la.copy_dst);
            for (long long i = tid; i < n16; i += stride) d16[i] = __ldcs(s16 + i);
            const long long n4 = la.copy_bytes >> 2;
            for (long long i = n16 * 4 + tid; i < n4; i += stride)
                reinterpret_cast<unsigned*>(la.copy_dst)[i] = reinterpret_cast<const unsigned*>(la.copy_src)[i];
        }
        if (tid < 2 && la.clear_stats) la.clear_stats[tid] = 0;
        if (tid == 0 && la.count_dst) *la.count_dst = __ldcg(la.count_src);
    }

    // the last CTA to finish resets the queue for the next launch (its last warp reports it: one
    // same-address global atomic per CTA)
    if (lane == 0 && atomicAdd(&s_q.finished, 1) == kWpc - 1) {
        const unsigned long long e = atomicAdd(la.queue + 1, 1ull);
        if (e == (unsigned long long)gridDim.x - 1) {
            la.queue[0] = 0;
            la.queue[1] = 0;
        }
    }
}

// ---------------------------------------------------------------- finalize kernel
// What a finalize CTA shares: its hits' ray numbers, every ray's light by channel and task
// (kFinStride: 32 and one, so that lanes reading different tasks hit different banks), counters.
constexpr int kFinStride = kTaskRays + 1;
struct FinShared {
    float light[3 * kFinWarps * kFinStride];
    uint8_t hit[kFinWarps * kTaskRays];
    int n_hits;
    unsigned lookups;
    int irregular;               // whether a hit's ray is not regular
    __device__ __forceinline__ void put_light(int task, int lane, float3 v) {
        float* s = light + task * kFinStride + lane;
        s[0] = v.x;
        s[kFinWarps * kFinStride] = v.y;
        s[2 * kFinWarps * kFinStride] = v.z;
    }
};
static_assert(kFinWarps * kTaskRays <= 256 && 3 * kFinWarps <= 32 && (kFinWarps & (kFinWarps - 1)) == 0,
              "ray numbers fit 8 bits, one lane per channel and task");

// A hit ray by the general forms, its light into the CTA's; returns its lookups.  (Out of line, and with
// nothing of the caller's passed by address: the regular rays' path keeps its values in registers.)
template <class Store, bool RECORD>
__device__ __noinline__ uint32_t finalize_general(const WorldPass& w, const RayBuffer& rays, const int* ray_blk, int idx, int ray,
                                                  long long gr, FinShared& sh) {
    const uint2 res = rays.res[idx];
    const float4 od = rays.od[idx];
    const float2 dd = rays.dd[idx];
    float3 u;
    float4 m;
    const uint32_t n = refine_general<RECORD>(w, make_float3(od.x, od.y, od.z), make_float3(od.w, dd.x, dd.y), __uint_as_float(res.x),
                                              res.y, RECORD ? __ldcg(ray_blk + idx) : 0, gr, u, m);
    grid_dependency_wait();
    sh.put_light(ray >> 5, ray & 31, shade_hit<Store>(w, u, m));
    return n;
}

// Warps per CTA, and CTAs per SM of the lean and the general form.  The kernel waits on its chain of
// dependent lookups and its barriers, so small CTAs pay: two warps for a group's eight tasks.  Of the
// SM's 256 KB their shared memory (3.4 + 1 KB a CTA) leaves the L1 less the more of them run, and the
// L1 (47% hits; 8 KB of rays a CTA, the world, the taps) decides: 21 CTAs, at 40 registers.
// On the demo's 8-pass step / a 64-ray demo frame / 64 worlds batched: 673 / 166.5 / 2,188 us (with 24
// CTAs, of which 22 ran, 688 / 170.7 / 2,203; 18: 722 / 175.6 / 2,245; 16: 724 / 180 /
// 2,265; 132 KB of shared memory for all 24: 725 / 174 / 2,247).  Before these lines, at 717 / 186 /
// 2,601: four warps 730 / 191 / 2,700; eight warps, one task each, 725 / 197 / 2,775; one warp 793 / 190 /
// 2,648.
constexpr int kFinCtaWarps = 2;
constexpr int kFinLeanCtas = 21, kFinGeneralCtas = 16;
// A launch of at most this many groups per SM has no second round of CTAs to keep the SMs busy: it
// runs a warp per task (6 CTAs per SM), whose CTAs finish sooner.  One 64-ray pass of 79 / 306 / 832 /
// 1,728 / 2,693 / 4,224 groups on 152 SMs: 20.7 / 25.6 / 31.0 / 44.7 / 55.5 / 73.7 us against 20.8 /
// 32.4 / 36.8 / 46.5 / 55.4 / 73.5 us with two warps; the lines cross near 2,500.
// The general form's warp-per-task CTAs run 4 to an SM: an R = 96 pass of 459 groups 28.6 against 32.8
// us, of 1,570 groups 92.6 against 86.0.  Over a world table: a batch of one / two 8x8x8 worlds 47 / 49 us,
// of 64 lists of 5% of such worlds 54, a served request 160, against 54 / 54.4, 61 and 171 with two warps.
// Passes with hit records take it up to 16 groups per SM in both forms.  Their kernels, 64 rays over every
// probe of 8x8x8 (128 groups) / 2% of 64x64x16 (164): 36.8 / 46.2 us with two warps, 24.2 / 32.0; 96 rays
// over 20x20x8 (1,200) 60.7, 53.9; 64 rays over 20% of 64x64x16 (1,640) 92, 89; past the line two warps
// do as without records (96 rays, 20% of 64x64x16, 4,915 groups, 110 us; a warp per task 165).
constexpr int kFinFewGroups = 16, kFinFewGeneral = 4;
constexpr int kFinFewLeanCtas = 6, kFinFewGeneralCtas = 4;

// One group of eight consecutive tasks (one CTA's work).  A warp per task in lock step had 20 of 32
// lanes active: odd rays of a subgroup point the other way, so most tasks mix hits and misses.  Here
// the CTA's hits are refined and shaded 32 to a warp, and one lane per task and channel sums the
// subgroup in the butterfly's order from shared memory: 38.3 -> 28.1 M warp instructions per pass of
// the demo step when it was made, 25.3 M with the steps since.
// IN_CTA: every probe of the launch combines inside one CTA (R/32 divides kFinWarps); the kernel
// then has no global-memory combine.  SINGLE: the launch covers one world (a single pass, or one
// pass of a several-pass call), read from the kernel's parameters, whose fields are operands from
// the constant bank; else the world table's entry for the group through a generic pointer.
template <class Store, bool RECORD, bool IN_CTA, bool SINGLE, int CW>
__device__ __forceinline__ void finalize_group(const LaunchArgs& la, int group, FinShared& sh) {
    const int lane = threadIdx.x & 31;
    const int w = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        sh.n_hits = 0;
        sh.lookups = 0;
        sh.irregular = 0;
    }
    __syncthreads();
    const int t0 = la.chunk_begin + group * kFinWarps;   // worlds start at multiples of 8
    const WorldPass* wp = SINGLE ? &la.single : la.worlds ? la.worlds + world_of(la, t0) : &la.single;
    const int t0_local = t0 - (int)wp->task_begin;
    long long n_tasks = min(wp->n_tasks, (long long)la.chunk_end - wp->task_begin);
    if (la.dev_count)   // a list built on the device (single world): its own length bounds the tasks
        n_tasks = min(n_tasks, (long long)(__ldcg(la.dev_count) / wp->size) * (wp->R >> 5));
    const int first = (t0 - la.ray_origin) * kTaskRays;   // the group's first ray in the ray buffer
    // 1. the tasks' rays, one warp a task: the hits into the CTA's list, the misses' light.  (Every
    // ray is read here, through L1: a hit's origin and direction then wait there for step 2.  Two
    // tasks' loads at a time: every probe of 64x64x32 / 64 worlds batched / a 64-ray demo frame 1,741 / 2,214 /
    // 167.4 -> 1,735 / 2,198 / 167.0 us; four at a time 0.6% slower than two.)
    unsigned lookups = 0;
    constexpr int kBatch = CW < kFinWarps ? 2 : 1;   // tasks whose rays a warp reads before it uses them
#pragma unroll
    for (int k0 = w; k0 < kFinWarps; k0 += kBatch * CW) {
        uint2 res[kBatch];
        float2 dd[kBatch];
        float4 od[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; u++) {
            const int k = k0 + u * CW, idx = first + k * kTaskRays + lane;
            if (t0_local + k >= n_tasks) break;
            res[u] = la.rays.res[idx];
            dd[u] = la.rays.dd[idx];
            od[u] = la.rays.od[idx];
        }
#pragma unroll
        for (int u = 0; u < kBatch; u++) {
            const int k = k0 + u * CW;
            if (t0_local + k >= n_tasks) break;
            const bool hit = res[u].y & kInfoHit;
            lookups += res[u].y & 0xffffu;
            const unsigned hm = __ballot_sync(kFull, hit);
            int base = 0;
            if (lane == 0 && hm) base = atomicAdd(&sh.n_hits, __popc(hm));
            base = __shfl_sync(kFull, base, 0);
            if (hit) {
                sh.hit[base + __popc(hm & ((1u << lane) - 1u))] = (uint8_t)(k * kTaskRays + lane);
                if (!(res[u].y & kInfoRegular)) sh.irregular = 1;
            } else {
                sh.put_light(k, lane, sky_light(make_float3(od[u].w, dd[u].x, dd[u].y)));
                if (RECORD)
                    record_miss(*wp, __uint_as_float(res[u].x), res[u].y, __ldcg(la.ray_blk + first + k * kTaskRays + lane),
                                (long long)(t0_local + k) * kTaskRays + lane);
            }
        }
    }
    __syncthreads();
    // 2. the hits, packed 32 to a warp (the first 32 to another warp in each group, so that every
    // scheduler of the SM gets its share).  Their rays leave the L1 with this read: keeping them costs the
    // 8-pass step 0.6%, not reading the hits' in step 1 1.4%.  (The general form's 16 CTAs leave the L1
    // larger: there an R = 96 pass takes 71.7 us with them kept, 73.2 without.)
    const int n_hits = sh.n_hits;
#pragma unroll 1
    for (int j = (int)(threadIdx.x + 32 * (group % CW)) % (32 * CW); !RECORD && j < n_hits; j += 32 * CW) {
        const int ray = sh.hit[j], idx = first + ray;
        const uint2 res = la.rays.res[idx];
        if (!(res.y & kInfoRegular)) continue;   // below
        const float4 od = IN_CTA ? load_last(la.rays.od + idx) : la.rays.od[idx];
        const float2 dd = IN_CTA ? load_last(la.rays.dd + idx) : la.rays.dd[idx];
        const float3 o = make_float3(od.x, od.y, od.z), d = make_float3(od.w, dd.x, dd.y);
        const float frac = __uint_as_float(res.x);
        float3 u;
        float4 m;
        const MarchView mv = march_view(*wp);
        lookups += mv.wide ? refine_regular<true>(*wp, mv, o, d, frac, u, m) : refine_regular<false>(*wp, mv, o, d, frac, u, m);
        grid_dependency_wait();   // from here on the volumes: the previous pass's launch has finished
        sh.put_light(ray >> 5, ray & 31, shade_hit<Store>(*wp, u, m));
    }
    // the hits of rays that are not regular (apart, so that the loop above has no call to keep values
    // for), or every hit if they are recorded
    if (RECORD || sh.irregular) {
        for (int j = threadIdx.x; j < n_hits; j += 32 * CW) {
            const int ray = sh.hit[j], idx = first + ray;
            if (RECORD || !(la.rays.res[idx].y & kInfoRegular))
                lookups += finalize_general<Store, RECORD>(*wp, la.rays, la.ray_blk, idx, ray, (long long)t0_local * kTaskRays + ray, sh);
        }
    }
    lookups = __reduce_add_sync(kFull, lookups);
    if (lane == 0 && lookups) atomicAdd(&sh.lookups, lookups);
    __syncthreads();
    // 3. one warp: lane 8*c + k sums channel c of task k, then the tasks of a probe in order
    if (w != group % CW) return;
    const int k8 = lane & (kFinWarps - 1);
    const int t_local = t0_local + k8;
    const bool valid = lane < 3 * kFinWarps && t_local < n_tasks;
    const float mean = valid ? fmul(butterfly_sum(sh.light + lane * kFinStride), 0.03125f) : 0.0f;   // /32
    grid_dependency_wait();
    const int nsub = wp->R >> 5;
    // a probe's subgroups share this CTA when R/32 divides 8 (task_begin is a multiple of 8)
    const bool local = (kFinWarps % nsub) == 0 && (wp->task_begin % kFinWarps) == 0;
    float acc = mean;
    if (local) {   // the subgroups' means summed in subgroup order (radiance.comp:401-407)
        acc = 0.0f;
        const int head = lane & ~(nsub - 1);
        for (int i = 0; i < nsub; i++) acc = fadd(acc, __shfl_sync(kFull, mean, head + i));
        acc = fdiv_by(acc, (float)nsub, wp->inv_nsub);
    }
    const float3 v = make_float3(acc, __shfl_sync(kFull, acc, kFinWarps + k8), __shfl_sync(kFull, acc, 2 * kFinWarps + k8));
    if (lane < kFinWarps && valid) {
        const int g = div_nsub(t_local, nsub);
        const int k = t_local - g * nsub;
        if (local) {
            if (k == 0) store_probe<Store>(*wp, g, v);
        } else if (IN_CTA) {
            atomicOr(la.error, 2);   // launched with the wrong kernel: reported, never stored
        } else {
            subgroup_done<Store>(*wp, g, k, v);
        }
    }
    // the CTA's counters in one atomic each: one world per CTA; same-address atomics from every
    // task serialise at one L2 slice and held warps at exit (measured 5% of the pass)
    if (lane == 0) {
        if (sh.lookups) atomicAdd(wp->stats, (unsigned long long)sh.lookups);
        if (sh.n_hits) atomicAdd(wp->stats + 1, (unsigned long long)sh.n_hits);
        if (la.time_end) atomicMax(la.time_end + 1, globaltimer_ns());
    }
}

// PERSIST (launches sized on the device): a fixed grid walks the 8-task groups of the device's
// task count; otherwise one CTA per group.
template <class Store, bool RECORD, bool IN_CTA, bool PERSIST = false, bool SINGLE = false, int CW = kFinCtaWarps>
__global__ void __launch_bounds__(CW * 32, CW == kFinCtaWarps ? (IN_CTA ? kFinLeanCtas : kFinGeneralCtas)
                                              : (IN_CTA ? kFinFewLeanCtas : kFinFewGeneralCtas))
finalize_kernel(const __grid_constant__ LaunchArgs la) {
    if (la.after_march) grid_dependency_wait();
    grid_launch_dependents();   // the next pass's launch may start its volume-free part
    if (la.pass_mask && (int)blockIdx.x >= la.fin_ctas) {   // copy role (see LaunchArgs)
        grid_dependency_wait();
        using T = typename Store::T;
        const T* src = reinterpret_cast<const T*>(la.copy_src);
        T* dst = reinterpret_cast<T*>(la.copy_dst);
        const long long n = la.copy_bytes / (long long)sizeof(T);
        const long long stride = (long long)(gridDim.x - la.fin_ctas) * blockDim.x;
        for (long long p = (long long)(blockIdx.x - la.fin_ctas) * blockDim.x + threadIdx.x; p < n; p += stride) {
            const uint32_t m = la.pass_mask[p];
            if (!((m >> la.mask_bit) & 1u)) dst[p] = __ldcs(src + p);
            if (la.mask_clear && m) la.pass_mask[p] = 0;
        }
        __syncthreads();
        if (threadIdx.x == 0 && la.time_end) atomicMax(la.time_end + 1, globaltimer_ns());
        return;
    }
    __shared__ FinShared sh;
    if (!PERSIST) {
        finalize_group<Store, RECORD, IN_CTA, SINGLE, CW>(la, (int)blockIdx.x, sh);
        return;
    }
    const long long total = la.dev_total ? __ldcg(la.dev_total) : (long long)la.chunk_end;
    const int groups = (int)((min(total, (long long)la.chunk_end) - la.chunk_begin + kFinWarps - 1) / kFinWarps);
    for (int g = (int)blockIdx.x; g < groups; g += (int)gridDim.x) {
        finalize_group<Store, RECORD, IN_CTA, false, CW>(la, g, sh);
        __syncthreads();   // the group's counters and light are read before the next group's
    }
}

// CTAs of a march launch: the occupancy limit (or ctas_per_sm) on every SM, but no more than the
// largest round has tasks (a small world spreads over the SMs, a warp or two of work in each CTA)
int march_grid(bool record, int num_sms, long long round_tasks, int ctas_per_sm = 0) {
    int per_sm = 0;
    const cudaError_t e = record
        ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, march_kernel<true>, kWarps * 32, 0)
        : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, march_kernel<false>, kWarps * 32, 0);
    if (e != cudaSuccess || per_sm < 1) per_sm = 1;
    if (ctas_per_sm > 0 && ctas_per_sm < per_sm) per_sm = ctas_per_sm;
    return (int)std::min<long long>((long long)num_sms * per_sm, std::max(round_tasks, 1LL));
}

// Whether a launch over these worlds (all with the same compact world) can stage it in shared
// memory, and the dynamic shared bytes it then takes (0 if not).  The kernel's opt-in limit is set
// once per device.
size_t stage_bytes(const WorldPass& w) {
    static int max_optin[64];
    static bool ready[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    if (!ready[dev]) {
        int v = 0;
        cudaFuncAttributes fa{}, fq{};
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
            cudaFuncGetAttributes(&fa, march_kernel<false, true>) != cudaSuccess ||
            cudaFuncGetAttributes(&fq, march_kernel<false, true, true>) != cudaSuccess)
            v = 0;
        // the kernels' static shared words (the CTA queue's block in one form)
        v = std::max(0, v - (int)std::max(fa.sharedSizeBytes, fq.sharedSizeBytes));
        if (v > 0 && (cudaFuncSetAttribute(march_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, v) !=
                          cudaSuccess ||
                      cudaFuncSetAttribute(march_kernel<false, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           v) != cudaSuccess))
            v = 0;
        max_optin[dev] = v;
        ready[dev] = true;
    }
    if (w.n_compact <= 0) return 0;
    const size_t cg = (compact_cells(w.X, w.Y, w.Z) * (w.cgrid_wide ? 2 : 1) + 15) & ~(size_t)15;
    const size_t bytes = kStagePoolBytes + cg + (size_t)w.n_compact * 512;
    return bytes <= (size_t)max_optin[dev] ? bytes : 0;
}

// The march launch of a round (no hit records): staged when the world fits shared memory; the
// CTA queue when the round has few tasks per warp.  dependent: see launch_kernel (the previous kernel
// is the previous pass's finalize, and the march writes the other ray buffer; or the list's, and the
// march waits for it before it reads the list).  Returns whether it took the CTA queue: its finalize
// may then be its programmatic dependent.
bool launch_march(LaunchArgs args, const WorldPass& w, long long round_tasks, int num_sms, cudaStream_t stream,
                  bool dependent = false) {
    const size_t smem = stage_bytes(w);
    if (smem > 0) {
        const int blocks = (int)std::min<long long>(num_sms, std::max(round_tasks, 1LL));
        args.total_warps = blocks * kStageWarps;
        const bool q = round_tasks < (long long)kCtaQueueTasksPerWarp * args.total_warps;
        launch_kernel(q ? march_kernel<false, true, true> : march_kernel<false, true>, blocks, kStageWarps * 32, smem, stream,
                      dependent, args);
        return q;
    }
    const int blocks = march_grid(false, num_sms, round_tasks, args.march_ctas);
    args.total_warps = blocks * kWarps;
    const bool q = round_tasks < (long long)kCtaQueueTasksPerWarp * args.total_warps;
    launch_kernel(q ? march_kernel<false, false, true> : march_kernel<false>, blocks, kWarps * 32, 0, stream, dependent, args);
    return q;
}

// Whether a finalize launch of n tasks is one of few groups (kFinFewGroups): a warp per task, and a
// programmatic dependent of its march (8x8x8 / 20x20x8 / 32x32x12 blocks, 64 rays, a pass 16.5 / 20.6 /
// 42.9 -> 11.4 / 19.0 / 40.1 us; with more groups the waiting CTAs are in the way of the march's end:
// the 64-ray demo frame 181.3 us without, 185.4 with).
bool few_groups(int n, bool in_cta, int num_sms) {
    return (n + kFinWarps - 1) / kFinWarps <= (in_cta ? kFinFewGroups : kFinFewGeneral) * num_sms;
}

// overlap: launched as a programmatic dependent of the stream's previous kernel (a finalize launch
// of the previous pass), whose CTAs let it start early (griddepcontrol.launch_dependents); its
// volume reads and writes wait for that kernel's end (griddepcontrol.wait).  single: every task of
// the launch belongs to args.single.
template <class Store, bool RECORD>
void launch_finalize(const LaunchArgs& args, int n, bool in_cta, cudaStream_t stream, bool overlap, bool single, int num_sms) {
    const int groups = (n + kFinWarps - 1) / kFinWarps;
    const int blocks = groups + (args.pass_mask ? args.fin_copy : 0);
    if (blocks <= 0) return;
    auto pick = [&](auto warps) {   // (hit records are of one world)
        constexpr int CW = decltype(warps)::value;
        if (RECORD || single)
            return in_cta ? finalize_kernel<Store, RECORD, true, false, true, CW> : finalize_kernel<Store, RECORD, false, false, true, CW>;
        return in_cta ? finalize_kernel<Store, false, true, false, false, CW> : finalize_kernel<Store, false, false, false, false, CW>;
    };
    if (few_groups(n, in_cta || RECORD, num_sms)) {
        launch_kernel(pick(std::integral_constant<int, kFinWarps>{}), blocks, kFinWarps * 32, 0, stream, overlap, args);
        return;
    }
    auto k = pick(std::integral_constant<int, kFinCtaWarps>{});
    launch_kernel(k, blocks, kFinCtaWarps * 32, 0, stream, overlap, args);
}

template <class Store, bool RECORD>
cudaError_t launch_t(const LaunchArgs& a, int num_sms, cudaStream_t stream, bool dependent) {
    const long long round = a.round_tasks > 0 ? a.round_tasks : kChunkTasks;
    const int blocks = march_grid(RECORD, num_sms, std::min(a.n_tasks, round), a.march_ctas);
    LaunchArgs args = a;
    args.total_warps = blocks * kWarps;
    for (long long c0 = 0; c0 < a.n_tasks; c0 += round) {
        args.chunk_begin = (int)c0;
        args.chunk_end = (int)min(c0 + round, a.n_tasks);
        args.ray_origin = args.chunk_begin;
        const int n = args.chunk_end - args.chunk_begin;
        bool queue = false;
        if (RECORD) march_kernel<RECORD><<<blocks, kWarps * 32, 0, stream>>>(args);
        else queue = launch_march(args, a.single, std::min(a.n_tasks, round), num_sms, stream, dependent && c0 == 0);
        args.copy_dst = nullptr;   // the pass's start: in the first round's march only
        args.clear_stats = nullptr;
        args.count_dst = nullptr;
        args.time_start = nullptr;
        const bool lean = a.force_lean || (a.worlds ? a.in_cta != 0 : combines_in_cta(&a.single, 1));
        queue = queue && few_groups(n, lean, num_sms);
        args.after_march = queue ? 1 : 0;
        launch_finalize<Store, RECORD>(args, n, lean, stream, queue, a.worlds == nullptr, num_sms);
    }
    return cudaGetLastError();
}

template <class Store>
cudaError_t passes_t(const LaunchArgs& a, const WorldPass* h_tab, int n_passes, size_t vol_bytes, int num_sms,
                     cudaStream_t stream, bool dependent) {
    const int blocks = march_grid(false, num_sms, a.n_tasks, a.march_ctas);
    LaunchArgs args = a;
    args.total_warps = blocks * kWarps;
    args.chunk_begin = 0;
    args.chunk_end = (int)a.n_tasks;
    args.ray_origin = 0;
    if (a.n_tasks > 0) {
        launch_march(args, h_tab[0], a.n_tasks, num_sms, stream, dependent);
    } else {   // every pass empty: plain copies
        for (int i = 0; i < n_passes; i++) {
            cudaError_t e = cudaMemcpyAsync(h_tab[i].next, h_tab[i].prev, vol_bytes, cudaMemcpyDeviceToDevice, stream);
            if (e != cudaSuccess) return e;
        }
        if (a.clear_stats) return cudaMemsetAsync(a.clear_stats, 0, 2 * sizeof(unsigned long long), stream);
        return cudaSuccess;
    }
    args.clear_stats = nullptr;
    args.time_start = nullptr;
    const bool in_cta = combines_in_cta(h_tab, n_passes);
    const long long probes = (long long)(vol_bytes / sizeof(typename Store::T));
    const int copy_ctas = (int)std::max<long long>(1, std::min<long long>((probes + 255) / 256, 8LL * num_sms));
    for (int i = 0; i < n_passes; i++) {
        const WorldPass& w = h_tab[i];
        args.chunk_begin = (int)w.task_begin;
        args.chunk_end = (int)(w.task_begin + w.n_tasks);
        const int n = args.chunk_end - args.chunk_begin;
        args.copy_src = w.prev;
        args.copy_dst = w.next;
        args.copy_bytes = (long long)vol_bytes;
        args.mask_bit = i;
        args.mask_clear = i == n_passes - 1;
        args.fin_ctas = (n + kFinWarps - 1) / kFinWarps;
        args.fin_copy = copy_ctas;
        args.single = w;   // the launch's tasks are pass i's
        // from the second pass on, the launch overlaps the previous pass's tail: its refine and
        // materials read no volume (the first pass's rays come from the march launch before it)
        launch_finalize<Store, false>(args, n, in_cta, stream, i > 0, true, num_sms);
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_passes(const LaunchArgs& args, const WorldPass* h_tab, int n_passes, size_t vol_bytes,
                          int precision, int num_sms, cudaStream_t stream, bool dependent) {
    if (args.n_tasks > kMultiTasks || n_passes > kMultiPasses || !args.pass_mask) return cudaErrorInvalidValue;
    switch (precision) {
        case LUMRAD_PRECISION_FP16: return passes_t<StoreF16>(args, h_tab, n_passes, vol_bytes, num_sms, stream, dependent);
        case LUMRAD_PRECISION_BF16:
            return passes_t<StoreBF16>(args, h_tab, n_passes, vol_bytes, num_sms, stream, dependent);
        case LUMRAD_PRECISION_RGB10A2:
            return passes_t<StoreRGB10A2>(args, h_tab, n_passes, vol_bytes, num_sms, stream, dependent);
        default: return passes_t<StoreF32>(args, h_tab, n_passes, vol_bytes, num_sms, stream, dependent);
    }
}

cudaError_t launch_table_pass(const LaunchArgs& a, int precision, int num_sms, cudaStream_t stream) {
    const int blocks = march_grid(false, num_sms, a.n_tasks, a.march_ctas);
    LaunchArgs args = a;
    args.total_warps = blocks * kWarps;
    args.chunk_begin = 0;
    args.chunk_end = (int)a.n_tasks;
    args.ray_origin = 0;
    // the CTA queue: the host cannot see the task count, and the device loop's iterations are
    // mostly small (p50 5-8% lower at 2,000-10,000 requests/s than the per-warp queue; 2% less
    // throughput saturated, where the host loop is the faster one anyway)
    march_kernel<false, false, true><<<blocks, kWarps * 32, 0, stream>>>(args);
    const int fin = num_sms * kFinLeanCtas;
    switch (precision) {
        case LUMRAD_PRECISION_FP16: finalize_kernel<StoreF16, false, true, true><<<fin, kFinCtaWarps * 32, 0, stream>>>(args); break;
        case LUMRAD_PRECISION_BF16: finalize_kernel<StoreBF16, false, true, true><<<fin, kFinCtaWarps * 32, 0, stream>>>(args); break;
        case LUMRAD_PRECISION_RGB10A2:
            finalize_kernel<StoreRGB10A2, false, true, true><<<fin, kFinCtaWarps * 32, 0, stream>>>(args);
            break;
        default: finalize_kernel<StoreF32, false, true, true><<<fin, kFinCtaWarps * 32, 0, stream>>>(args);
    }
    return cudaGetLastError();
}

cudaError_t launch_radiance(const LaunchArgs& args, int precision, bool record, int num_sms, cudaStream_t stream,
                            bool dependent) {
    if (args.n_tasks <= 0) {   // no march launch: the pass's start as copies
        cudaError_t e = cudaSuccess;
        if (args.copy_dst && args.copy_bytes > 0)
            e = cudaMemcpyAsync(args.copy_dst, args.copy_src, (size_t)args.copy_bytes, cudaMemcpyDeviceToDevice, stream);
        if (e == cudaSuccess && args.clear_stats)
            e = cudaMemsetAsync(args.clear_stats, 0, 2 * sizeof(unsigned long long), stream);
        if (e == cudaSuccess && args.count_dst)
            e = cudaMemcpyAsync(args.count_dst, args.count_src, sizeof(int), cudaMemcpyDeviceToDevice, stream);
        return e;
    }
    switch (precision) {
        case LUMRAD_PRECISION_FP16:
            return record ? launch_t<StoreF16, true>(args, num_sms, stream, false) : launch_t<StoreF16, false>(args, num_sms, stream, dependent);
        case LUMRAD_PRECISION_BF16:
            return record ? launch_t<StoreBF16, true>(args, num_sms, stream, false) : launch_t<StoreBF16, false>(args, num_sms, stream, dependent);
        case LUMRAD_PRECISION_RGB10A2:
            return record ? launch_t<StoreRGB10A2, true>(args, num_sms, stream, false)
                          : launch_t<StoreRGB10A2, false>(args, num_sms, stream, dependent);
        default:
            return record ? launch_t<StoreF32, true>(args, num_sms, stream, false) : launch_t<StoreF32, false>(args, num_sms, stream, dependent);
    }
}

}  // namespace lumrad

namespace lumrad {
namespace {

// Start of a batched pass: each world's next volume becomes a copy of its previous one (probes
// not in its list keep their value) and its counters are cleared.  blockIdx.y = world.
template <typename V>
__global__ void prep_kernel(const WorldPass* __restrict__ worlds, const int* dev_n) {
    if (dev_n && (int)blockIdx.y >= __ldcg(dev_n)) return;   // a table built on the device
    const WorldPass& w = worlds[blockIdx.y];
    const long long n = (long long)w.X * w.Y * w.Z;
    const V* src = reinterpret_cast<const V*>(w.prev);
    V* dst = reinterpret_cast<V*>(w.next);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = src[i];
    if (blockIdx.x == 0 && threadIdx.x < 2) w.stats[threadIdx.x] = 0;
}

}  // namespace

cudaError_t launch_prep(const WorldPass* d_worlds, int n_worlds, int precision, cudaStream_t stream, const int* dev_n) {
    if (n_worlds <= 0) return cudaSuccess;
    const dim3 grid(32, n_worlds);
    if (precision == LUMRAD_PRECISION_FP32) prep_kernel<uint4><<<grid, 256, 0, stream>>>(d_worlds, dev_n);
    else if (precision == LUMRAD_PRECISION_RGB10A2) prep_kernel<unsigned><<<grid, 256, 0, stream>>>(d_worlds, dev_n);
    else prep_kernel<uint2><<<grid, 256, 0, stream>>>(d_worlds, dev_n);
    return cudaGetLastError();
}

namespace {

__global__ void apply_edits_kernel(const WorldPass* __restrict__ worlds, const EditRecord* __restrict__ edits, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const EditRecord e = edits[i];
    const WorldPass& w = worlds[e.world];
    const_cast<int16_t*>(w.grid)[e.index] = (int16_t)e.block;
    const int x = e.index % w.X, q = e.index / w.X;
    const size_t cell = x + (size_t)(w.X + 1) * (q % w.Y + (size_t)(w.Y + 1) * (q / w.Y));
    if (w.cgrid_wide) static_cast<uint16_t*>(const_cast<void*>(w.cgrid))[cell] = (uint16_t)e.compact;
    else static_cast<uint8_t*>(const_cast<void*>(w.cgrid))[cell] = (uint8_t)e.compact;
}

}  // namespace

cudaError_t launch_apply_edits(const WorldPass* d_worlds, const EditRecord* d_edits, int n, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    apply_edits_kernel<<<(n + 255) / 256, 256, 0, stream>>>(d_worlds, d_edits, n);
    return cudaGetLastError();
}

}  // namespace lumrad

// ================================================================ no-allocation entry point
//
// lumrad_radiance_pass_noalloc runs the same two kernels as a context's pass, but every working
// buffer lives in one fixed array compiled into this library (g_noalloc_scratch below), so the
// call itself never allocates device memory.  It exists for callers that may not allocate while
// they run a frame: engines that reserve their whole device-memory budget at start-up and forbid
// allocation afterwards (an allocation can synchronise the device and stall the frame), and hosts
// whose own allocator owns the device heap.  Such a caller owns the inputs and outputs and passes
// them as device pointers; the array holds the rest: the compact copy of the world, the rays of
// one round, the direction table and the queue.
//
// Limits: worlds of at most LUMRAD_NOALLOC_MAX_BLOCKS blocks, 32/64/128/256 rays per probe (a
// probe's subgroups then combine inside one CTA, so no per-probe scratch is needed), FP32
// radiance, no hit records.  Rounds of kNoAllocRoundTasks tasks.

#include "lumrad_world.h"
#include <mutex>

namespace lumrad {
namespace {

constexpr int kNoAllocMaxBlocks = LUMRAD_NOALLOC_MAX_BLOCKS;
// The most tasks of a round: 4,096, as many as the array holds beside the compact grid (noalloc_round_tasks).  (At
// 3,840, beside room for the largest grid of all, a pass of 4,096 tasks took two rounds: 16x16x8 blocks, 64
// rays, 70.2 us a call; one round, and its finalize with a warp per task, 44.2.)
constexpr int kNoAllocRoundTasks = 4096;
// the most cells of a compact grid of kNoAllocMaxBlocks blocks (compact_cells): a world of one
// block's height, 2047 blocks long
constexpr size_t kNoAllocMaxCells = 2 * ((size_t)kNoAllocMaxBlocks + 2047 + kNoAllocMaxBlocks / 2047 + 1);
constexpr size_t align256(size_t v) { return (v + 255) & ~size_t(255); }
// byte offsets of the parts of the array
constexpr size_t kNaCbits = 0;                                                        // 512 B per compact id
// the direction tables for R = 32, 64, 128, 256 back to back (480 entries), uploaded once per device
constexpr size_t kNaDirs = align256(kNaCbits + (size_t)(LUMRAD_MAX_BLOCK_SLOTS + 2) * 512);
constexpr int kNaDirEntries = 32 + 64 + 128 + 256;
constexpr size_t kNaQueue = align256(kNaDirs + kNaDirEntries * sizeof(float4));
constexpr size_t kNaError = kNaQueue + kQueueWords * sizeof(unsigned long long);
constexpr size_t kNaStats = align256(kNaError + sizeof(int));
constexpr size_t kNaCgrid = align256(kNaStats + 2 * sizeof(unsigned long long));     // uint16 per cell, then the rays
constexpr size_t kNaBytes = 8u << 20;
// Tasks of a round over a world of `cells` compact-grid cells: a multiple of 8 (a probe's subgroups share a
// CTA of the finalize).
constexpr int noalloc_round_tasks(size_t cells) {
    const size_t room = (kNaBytes - align256(kNaCgrid + 2 * cells)) / (kTaskRays * kRayBytes) / kFinWarps * kFinWarps;
    return room < (size_t)kNoAllocRoundTasks ? (int)room : kNoAllocRoundTasks;
}
static_assert(noalloc_round_tasks(kNoAllocMaxCells) >= 4000, "rounds as long beside any grid");

}  // namespace
}  // namespace lumrad

// The scratch array: one per GPU that loads this library, held until the process exits.  In host
// code `g_noalloc_scratch` only names the symbol; its device address comes from
// cudaGetSymbolAddress (done once per device, below).
static __device__ __align__(256) unsigned char g_noalloc_scratch[lumrad::kNaBytes];

namespace lumrad {
namespace {

// Compact ids for the no-allocation form: 0 for block id 0 (palette slot 0), 1 + slot for a
// non-zero id with a palette slot, n_slots + 1 (all empty) for any other id.
__global__ void noalloc_compact_grid(const int16_t* __restrict__ grid, int X, int Y, int Z, int n_slots,
                                     uint16_t* __restrict__ cgrid) {
    const int n = (X + 1) * (Y + 1) * (Z + 1);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int x = i % (X + 1), q = i / (X + 1), y = q % (Y + 1), z = q / (Y + 1);
        const int b = x < X && y < Y && z < Z ? grid[x + X * (y + Y * z)] : 0;
        const int slot = b < 0 ? b + 64 : b;
        const bool has = b >= -63 && slot < n_slots;
        cgrid[i] = (uint16_t)(b == 0 ? 0 : (has ? slot + 1 : n_slots + 1));
    }
}

// Occupancy words: entry 0 = slot 0, entry 1 + s = slot s, entry n_slots + 1 = empty.
__global__ void noalloc_compact_bits(const uint8_t* __restrict__ pal, int n_slots, uint32_t* __restrict__ bits) {
    const int n_words = (n_slots + 2) * 128;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_words; i += gridDim.x * blockDim.x) {
        const int e = i >> 7, word = i & 127;
        const int slot = e == 0 ? 0 : e - 1;
        uint32_t v = 0;
        if (e <= n_slots) {
            const uint8_t* p = pal + (size_t)slot * 4096 + word * 32;
            for (int b = 0; b < 32; b++) v |= (p[b] != 0 ? 1u : 0u) << b;
        }
        bits[i] = v;
    }
}

struct NoAllocDevice {
    bool ready = false;
    unsigned char* base = nullptr;   // device address of g_noalloc_scratch on this device
    int num_sms = 0;
};
std::mutex g_noalloc_mutex;
NoAllocDevice g_noalloc_dev[64];

// Offset (entries) of the direction table for R rays in the array's table area.
int noalloc_dir_offset(int R) { return R == 32 ? 0 : R == 64 ? 32 : R == 128 ? 96 : 224; }

// The array's device address on the current device, set up on the first call there: the address
// lookup, the SM count and the four direction tables (one synchronous upload, before any pass of
// this device can read them).  Sets *out to null on failure (and returns the status).
int noalloc_device(NoAllocDevice** out) {
    *out = nullptr;
    int dev = 0;
    LUMRAD_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(LUMRAD_EINVAL, "device ordinal beyond 63");
    NoAllocDevice* nd = &g_noalloc_dev[dev];
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!nd->ready) {
        void* addr = nullptr;
        LUMRAD_TRY(cudaGetSymbolAddress(&addr, g_noalloc_scratch));
        LUMRAD_TRY(cudaDeviceGetAttribute(&nd->num_sms, cudaDevAttrMultiProcessorCount, dev));
        float4 tab[kNaDirEntries];
        float xyz[3 * 256];
        for (int R = 32; R <= 256; R *= 2) {
            fibonacci_table(R, xyz);
            for (int i = 0; i < R; i++)
                tab[noalloc_dir_offset(R) + i] = make_float4(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], 0.0f);
        }
        unsigned char* base = static_cast<unsigned char*>(addr);
        LUMRAD_TRY(cudaMemcpy(base + kNaDirs, tab, sizeof tab, cudaMemcpyHostToDevice));
        nd->base = base;
        nd->ready = true;
    }
    *out = nd;
    return LUMRAD_OK;
}

}  // namespace
}  // namespace lumrad

using namespace lumrad;

extern "C" int lumrad_radiance_pass_noalloc(const int* world_size, const int16_t* d_grid, const uint8_t* d_palette,
                                            int n_slots, const float* d_materials, const int16_t* d_requests, int n,
                                            const float* d_prev, float* d_next, const LumRadPassParams* p,
                                            void* stream_handle) {
    if (!world_size || !d_grid || !d_palette || !d_materials || !d_prev || !d_next || !p || (n > 0 && !d_requests))
        return fail(LUMRAD_EINVAL, "null argument");
    int rc = check_params(p);
    if (rc) return rc;
    if (p->size < 1) return fail(LUMRAD_EINVAL, "size must be >= 1 (no adaptive slicing here)");
    if (p->record_hits) return fail(LUMRAD_EINVAL, "hit records need lumrad_radiance_pass");
    const int R = p->rays_per_probe;
    if (R != 32 && R != 64 && R != 128 && R != 256) return fail(LUMRAD_EINVAL, "rays_per_probe must be 32, 64, 128 or 256");
    for (int i = 0; i < 3; i++)
        if (world_size[i] < 1 || world_size[i] > 2047) return fail(LUMRAD_EINVAL, "world_size must be in [1, 2047] per axis");
    const long long W = (long long)world_size[0] * world_size[1] * world_size[2];
    if (W > kNoAllocMaxBlocks) return fail(LUMRAD_EINVAL, "world larger than LUMRAD_NOALLOC_MAX_BLOCKS blocks");
    {   // the pass reads prev while it writes next: the two volumes must not share bytes
        const uintptr_t a = reinterpret_cast<uintptr_t>(d_prev), b = reinterpret_cast<uintptr_t>(d_next);
        const uintptr_t bytes = (uintptr_t)W * sizeof(float4);
        if (a < b + bytes && b < a + bytes) return fail(LUMRAD_EINVAL, "d_prev and d_next overlap");
    }
    if (n_slots < 1 || n_slots > LUMRAD_MAX_BLOCK_SLOTS) return fail(LUMRAD_EINVAL, "n_slots must be in [1, 4096]");
    if (n < 0) return fail(LUMRAD_EINVAL, "negative request count");
    const long long groups = n / p->size;
    const long long n_tasks = groups * (R / 32);
    if (n_tasks >= (1LL << 31)) return fail(LUMRAD_EINVAL, "pass has too many subgroups (>= 2^31)");
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_handle);

    // set-up, once per device (the first call there; make that call before capturing a stream
    // into a graph): the array's device address and the direction tables
    NoAllocDevice* nd = nullptr;
    if ((rc = noalloc_device(&nd))) return rc;
    unsigned char* base = nd->base;
    uint16_t* cgrid = reinterpret_cast<uint16_t*>(base + kNaCgrid);
    uint32_t* cbits = reinterpret_cast<uint32_t*>(base + kNaCbits);
    const float4* dirs = reinterpret_cast<const float4*>(base + kNaDirs) + noalloc_dir_offset(R);
    unsigned long long* queue = reinterpret_cast<unsigned long long*>(base + kNaQueue);
    int* error = reinterpret_cast<int*>(base + kNaError);
    unsigned long long* stats = reinterpret_cast<unsigned long long*>(base + kNaStats);

    // what must start at zero (the error word is kept until lumrad_radiance_pass_noalloc_status
    // reads it), and this call's inputs derived into the array
    LUMRAD_TRY(cudaMemsetAsync(queue, 0, kQueueWords * sizeof(unsigned long long), stream));
    LUMRAD_TRY(cudaMemsetAsync(stats, 0, 2 * sizeof(unsigned long long), stream));
    noalloc_compact_grid<<<256, 256, 0, stream>>>(d_grid, world_size[0], world_size[1], world_size[2], n_slots, cgrid);
    noalloc_compact_bits<<<256, 256, 0, stream>>>(d_palette, n_slots, cbits);
    LUMRAD_TRY(cudaGetLastError());
    // probes outside the list keep their value
    LUMRAD_TRY(cudaMemcpyAsync(d_next, d_prev, (size_t)W * sizeof(float4), cudaMemcpyDeviceToDevice, stream));
    if (n_tasks == 0) return LUMRAD_OK;

    LaunchArgs la;
    std::memset(&la, 0, sizeof la);
    WorldPass& w = la.single;
    w.X = world_size[0]; w.Y = world_size[1]; w.Z = world_size[2];
    w.cgrid_wide = 1;
    w.cgrid = cgrid;
    w.cbits = cbits;
    w.grid = d_grid;
    w.pal = d_palette;
    w.n_slots = n_slots;
    w.mats = reinterpret_cast<const float4*>(d_materials);
    w.prev = d_prev;
    w.next = d_next;
    w.req = reinterpret_cast<const short4*>(d_requests);
    w.n_groups = (int)groups;
    w.size = p->size;
    w.shift = p->shift;
    w.R = R;
    w.max_dist = p->max_dist;
    w.max_steps = (int)(2.0f * p->max_dist) + 2;
    w.alpha = p->blend;
    w.one_minus_alpha = 1.0f - p->blend;
    w.seed = (uint32_t)p->time_seed;
    for (int i = 0; i < 3; i++) {
        w.inv_dim[i] = 1.0f / (float)world_size[i];
    }
    w.inv_nsub = 1.0f / (float)(R / 32);
    w.dirs = dirs;
    w.stats = stats;
    w.task_begin = 0;
    w.n_tasks = n_tasks;
    la.n_worlds = 1;
    la.n_tasks = n_tasks;
    la.queue = queue;
    la.error = error;
    const size_t cells = compact_cells(w.X, w.Y, w.Z);
    const int round = noalloc_round_tasks(cells);
    la.rays = ray_buffer(base + align256(kNaCgrid + 2 * cells), (size_t)round * kTaskRays);
    const int blocks = march_grid(false, nd->num_sms, std::min<long long>(n_tasks, round));
    la.total_warps = blocks * kWarps;
    for (long long c0 = 0; c0 < n_tasks; c0 += round) {
        la.chunk_begin = (int)c0;
        la.chunk_end = (int)std::min(c0 + (long long)round, n_tasks);
        la.ray_origin = la.chunk_begin;
        const int tasks = la.chunk_end - la.chunk_begin;
        if (tasks < kCtaQueueTasksPerWarp * la.total_warps) march_kernel<false, false, true><<<blocks, kWarps * 32, 0, stream>>>(la);
        else march_kernel<false><<<blocks, kWarps * 32, 0, stream>>>(la);
        // (a round has few groups: kFinFewGroups)
        finalize_kernel<StoreF32, false, true, false, true, kFinWarps>
            <<<(tasks + kFinWarps - 1) / kFinWarps, kFinWarps * 32, 0, stream>>>(la);
    }
    LUMRAD_TRY(cudaGetLastError());
    return LUMRAD_OK;
}

extern "C" int lumrad_radiance_pass_noalloc_status(void* stream_handle, int* device_error) {
    if (!device_error) return fail(LUMRAD_EINVAL, "null argument");
    *device_error = 0;
    NoAllocDevice* nd = nullptr;
    if (int rc = noalloc_device(&nd)) return rc;
    cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_handle);
    int* error = reinterpret_cast<int*>(nd->base + kNaError);
    int word = 0;
    LUMRAD_TRY(cudaMemcpyAsync(&word, error, sizeof(int), cudaMemcpyDeviceToHost, stream));
    LUMRAD_TRY(cudaStreamSynchronize(stream));
    if (word == 0) return LUMRAD_OK;
    LUMRAD_TRY(cudaMemsetAsync(error, 0, sizeof(int), stream));
    LUMRAD_TRY(cudaStreamSynchronize(stream));
    *device_error = word;
    return fail(LUMRAD_EDEVICE, "a no-allocation pass since the last status call did not complete (radiance "
                                "kernel scheduler stopped making progress, code " + std::to_string(word) + ")");
}
