// radiance_aux.cu — the device work either side of the radiance pass:
//
//   update list   the probes update_radiance relights each frame (internal_render.cpp:1142-1168):
//                 every block whose clamped 3x3x3 neighbourhood has a positive id sum, in scan
//                 order, then each special request whose block is not already listed, in request
//                 order.  Two launches: flag (one bit per block, ballot) + per-CTA counts, and an
//                 order-preserving write; a scan of the counts between them for worlds of more than a
//                 million blocks, and a third launch when there are specials.
//   scroll        shift_radiance (internal_render.cpp:1218-1335): new(p) = old(p + shift) where
//                 p + shift is inside the world, old(p) elsewhere; one pass into the other
//                 ping-pong volume.
//   gather        the 8-probe consumer read of diffuse.frag:36-90 (sample_radiance(position,
//                 normal)): trilinear weights times a clamped directional weight over the 8
//                 surrounding probes, probe values clamped to [0, 2].
//
// All FP32 arithmetic is written out in the shader's order with round-to-nearest intrinsics (no
// contraction), so results are reproducible bit for bit.

#include "radiance_device.cuh"
#include "lumrad_launch.h"

#include <algorithm>

namespace lumrad {
namespace {

constexpr int kListCta = 256;      // blocks per CTA of the list kernels (8 warps)
constexpr int kScanCta = 1024;

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// The list kernels are bound by launch latency (a few us each, about 1 us of work at 65,536 blocks): two
// launches instead of four, and the frame's kernels (scroll, list, march, finalize of few groups,
// gather) each a programmatic dependent of the one before.  A lone 8x8x8 / 19x38x9 / 45x38x11 frame:
// 39.6 / 57.2 / 81.2 -> 22.6 / 38.8 / 62.8 us from call to result; among others (frames back to back) 8x8x8
// 18.9 -> 13.4 us.
//
// The flags and counts (the grid does not come from a kernel: they are formed while the stream's
// previous kernel still runs, then this one waits for it; see launch_kernel).
__global__ void __launch_bounds__(kListCta)
list_flags_kernel(const int16_t* __restrict__ grid, int X, int Y, int Z, unsigned W, uint32_t* __restrict__ bits,
                  int* __restrict__ cta_counts) {
    grid_launch_dependents();
    __shared__ int s_cnt[kListCta / 32];
    const unsigned i = blockIdx.x * kListCta + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    bool flag = false;
    if (i < W) {
        const unsigned q = i / (unsigned)X;
        const int x = (int)(i - q * X), z = (int)(q / (unsigned)Y), y = (int)(q - (unsigned)z * Y);
        const int xs[3] = {max(x - 1, 0), x, min(x + 1, X - 1)};
        int sum = 0;   // sum of the 27 clamped neighbours' ids (internal_render.cpp:1147-1156)
#pragma unroll
        for (int dz = -1; dz <= 1; dz++) {
            const int tz = clampi(z + dz, 0, Z - 1);
#pragma unroll
            for (int dy = -1; dy <= 1; dy++) {
                const int ty = clampi(y + dy, 0, Y - 1);
                const int16_t* row = grid + (size_t)X * ((size_t)ty + (size_t)Y * tz);
#pragma unroll
                for (int k = 0; k < 3; k++) sum += __ldg(row + xs[k]);
            }
        }
        flag = sum > 0;
    }
    const unsigned b = __ballot_sync(kFull, flag);
    if (lane == 0) s_cnt[warp] = __popc(b);
    __syncthreads();
    grid_dependency_wait();
    if (lane == 0 && i < W) bits[i >> 5] = b;
    if (threadIdx.x == 0) {
        int c = 0;
        for (int w = 0; w < kListCta / 32; w++) c += s_cnt[w];
        cta_counts[blockIdx.x] = c;
    }
}

// Exclusive scan of `v` over the CTA (kScanCta threads); returns the CTA total through *total.
__device__ __forceinline__ int cta_exclusive_scan(int v, int* s_warp, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += t;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(kFull, w, o);
            if (lane >= o) w += t;
        }
        s_warp[lane] = w;
    }
    __syncthreads();
    const int excl = x - v + (warp > 0 ? s_warp[warp - 1] : 0);
    *total = s_warp[31];
    __syncthreads();   // s_warp is reused by the next call
    return excl;
}

__global__ void __launch_bounds__(kScanCta)
list_scan_kernel(const int* __restrict__ counts, int n, int* __restrict__ offsets, int* __restrict__ total) {
    __shared__ int s_warp[32];
    int carry = 0;
    for (int base = 0; base < n; base += kScanCta) {
        const int i = base + threadIdx.x;
        const int v = i < n ? counts[i] : 0;
        int chunk = 0;
        const int excl = cta_exclusive_scan(v, s_warp, &chunk);
        if (i < n) offsets[i] = carry + excl;
        carry += chunk;
    }
    if (threadIdx.x == 0) *total = carry;
}

// The list from the bits.  A CTA's offset: offsets[blockIdx.x] of a scan of the counts; or, offsets
// null (up to kDirectCtas CTAs), the sum of the counts before its own; or, both null (up to
// kBitsCtas), of the bits before its own; the last CTA then also writes the length.
// The lines: with the scan / the counts summed, the update list of 65,536 / 524,288 / 1,081,344 / 2,097,152 /
// 4,194,304 blocks takes 27.8 / 31.3 / 41.0 / 64 / 98 and 17.3 / 26 / 38.6 / 53 / 100 us a call (the sums grow
// with the square of the CTAs); the dirty list of 328 edits, by the dilation / from the bits, in
// 262,144 / 524,288 / 1,048,576 / 2,097,152 blocks 66 / 70 / 82 / 106 and 39 / 44 / 56 / 98.
constexpr int kDirectCtas = 4096, kBitsCtas = 1024;
__global__ void __launch_bounds__(kListCta)
list_write_kernel(const uint32_t* bits, const int* counts, const int* offsets, int X, int Y, unsigned W, short4* out, int* total,
                  int* total2) {
    grid_launch_dependents();
    __shared__ int s_pre[kListCta / 32], s_sum[kListCta / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned i = blockIdx.x * kListCta + threadIdx.x;
    const unsigned q = i / (unsigned)X, z = q / (unsigned)Y;
    grid_dependency_wait();
    const uint32_t b = i < W ? __ldcg(bits + (i >> 5)) : 0u;
    int sum = 0;
    if (!counts) {   // (a CTA's words: two uint4)
        const uint4* v = reinterpret_cast<const uint4*>(bits);
        for (int c = threadIdx.x; c < 2 * (int)blockIdx.x; c += kListCta) {
            const uint4 x = __ldcg(v + c);
            sum += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
        }
    } else if (!offsets)
        for (int c = threadIdx.x; c < (int)blockIdx.x; c += kListCta) sum += __ldcg(counts + c);
    sum = __reduce_add_sync(kFull, sum);
    if (lane == 0) {
        s_pre[warp] = __popc(b);
        s_sum[warp] = sum;
    }
    __syncthreads();
    int pos = offsets ? offsets[blockIdx.x] : 0, all = 0;
    for (int w = 0; w < kListCta / 32; w++) {
        pos += s_sum[w] + (w < warp ? s_pre[w] : 0);
        all += s_pre[w];
    }
    if (total && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        *total = pos + all;
        if (total2) *total2 = pos + all;
    }
    if (!((b >> lane) & 1u)) return;
    out[pos + __popc(b & ((1u << lane) - 1u))] = make_short4((short)(i - q * X), (short)(q - z * Y), (short)z, 0);
}

// Launches of the list from bits and counts: the length into *total (and *total2 if not null).
cudaError_t launch_list_write(const ListScratch& s, int X, int Y, long long W, short4* out, int* total, int* total2,
                              cudaStream_t stream) {
    const int ctas = (int)((W + kListCta - 1) / kListCta);
    if (ctas <= kDirectCtas)
        return launch_kernel(list_write_kernel, ctas, kListCta, 0, stream, true, s.bits, s.cta_counts, nullptr, X, Y, (unsigned)W,
                             out, total, total2);
    list_scan_kernel<<<1, kScanCta, 0, stream>>>(s.cta_counts, ctas, s.cta_offsets, total);
    if (total2) {
        const cudaError_t e = cudaMemcpyAsync(total2, total, sizeof(int), cudaMemcpyDeviceToDevice, stream);
        if (e != cudaSuccess) return e;
    }
    return launch_kernel(list_write_kernel, ctas, kListCta, 0, stream, false, s.bits, s.cta_counts, s.cta_offsets, X, Y,
                         (unsigned)W, out, nullptr, nullptr);
}

// Dirty probes of a few edits (Chebyshev distance <= r): each row of an edit's cube inside the world sets
// its run of bits, a thread per row; the list is then written from the bits.  A memset and two launches,
// where the dilation below takes a memset and five: used where dirty_rows_fit says.
__global__ void dirty_rows_kernel(const short4* __restrict__ edits, int rows, int X, int Y, int Z, int r,
                                  uint32_t* __restrict__ bits) {
    grid_launch_dependents();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= rows) return;
    const int ny = min(2 * r + 1, Y), nz = min(2 * r + 1, Z), row = k % (ny * nz);
    const short4 e = edits[k / (ny * nz)];
    const int y = max(e.y - r, 0) + row % ny, z = max(e.z - r, 0) + row / ny;
    if (y > min(e.y + r, Y - 1) || z > min(e.z + r, Z - 1)) return;
    const int x0 = max(e.x - r, 0), x1 = min(e.x + r, X - 1);   // at most 31 blocks: two words
    const unsigned i0 = (unsigned)x0 + (unsigned)X * ((unsigned)y + (unsigned)Y * (unsigned)z), i1 = i0 + (unsigned)(x1 - x0);
    const uint32_t m0 = ~0u << (i0 & 31), m1 = ~0u >> (31 - (i1 & 31));
    if ((i0 >> 5) == (i1 >> 5)) {
        atomicOr(bits + (i0 >> 5), m0 & m1);
    } else {
        atomicOr(bits + (i0 >> 5), m0);
        atomicOr(bits + (i1 >> 5), m1);
    }
}

// Dirty probes of block edits (Chebyshev distance <= r): a byte mask of the edited blocks, dilated
// along x, then y, then z; the last pass writes one bit per block and the CTA counts, as
// list_flags_kernel does, so list_scan_kernel and list_write_kernel emit the list in scan order.
__global__ void dirty_mark_kernel(const short4* __restrict__ edits, int n, int X, int Y, uint8_t* __restrict__ mask) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const short4 e = edits[k];
    mask[(size_t)e.x + (size_t)X * ((size_t)e.y + (size_t)Y * e.z)] = 1;
}

// one axis of the dilation: out[i] = OR of in over [-r, r] steps of `stride` along an axis of n
__global__ void dirty_dilate_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, int X, int Y, int Z,
                                    int axis, int r, long long W) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < W; i += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(i % X);
        const long long q = i / X;
        const int y = (int)(q % Y), z = (int)(q / Y);
        const int c = axis == 0 ? x : (axis == 1 ? y : z);
        const int n = axis == 0 ? X : (axis == 1 ? Y : Z);
        const long long stride = axis == 0 ? 1 : (axis == 1 ? (long long)X : (long long)X * Y);
        uint8_t v = 0;
        for (int d = max(c - r, 0); d <= min(c + r, n - 1); d++) v |= __ldg(in + i + (long long)(d - c) * stride);
        out[i] = v;
    }
}

__global__ void __launch_bounds__(kListCta)
dirty_flags_kernel(const uint8_t* __restrict__ in, int X, int Y, int Z, int r, long long W, uint32_t* __restrict__ bits,
                   int* __restrict__ cta_counts) {
    __shared__ int s_cnt[kListCta / 32];
    const long long i = (long long)blockIdx.x * kListCta + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    bool flag = false;
    if (i < W) {   // the z pass of the dilation
        const long long XY = (long long)X * Y;
        const int z = (int)(i / XY);
        for (int d = max(z - r, 0); d <= min(z + r, Z - 1) && !flag; d++) flag = __ldg(in + i + (long long)(d - z) * XY) != 0;
    }
    const unsigned b = __ballot_sync(kFull, flag);
    const long long word = i >> 5;
    if (lane == 0) {
        if (word < (W + 31) / 32) bits[word] = b;
        s_cnt[warp] = __popc(b);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int c = 0;
        for (int w = 0; w < kListCta / 32; w++) c += s_cnt[w];
        cta_counts[blockIdx.x] = c;
    }
}

// Specials in request order, each unless its block is already listed (duplicates are kept, as
// in the reference: `set` only marks rule-listed blocks).
__global__ void __launch_bounds__(kScanCta)
list_specials_kernel(const short4* __restrict__ sp, int ns, const uint32_t* __restrict__ bits, int X, int Y,
                     const int* __restrict__ listed, short4* __restrict__ out, int* __restrict__ count) {
    __shared__ int s_warp[32];
    int carry = *listed;
    for (int base = 0; base < ns; base += kScanCta) {
        const int i = base + threadIdx.x;
        int keep = 0;
        short4 s = make_short4(0, 0, 0, 0);
        if (i < ns) {
            s = sp[i];
            const long long idx = (long long)s.x + (long long)X * ((long long)s.y + (long long)Y * s.z);
            keep = ((bits[idx >> 5] >> (idx & 31)) & 1u) ? 0 : 1;
        }
        int chunk = 0;
        const int excl = cta_exclusive_scan(keep, s_warp, &chunk);
        if (keep) out[carry + excl] = s;
        carry += chunk;
    }
    if (threadIdx.x == 0) *count = carry;
}

template <typename V>
__global__ void shift_kernel(const V* src, V* dst, int X, int Y, int Z, int sx, int sy,
                             int sz, long long W) {
    grid_launch_dependents();
    grid_dependency_wait();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < W; i += (long long)gridDim.x * blockDim.x) {
        const unsigned q = (unsigned)i / (unsigned)X;
        const int x = (int)((unsigned)i - q * X), z = (int)(q / (unsigned)Y), y = (int)(q - (unsigned)z * Y);
        const int qx = x + sx, qy = y + sy, qz = z + sz;
        const bool inside = qx >= 0 && qx < X && qy >= 0 && qy < Y && qz >= 0 && qz < Z;
        dst[i] = inside ? src[(size_t)qx + (size_t)X * ((size_t)qy + (size_t)Y * qz)] : src[i];
    }
}

// sample_probe (diffuse.frag:25-33): texelFetch at the clamped probe (outside the volume reads 0,
// the robust-access definition), clamped to [0, 2].
template <class Store>
__device__ __forceinline__ float3 gather_probe(const typename Store::T* rad, int X, int Y, int Z, int px, int py,
                                               int pz) {
    px = clampi(px, 0, X);
    py = clampi(py, 0, Y);
    pz = clampi(pz, 0, Z);
    float3 v = make_float3(0.0f, 0.0f, 0.0f);
    if (px < X && py < Y && pz < Z) v = Store::load(rad, (int)((size_t)px + (size_t)X * ((size_t)py + (size_t)Y * pz)));
    return make_float3(gmin(gmax(v.x, 0.0f), 2.0f), gmin(gmax(v.y, 0.0f), 2.0f), gmin(gmax(v.z, 0.0f), 2.0f));
}

// One point by the shader's own steps, for every input (NaN, infinities, a point on a probe).
template <class Store>
__device__ __noinline__ float3 gather_general(const typename Store::T* rad, int X, int Y, int Z, float px, float py,
                                              float pz, float nx, float ny, float nz) {
    // zero probe: clamp(ivec3(floor(position - 8.0)) / 16, 0, world_size)   (:42)
    const int zx = clampi(f2i(floorf(fsub(px, 8.0f))) / 16, 0, X);
    const int zy = clampi(f2i(floorf(fsub(py, 8.0f))) / 16, 0, Y);
    const int zz = clampi(f2i(floorf(fsub(pz, 8.0f))) / 16, 0, Z);
    const float cx = fadd(fmul((float)zx, 16.0f), 8.0f);   // (:43)
    const float cy = fadd(fmul((float)zy, 16.0f), 8.0f);
    const float cz = fadd(fmul((float)zz, 16.0f), 8.0f);
    // alpha = clamp((position - zero_probe_pos) / 16, 0, 1)   (:45); x/16 == x*0.0625 exactly
    const float ax = gmin(gmax(fmul(fsub(px, cx), 0.0625f), 0.0f), 1.0f);
    const float ay = gmin(gmax(fmul(fsub(py, cy), 0.0625f), 0.0f), 1.0f);
    const float az = gmin(gmax(fmul(fsub(pz, cz), 0.0625f), 0.0f), 1.0f);
    float tw = 0.0f, tr = 0.0f, tg = 0.0f, tb = 0.0f;
#pragma unroll 1
    for (int i = 0; i < 8; i++) {
        const int ox = i & 1, oy = (i >> 1) & 1, oz = (i >> 2) & 1;   // (:50)
        const float fx = (float)ox, fy = (float)oy, fz = (float)oz;
        const float3 ptp = make_float3(fsub(fadd(cx, fmul(fx, 16.0f)), px), fsub(fadd(cy, fmul(fy, 16.0f)), py),
                                       fsub(fadd(cz, fmul(fz, 16.0f)), pz));   // (:55-57)
        const float3 dir = normalize3(ptp);   // (:58)
        // mix(1 - alpha, alpha, offset) = (1-alpha)*(1-offset) + alpha*offset   (:60)
        const float tx = fadd(fmul(fsub(1.0f, ax), fsub(1.0f, fx)), fmul(ax, fx));
        const float ty = fadd(fmul(fsub(1.0f, ay), fsub(1.0f, fy)), fmul(ay, fy));
        const float tz = fadd(fmul(fsub(1.0f, az), fsub(1.0f, fz)), fmul(az, fz));
        float w = fmul(fmul(tx, ty), tz);   // (:61)
        const float d = fadd(fadd(fmul(dir.x, nx), fmul(dir.y, ny)), fmul(dir.z, nz));
        w = fmul(w, gmin(gmax(d, 0.1f), 1.0f));   // (:70-74)
        const float3 c = gather_probe<Store>(rad, X, Y, Z, zx + ox, zy + oy, zz + oz);   // (:81)
        w = gmax(1e-7f, w);   // (:84)
        tw = fadd(tw, w);
        tr = fadd(tr, fmul(w, c.x));
        tg = fadd(tg, fmul(w, c.y));
        tb = fadd(tb, fmul(w, c.z));
    }
    return make_float3(fdiv(tr, tw), fdiv(tg, tw), fdiv(tb, tw));   // (:89)
}

// The same bits for a finite point within 2^18 of the origin, 2^-20 or more from every probe, with a
// normal below 2^60 (no NaN or infinity can occur, so the hardware's min/max serve), with the parts
// that corners share formed once, the two corners of an x pair in one register pair, and the
// normalisations without range checks (sqrt_normal and rcp_normal).  The volume holds values in
// [0, 1], on which the [0, 2] clamp does nothing.  Squares and distances are kept negated, so that
// each residual is one paired FMA.
template <class Store>
__device__ __forceinline__ float3 gather_point(const typename Store::T* rad, int X, int Y, int Z, float px,
                                               float py, float pz, float nx, float ny, float nz) {
    const int zx = min(max(__float2int_rd(fsub(px, 8.0f)), 0) >> 4, X);
    const int zy = min(max(__float2int_rd(fsub(py, 8.0f)), 0) >> 4, Y);
    const int zz = min(max(__float2int_rd(fsub(pz, 8.0f)), 0) >> 4, Z);
    const float cx = (float)(zx * 16 + 8), cy = (float)(zy * 16 + 8), cz = (float)(zz * 16 + 8);
    const float x[2] = {fsub(cx, px), fsub(fadd(cx, 16.0f), px)};
    const float y[2] = {fsub(cy, py), fsub(fadd(cy, 16.0f), py)};
    const float z[2] = {fsub(cz, pz), fsub(fadd(cz, 16.0f), pz)};
    const float xx[2] = {fmul(-x[0], x[0]), fmul(-x[1], x[1])};
    const float yy[2] = {fmul(-y[0], y[0]), fmul(-y[1], y[1])};
    const float zz2[2] = {fmul(-z[0], z[0]), fmul(-z[1], z[1])};
    const bool plain = fadd(fadd(fmaxf(xx[0], xx[1]), fmaxf(yy[0], yy[1])), fmaxf(zz2[0], zz2[1])) <= -9.094947017729282e-13f &&
                       fabsf(px) < 262144.0f && fabsf(py) < 262144.0f && fabsf(pz) < 262144.0f &&
                       fabsf(nx) < 1.152921504606847e18f && fabsf(ny) < 1.152921504606847e18f && fabsf(nz) < 1.152921504606847e18f;
    if (!plain) return gather_general<Store>(rad, X, Y, Z, px, py, pz, nx, ny, nz);
    const float ax = __saturatef(fmul(fsub(px, cx), 0.0625f));
    const float ay = __saturatef(fmul(fsub(py, cy), 0.0625f));
    const float az = __saturatef(fmul(fsub(pz, cz), 0.0625f));
    const f32x2 x2 = pack2(x[0], x[1]), xx2 = pack2(xx[0], xx[1]);
    const f32x2 nx2 = pack2(nx, nx), ny2 = pack2(ny, ny), nz2 = pack2(nz, nz);
    const f32x2 tx2 = pack2(fsub(1.0f, ax), ax), half2v = pack2(0.5f, 0.5f), one2v = pack2(1.0f, 1.0f);
    const float ty[2] = {fsub(1.0f, ay), ay}, tz[2] = {fsub(1.0f, az), az};
    // probes past the volume read 0: their colour weight is 0
    const bool vx[2] = {zx < X, zx + 1 < X}, vy[2] = {zy < Y, zy + 1 < Y}, vz[2] = {zz < Z, zz + 1 < Z};
    const int ix[2] = {min(zx, X - 1), min(zx + 1, X - 1)};
    const int iy[2] = {X * min(zy, Y - 1), X * min(zy + 1, Y - 1)};
    const int iz[2] = {X * Y * min(zz, Z - 1), X * Y * min(zz + 1, Z - 1)};
    float tw = 0.0f, tr = 0.0f, tg = 0.0f, tb = 0.0f;   // in corner order
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int oy = j & 1, oz = j >> 1;
        const float3 c[2] = {Store::load(rad, ix[0] + iy[oy] + iz[oz]), Store::load(rad, ix[1] + iy[oy] + iz[oz])};
        const f32x2 dd = add2(add2(xx2, pack2(yy[oy], yy[oy])), pack2(zz2[oz], zz2[oz]));   // -distance^2
        float a, b, u, v;
        unpack2(dd, a, b);
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(u) : "f"(-a));
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(v) : "f"(-b));
        const f32x2 q = pack2(u, v), g = mul2(dd, q);
        const f32x2 m = fma2(fma2(g, g, dd), mul2(half2v, q), g);   // -distance (sqrt_normal)
        // g*g + dd has the sign of g^2 - distance^2; g and m are negative, so this adds r*h to g
        unpack2(m, a, b);
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(u) : "f"(-a));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(v) : "f"(-b));
        const f32x2 t = pack2(u, v), s = fma2(t, fma2(m, t, one2v), t);   // 1/distance (rcp_normal)
        const f32x2 p1 = mul2(mul2(x2, s), nx2), p2 = mul2(mul2(pack2(y[oy], y[oy]), s), ny2),
                    p3 = mul2(mul2(pack2(z[oz], z[oz]), s), nz2);
        float d0, d1, w0, w1;
        unpack2(add_product2(add_product2(p1, p2), p3), d0, d1);
        const f32x2 d2 = pack2(fminf(fmaxf(d0, 0.1f), 1.0f), fminf(fmaxf(d1, 0.1f), 1.0f));
        unpack2(mul2(mul2(mul2(tx2, pack2(ty[oy], ty[oy])), pack2(tz[oz], tz[oz])), d2), w0, w1);
#pragma unroll
        for (int ox = 0; ox < 2; ox++) {
            const float w = fmaxf(ox ? w1 : w0, 1e-7f);
            const float k = vx[ox] && vy[oy] && vz[oz] ? w : 0.0f;
            tw = fadd(tw, w);
            tr = fadd(tr, fmul(k, c[ox].x));
            tg = fadd(tg, fmul(k, c[ox].y));
            tb = fadd(tb, fmul(k, c[ox].z));
        }
    }
    // tr / tw: with y = RN(1/tw), one residual step on tr*y is the rounded quotient (Markstein 1990)
    // unless a residual could be subnormal (a non-zero sum below 2^-100)
    const unsigned small = 0x0D800000u - 1u;
    if (__float_as_uint(tr) - 1u < small || __float_as_uint(tg) - 1u < small || __float_as_uint(tb) - 1u < small)
        return make_float3(fdiv(tr, tw), fdiv(tg, tw), fdiv(tb, tw));
    const float yw = rcp_normal(tw);
    auto quot = [&](float n) {
        const float q = fmul(n, yw);
        return __fmaf_rn(__fmaf_rn(-q, tw, n), yw, q);
    };
    return make_float3(quot(tr), quot(tg), quot(tb));
}

// Bound by instruction issue (454 warp instructions per 32 points, 72% of the slots; 519 without the
// register pairs; two points per thread, each operation of both paired: 449 at 22 instead of 36
// warps per SM, no faster).  2,073,600 points of a 1920x1080 view: 57.0 -> 30.8 us a call (8 corners
// in a loop before, with checked divisions and square roots: about 830 instructions).
// One point per thread; a CTA's points come in and its colours go out through shared memory, in
// 16-byte words (V = float4; float where an array is not 16-byte aligned): reading 24-byte points and
// writing 12-byte colours per thread takes three times the memory transactions.
constexpr int kGatherCta = 256;
template <class Store, class V>
__global__ void __launch_bounds__(kGatherCta)
gather_kernel(const typename Store::T* rad, int X, int Y, int Z, const float* pts, int n, float* out) {
    __shared__ __align__(16) float s_buf[6 * kGatherCta];
    grid_launch_dependents();
    grid_dependency_wait();
    constexpr int kW = sizeof(V) / sizeof(float);
    const int first = blockIdx.x * kGatherCta, here = min(kGatherCta, n - first);
    const float* in = pts + 6 * (size_t)first;
    for (int i = threadIdx.x; i < 6 * here / kW; i += kGatherCta)
        reinterpret_cast<V*>(s_buf)[i] = __ldcs(reinterpret_cast<const V*>(in) + i);
    for (int i = 6 * here / kW * kW + (int)threadIdx.x; i < 6 * here; i += kGatherCta) s_buf[i] = in[i];
    __syncthreads();
    float3 c = make_float3(0.0f, 0.0f, 0.0f);
    if ((int)threadIdx.x < here) {
        const float2* q = reinterpret_cast<const float2*>(s_buf) + 3 * threadIdx.x;
        const float2 a = q[0], b = q[1], d = q[2];
        c = gather_point<Store>(rad, X, Y, Z, a.x, a.y, b.x, b.y, d.x, d.y);
    }
    __syncthreads();
    s_buf[3 * threadIdx.x] = c.x;
    s_buf[3 * threadIdx.x + 1] = c.y;
    s_buf[3 * threadIdx.x + 2] = c.z;
    __syncthreads();
    float* o = out + 3 * (size_t)first;
    for (int i = threadIdx.x; i < 3 * here / kW; i += kGatherCta) __stcs(reinterpret_cast<V*>(o) + i, reinterpret_cast<const V*>(s_buf)[i]);
    for (int i = 3 * here / kW * kW + (int)threadIdx.x; i < 3 * here; i += kGatherCta) o[i] = s_buf[i];
}

// exec_copies' block copies (internal_render.cpp:1446-1451): palette slot dst = slot src, one CTA
// of 256 threads x 16 bytes per copy.
__global__ void __launch_bounds__(256) palette_copy_kernel(uint8_t* __restrict__ pal, const int2* __restrict__ copies) {
    const int2 c = copies[blockIdx.x];
    const uint4* src = reinterpret_cast<const uint4*>(pal + (size_t)c.x * 4096);
    uint4* dst = reinterpret_cast<uint4*>(pal + (size_t)c.y * 4096);
    dst[threadIdx.x] = src[threadIdx.x];
}

// map.comp:33-67 for one mesh.  Invocation g covers world voxel g + 0.5 + shift; the model voxel is
// inverse_trans * (world_voxel, 1) truncated; a non-zero model voxel goes to the temporary block
// (id >= static_blocks) that holds the world voxel.  Truncation sends world voxels in (-1, 1) to
// coordinate 0 and those in [-15, -1] onto block 0's far side, so several invocations can target
// one palette voxel (the reference races there).  Writes are resolved as if the invocations ran
// one after another in linear order (x fastest) and the meshes in order: each invocation
// atomicMax-es (mesh, invocation, value) into the target's 64-bit owner word; a resolve pass
// writes the winning values.
//
// One launch covers up to kMapMeshes meshes (a frame's eight took eight launches of about 3.7 us, most
// of it latency): group g of mesh k is CTA group0[k] + g, its 4x4x4 invocations the CTA's threads.
constexpr int kMapMeshes = 24;
struct MapBatch {
    MapMesh mesh[kMapMeshes];
    unsigned group0[kMapMeshes + 1];
    int n, first;
};
static_assert(sizeof(MapBatch) <= 3584, "kernel parameters");
__global__ void __launch_bounds__(64)
map_kernel(const int16_t* __restrict__ grid, int X, int Y, int Z, int n_slots, int static_blocks,
           const __grid_constant__ MapBatch batch, unsigned long long* __restrict__ owner) {
    int k = 0;
    while (blockIdx.x >= batch.group0[k + 1]) k++;
    const MapArgs& a = batch.mesh[k].a;
    const unsigned gw = (unsigned)a.dims[0] / 4u, gh = (unsigned)a.dims[1] / 4u;
    const unsigned group = blockIdx.x - batch.group0[k], gq = group / gw;
    const int gx = (int)(4u * (group - gq * gw) + (threadIdx.x & 3u));
    const int gy = (int)(4u * (gq % gh) + ((threadIdx.x >> 2) & 3u));
    const int gz = (int)(4u * (gq / gh) + (threadIdx.x >> 4));
    const int mx = batch.mesh[k].size[0], my = batch.mesh[k].size[1], mz = batch.mesh[k].size[2];
    // world_voxel = vec3(g) / 1.0 + vec3(0.5) + vec3(shift)   (:37-40)
    const float wx = fadd(fadd((float)gx, 0.5f), (float)a.shift[0]);
    const float wy = fadd(fadd((float)gy, 0.5f), (float)a.shift[1]);
    const float wz = fadd(fadd((float)gz, 0.5f), (float)a.shift[2]);
    const int ix = f2i(wx), iy = f2i(wy), iz = f2i(wz);   // (:41)
    // target block = iworld / 16 (OpSDiv); out of range reads block 0   (:50-52)
    const int bx = ix / 16, by = iy / 16, bz = iz / 16;
    int id = 0;
    if (bx >= 0 && by >= 0 && bz >= 0 && bx < X && by < Y && bz < Z)
        id = grid[(size_t)bx + (size_t)X * ((size_t)by + (size_t)Y * bz)];
    if (id < static_blocks || id >= n_slots) return;   // (:59); the palette ends at its last slot
    // model_voxel = (inverse_trans * vec4(world_voxel, 1)).xyz, columns summed in order   (:47-48)
    const float* m = a.inv;   // column-major m[4*col + row]
    const float vx = fadd(fadd(fadd(fmul(m[0], wx), fmul(m[4], wy)), fmul(m[8], wz)), m[12]);
    const float vy = fadd(fadd(fadd(fmul(m[1], wx), fmul(m[5], wy)), fmul(m[9], wz)), m[13]);
    const float vz = fadd(fadd(fadd(fmul(m[2], wx), fmul(m[6], wy)), fmul(m[10], wz)), m[14]);
    const int px = f2i(vx), py = f2i(vy), pz = f2i(vz);
    int v = 0;
    if (px >= 0 && py >= 0 && pz >= 0 && px < mx && py < my && pz < mz)
        v = batch.mesh[k].voxels[(size_t)px + (size_t)mx * ((size_t)py + (size_t)my * pz)];   // (:60)
    if (v == 0) return;
    const unsigned long long lin =
        (unsigned long long)gx + (unsigned long long)a.dims[0] * ((unsigned long long)gy + (unsigned long long)a.dims[1] * gz);
    const size_t t = ((size_t)(id - static_blocks) << 12) | (smod(iz, 16) << 8) | (smod(iy, 16) << 4) | smod(ix, 16);
    const unsigned long long mesh_key = (unsigned long long)(batch.first + k + 1) << 40;
    atomicMax(owner + t, mesh_key | (lin << 8) | (unsigned long long)v);   // (:54,62)
}

// Changed blocks of a context's world into its grid and compact grid (a block listed twice has the same
// value both times).
__global__ void apply_cells_kernel(const CellEdit* __restrict__ edits, int n, int16_t* __restrict__ grid, void* cgrid, int wide,
                                   int X, int Y) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const CellEdit e = edits[k];
    const unsigned q = e.index / (unsigned)X;
    const size_t cell = (e.index - q * (unsigned)X) + (size_t)(X + 1) * (q % (unsigned)Y + (size_t)(Y + 1) * (q / (unsigned)Y));
    grid[e.index] = e.block;
    if (wide) static_cast<uint16_t*>(cgrid)[cell] = e.compact;
    else static_cast<uint8_t*>(cgrid)[cell] = (uint8_t)e.compact;
}

__global__ void map_resolve_kernel(uint8_t* __restrict__ pal_tmp, const unsigned long long* __restrict__ owner,
                                   size_t n) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const unsigned long long o = owner[i];
        if (o) pal_tmp[i] = (uint8_t)(o & 0xffu);
    }
}

// Occupancy masks of compact ids from the device palette: CTA c, thread w -> word w of id c.
__global__ void __launch_bounds__(128) compact_bits_kernel(const uint8_t* __restrict__ pal, const int* __restrict__ slot_of,
                                                           uint32_t* __restrict__ cbits) {
    const int c = blockIdx.x, w = threadIdx.x;
    const int slot = slot_of[c];
    uint32_t bits = 0;
    if (slot >= 0) {
        const uint4* p = reinterpret_cast<const uint4*>(pal + (size_t)slot * 4096 + 32 * w);
        const uint4 a = p[0], b = p[1];
        const uint32_t words[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int k = 0; k < 32; k++)
            if ((words[k >> 2] >> (8 * (k & 3))) & 0xffu) bits |= 1u << k;
    }
    cbits[(size_t)c * 128 + w] = bits;
}

// A radiance volume as packed RGB floats (the storage type decoded exactly), and the error word,
// written straight into page-locked host memory (`out` and `err_out` are its device addresses): one
// launch instead of a launch and two copies.  Through shared memory, so that the writes leave in
// 16-byte words side by side (V = float4; float if `out` is not 16-byte aligned).  Bound by the launch
// and the wait for it: the read-back of 8x8x8 / 64x64x16 / 256x256x64 blocks 15.8 / 21.2 / 292 -> 11.9 /
// 15.5 / 272 us (185 GB/s).
constexpr int kPackCta = 256;
template <class Store, class V>
__global__ void __launch_bounds__(kPackCta)
pack_rgb_kernel(const typename Store::T* rad, float* out, long long W, const int* err, int* err_out) {
    __shared__ __align__(16) float s_buf[3 * kPackCta];
    constexpr int kW = sizeof(V) / sizeof(float);
    grid_dependency_wait();
    for (long long first = (long long)blockIdx.x * kPackCta; first < W; first += (long long)gridDim.x * kPackCta) {
        const int here = (int)min((long long)kPackCta, W - first);
        if ((int)threadIdx.x < here) {
            const float3 v = Store::load(rad, (int)(first + threadIdx.x));
            s_buf[3 * threadIdx.x] = v.x;
            s_buf[3 * threadIdx.x + 1] = v.y;
            s_buf[3 * threadIdx.x + 2] = v.z;
        }
        __syncthreads();
        float* o = out + 3 * first;
        for (int i = threadIdx.x; i < 3 * here / kW; i += kPackCta) reinterpret_cast<V*>(o)[i] = reinterpret_cast<const V*>(s_buf)[i];
        for (int i = 3 * here / kW * kW + (int)threadIdx.x; i < 3 * here; i += kPackCta) o[i] = s_buf[i];
        __syncthreads();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *err_out = *err;
}

}  // namespace

template <class Store>
static cudaError_t launch_pack_t(const void* rad, long long W, float* out, const int* err, int* err_out, cudaStream_t stream) {
    const int blocks = (int)std::min<long long>((W + kPackCta - 1) / kPackCta, 152LL * 8);
    const typename Store::T* r = static_cast<const typename Store::T*>(rad);
    if ((reinterpret_cast<uintptr_t>(out) & 15) == 0)
        return launch_kernel(pack_rgb_kernel<Store, float4>, blocks, kPackCta, 0, stream, true, r, out, W, err, err_out);
    return launch_kernel(pack_rgb_kernel<Store, float>, blocks, kPackCta, 0, stream, true, r, out, W, err, err_out);
}

cudaError_t launch_pack_rgb(const void* rad, int precision, long long W, float* out, const int* err, int* err_out,
                            cudaStream_t stream) {
    switch (precision) {
        case LUMRAD_PRECISION_FP16: return launch_pack_t<StoreF16>(rad, W, out, err, err_out, stream);
        case LUMRAD_PRECISION_BF16: return launch_pack_t<StoreBF16>(rad, W, out, err, err_out, stream);
        case LUMRAD_PRECISION_RGB10A2: return launch_pack_t<StoreRGB10A2>(rad, W, out, err, err_out, stream);
        default: return launch_pack_t<StoreF32>(rad, W, out, err, err_out, stream);
    }
}

cudaError_t launch_palette_copies(uint8_t* pal, const int2* copies, int n, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    palette_copy_kernel<<<n, 256, 0, stream>>>(pal, copies);
    return cudaGetLastError();
}

cudaError_t launch_map(const int16_t* grid, int X, int Y, int Z, int n_slots, int static_blocks, const MapMesh* meshes,
                       int n, int first, unsigned long long* owner, cudaStream_t stream) {
    for (int i = 0; i < n;) {   // as many meshes as fit a launch (2^31 groups, kMapMeshes)
        MapBatch batch;
        batch.n = 0;
        batch.first = first + i;
        batch.group0[0] = 0;
        unsigned long long groups = 0;
        for (; i < n && batch.n < kMapMeshes; i++) {
            const int* d = meshes[i].a.dims;
            const bool empty = d[0] <= 0 || d[1] <= 0 || d[2] <= 0;
            const unsigned long long g = empty ? 0 : (unsigned long long)(d[0] / 4) * (d[1] / 4) * (d[2] / 4);   // local_size 4x4x4 (:32)
            if (groups + g >= 1ull << 31) break;
            groups += g;
            batch.mesh[batch.n] = meshes[i];
            batch.group0[++batch.n] = (unsigned)groups;
        }
        if (batch.n == 0) return cudaErrorInvalidValue;   // (a mesh covers fewer than 2^32 voxels)
        if (groups > 0) map_kernel<<<(unsigned)groups, 64, 0, stream>>>(grid, X, Y, Z, n_slots, static_blocks, batch, owner);
    }
    return cudaGetLastError();
}

cudaError_t launch_apply_cells(const CellEdit* edits, int n, int16_t* grid, void* cgrid, bool wide, int X, int Y,
                               cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    apply_cells_kernel<<<(n + 127) / 128, 128, 0, stream>>>(edits, n, grid, cgrid, wide ? 1 : 0, X, Y);
    return cudaGetLastError();
}

cudaError_t launch_map_resolve(uint8_t* pal_tmp, const unsigned long long* owner, size_t n, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    const int blocks = (int)std::min<size_t>((n + 255) / 256, 152 * 16);
    map_resolve_kernel<<<blocks, 256, 0, stream>>>(pal_tmp, owner, n);
    return cudaGetLastError();
}

cudaError_t launch_compact_bits(const uint8_t* pal, const int* slot_of, int n_compact, uint32_t* cbits,
                                cudaStream_t stream) {
    if (n_compact <= 0) return cudaSuccess;
    compact_bits_kernel<<<n_compact, 128, 0, stream>>>(pal, slot_of, cbits);
    return cudaGetLastError();
}

cudaError_t launch_update_list(const int16_t* grid, int X, int Y, int Z, const short4* specials, int n_specials,
                               const ListScratch& s, short4* out, int* count, bool dependent, cudaStream_t stream) {
    const long long W = (long long)X * Y * Z;
    const int ctas = (int)((W + kListCta - 1) / kListCta);
    cudaError_t e = launch_kernel(list_flags_kernel, ctas, kListCta, 0, stream, dependent, grid, X, Y, Z, (unsigned)W, s.bits, s.cta_counts);
    if (e != cudaSuccess) return e;
    if ((e = launch_list_write(s, X, Y, W, out, count, n_specials > 0 ? s.listed : nullptr, stream)) != cudaSuccess) return e;
    if (n_specials > 0) list_specials_kernel<<<1, kScanCta, 0, stream>>>(specials, n_specials, s.bits, X, Y, s.listed, out, count);
    return cudaGetLastError();
}

cudaError_t launch_dirty_list(const short4* edits, int n_edits, int X, int Y, int Z, int radius, uint8_t* mask_a,
                              uint8_t* mask_b, const ListScratch& s, short4* out, int* count, cudaStream_t stream) {
    const long long W = (long long)X * Y * Z;
    const int ctas = (int)((W + kListCta - 1) / kListCta);
    const int blocks = (int)std::min<long long>((W + 255) / 256, 152LL * 16);
    cudaError_t e = cudaMemsetAsync(mask_a, 0, (size_t)W, stream);
    if (e != cudaSuccess) return e;
    if (n_edits > 0) dirty_mark_kernel<<<(n_edits + 255) / 256, 256, 0, stream>>>(edits, n_edits, X, Y, mask_a);
    dirty_dilate_kernel<<<blocks, 256, 0, stream>>>(mask_a, mask_b, X, Y, Z, 0, radius, W);
    dirty_dilate_kernel<<<blocks, 256, 0, stream>>>(mask_b, mask_a, X, Y, Z, 1, radius, W);
    dirty_flags_kernel<<<ctas, kListCta, 0, stream>>>(mask_a, X, Y, Z, radius, W, s.bits, s.cta_counts);
    return launch_list_write(s, X, Y, W, out, count, nullptr, stream);
}

static long long dirty_rows(int n_edits, int Y, int Z, int radius) {
    return (long long)n_edits * std::min(2 * radius + 1, Y) * std::min(2 * radius + 1, Z);
}

// The line between the rows of bits and the dilation, from calls of both (rows / dilation): the kernel reads the
// edits from the host's memory (200,000 of them, radius 0, 16x16x8 blocks: 410 / 330 us, 4,096: 25 / 61), rows
// close together wait for each other's words (8x8x8, 500,000 rows 115 / 85, 128,000 rows 29 / 55; 64x64x16,
// 992,000 rows 69 / 78), and the list goes to the host's memory block by block (64x64x64, a list of
// up to 262,144: 162 / 74, of 41,000: 40 / 89).  Neither form is slower than the dilation alone was.
bool dirty_rows_fit(int X, int Y, int Z, int n_edits, int radius) {
    const long long W = (long long)X * Y * Z, rows = dirty_rows(n_edits, Y, Z, radius);
    return list_scratch_ctas(W) <= kBitsCtas && n_edits <= 4096 && rows <= std::min(std::max(32 * W, 1LL << 17), 1LL << 20) &&
           std::min(W, rows * std::min(2 * radius + 1, X)) <= 1LL << 16;
}

cudaError_t launch_dirty_rows(const short4* edits, int n_edits, int X, int Y, int Z, int radius, uint32_t* bits, short4* out,
                              int* count, cudaStream_t stream) {
    const long long W = (long long)X * Y * Z;
    const long long rows = dirty_rows(n_edits, Y, Z, radius);
    cudaError_t e = cudaMemsetAsync(bits, 0, list_scratch_words(W) * sizeof(uint32_t), stream);
    if (e != cudaSuccess) return e;
    if (rows > 0) dirty_rows_kernel<<<(int)((rows + 255) / 256), 256, 0, stream>>>(edits, (int)rows, X, Y, Z, radius, bits);
    return launch_kernel(list_write_kernel, (int)list_scratch_ctas(W), kListCta, 0, stream, true, bits, nullptr, nullptr, X, Y,
                         (unsigned)W, out, count, nullptr);
}

// (whole CTAs' words: the list's writer reads its own and those before them)
size_t list_scratch_words(long long W) { return (size_t)((W + kListCta - 1) / kListCta) * (kListCta / 32); }
size_t list_scratch_ctas(long long W) { return (size_t)((W + kListCta - 1) / kListCta); }

cudaError_t launch_shift_radiance(const void* src, void* dst, int X, int Y, int Z, int sx, int sy, int sz,
                                  int precision, cudaStream_t stream) {
    const long long W = (long long)X * Y * Z;
    const int blocks = (int)std::min<long long>((W + 255) / 256, 152LL * 16);
    if (precision == LUMRAD_PRECISION_FP32)
        return launch_kernel(shift_kernel<uint4>, blocks, 256, 0, stream, true, static_cast<const uint4*>(src),
                             static_cast<uint4*>(dst), X, Y, Z, sx, sy, sz, W);
    if (precision == LUMRAD_PRECISION_RGB10A2)
        return launch_kernel(shift_kernel<unsigned>, blocks, 256, 0, stream, true, static_cast<const unsigned*>(src),
                             static_cast<unsigned*>(dst), X, Y, Z, sx, sy, sz, W);
    return launch_kernel(shift_kernel<uint2>, blocks, 256, 0, stream, true, static_cast<const uint2*>(src),
                         static_cast<uint2*>(dst), X, Y, Z, sx, sy, sz, W);
}

template <class Store>
static cudaError_t launch_gather_t(const void* rad, int X, int Y, int Z, const float* pts, int n, float* out, cudaStream_t stream) {
    const int blocks = (n + kGatherCta - 1) / kGatherCta;
    const typename Store::T* r = static_cast<const typename Store::T*>(rad);
    if (((reinterpret_cast<uintptr_t>(pts) | reinterpret_cast<uintptr_t>(out)) & 15) == 0)
        return launch_kernel(gather_kernel<Store, float4>, blocks, kGatherCta, 0, stream, true, r, X, Y, Z, pts, n, out);
    return launch_kernel(gather_kernel<Store, float>, blocks, kGatherCta, 0, stream, true, r, X, Y, Z, pts, n, out);
}

cudaError_t launch_gather(const void* rad, int X, int Y, int Z, int precision, const float* pts, int n, float* out,
                          cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    switch (precision) {
        case LUMRAD_PRECISION_FP16: return launch_gather_t<StoreF16>(rad, X, Y, Z, pts, n, out, stream);
        case LUMRAD_PRECISION_BF16: return launch_gather_t<StoreBF16>(rad, X, Y, Z, pts, n, out, stream);
        case LUMRAD_PRECISION_RGB10A2: return launch_gather_t<StoreRGB10A2>(rad, X, Y, Z, pts, n, out, stream);
        default: return launch_gather_t<StoreF32>(rad, X, Y, Z, pts, n, out, stream);
    }
}

}  // namespace lumrad
