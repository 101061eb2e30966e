// ConfidenceEvaluation (main.cpp:959-1109) and RunFusion / RunFusion_Sky_Strict
// (main.cpp:659-957) on the GPU with the reference's sequential semantics.
//
// The reference scans views in order and each view's pixels in raster order.
// A pixel is accepted when enough source views agree; accepting it marks the
// source pixels in `used_list` as used, and `used_list` keeps the last passing
// position of every source across pixels (it is declared per view, not per
// pixel), so stale positions are re-marked.  Later pixels skip marked source
// pixels.  The result depends on that order.
//
// Parallel form used here, per view i (views stay sequential):
//   1. candidates (parallel over pixels q and sources j): the source pixel
//      P[q][j] and whether the geometric test passes, T[q][j], ignoring the
//      marks that view i itself sets;
//   2. a causal fixed point: eff[q][j] = T[q][j] and P[q][j] not marked before q.
//      Each Jacobi round computes acceptance from eff, the first pixel that
//      marks each source pixel (atomicMin), and eff again.  eff[q] depends only
//      on pixels before q, so the system has one solution and a round that
//      changes nothing has reached it; rounds are capped and a sequential
//      pass takes over beyond the cap;
//   3. marks become permanent, confidences take the value of the last pixel
//      that marked them (atomicMax), points are compacted in raster order.
//
// Entry (q, j), an eff bit, is source j's used position from q until the next
// pixel with bit j.  It is marked by the accepted pixels of that interval, the
// first of them counts for the rounds and the last for the confidence.  A
// counted pixel is nearly always accepted itself, so the first is q; the other
// ends are looked up in bitmaps (one per source, one of accepted pixels), 32
// pixels at a time, and 1024 at a time where a summary word shows nothing set.
// (Prefix maxima of the last counted pixel for every pixel and source, ten
// words a pixel written and read again in every round, took two thirds of a
// scan: 11 views of 1600x1200 with 10 sources took 33.9 ms and take 11.4.  A
// further summary level of 32 chunks changed nothing.)
// Marks carry the round that set them, so no round clears them.
//
// Rounds are launched as many as the previous view needed; each kernel returns
// at once when the round before it changed nothing, so the host reads the change
// flags once a view instead of once a round.
//
// Arithmetic mirrors the host code of the reference (g++ without -ffast-math):
// float geometry, double where pow(float, int) promotes; exp(float) is the
// float function there (the double exp rounded to float here).  No implicit
// contraction.
#include "aux_kernels.cuh"
#include "ctx.hpp"

#include <algorithm>
#include <climits>
#include <vector>

namespace hpm {

constexpr int kScanBlock = 1024;  // pixels of a chunk: one word of summary bits
constexpr uint32_t kAccepted = 1u << 31;  // in a pixel's word beside the eff bits of at most 31 sources

// One source of the view being scanned.  slot: the mark buffers it uses (a source listed twice shares them).
struct ScanSource {
    hpm_camera cam;  // scaled to W x H
    float centre[3];
    int W, H, slot;
    const float* depth;
    const float* normal;
    uint8_t* mask;   // used pixels, persistent across the views of one scan
    float* cons;     // working confidence (confidence mode)
};

// One view of a scan against its sources; a kernel parameter.
struct ScanRun {
    hpm_camera cam;
    float centre[3];
    int W, H, npix, n;
    bool distinct;          // no source is listed twice: slot j for source j
    int stride;             // pixels rounded up to whole chunks: stride of the per-source arrays
    const float* depth;
    const float* normal;
    const uint8_t* color;   // BGR (fusion)
    const uint8_t* sky;     // BGR sky mask or null
    uint8_t* mask;
    float* cons;
    int32_t* pos;           // [j * stride + q] source pixel of a passing pair
    float* wexp;            // [j * stride + q] its weight
    uint32_t* test;         // T bits
    uint32_t* word;         // eff bits, kAccepted
    uint32_t* chunk;        // OR of a chunk's words
    uint32_t* map;          // [j * stride / 32 + q / 32] bit q % 32: eff bit j; j = n: accepted
    float* dyn;             // sum of the counted weights
    unsigned long long* first_mark;  // [slot * mark_stride + p]  (~round << 32) | first marking pixel
    unsigned long long* last_mark;   // [slot * mark_stride + p]  (view << 32) | last marking pixel
    size_t mark_stride;
    ScanSource src[31];
};
static_assert(sizeof(ScanRun) <= 32764, "ScanRun exceeds the kernel parameter limit");

// Camera centre, in the reference's float arithmetic (Get3DPointonWorld's C; the same on the host).
static void camera_centre(const hpm_camera& c, float C[3]) {
    for (int k = 0; k < 3; ++k) C[k] = -(c.R[k] * c.t[0] + c.R[3 + k] * c.t[1] + c.R[6 + k] * c.t[2]);
}

__device__ __forceinline__ float3 sc_world_point(int x, int y, float depth, const hpm_camera& c, const float* C) {
    const float X0 = depth * (x - c.K[2]) / c.K[0];
    const float X1 = depth * (y - c.K[5]) / c.K[4];
    const float X2 = depth;
    const float T0 = c.R[0] * X0 + c.R[3] * X1 + c.R[6] * X2;
    const float T1 = c.R[1] * X0 + c.R[4] * X1 + c.R[7] * X2;
    const float T2 = c.R[2] * X0 + c.R[5] * X1 + c.R[8] * X2;
    return make_float3(T0 + C[0], T1 + C[1], T2 + C[2]);
}

__device__ __forceinline__ float2 sc_project(float3 X, const hpm_camera& c, float& depth) {
    const float T0 = c.R[0] * X.x + c.R[1] * X.y + c.R[2] * X.z + c.t[0];
    const float T1 = c.R[3] * X.x + c.R[4] * X.y + c.R[5] * X.z + c.t[1];
    const float T2 = c.R[6] * X.x + c.R[7] * X.y + c.R[8] * X.z + c.t[2];
    depth = c.K[6] * T0 + c.K[7] * T1 + c.K[8] * T2;
    return make_float2((c.K[0] * T0 + c.K[1] * T1 + c.K[2] * T2) / depth,
                       (c.K[3] * T0 + c.K[4] * T1 + c.K[5] * T2) / depth);
}

// int(v) of the x86 host: truncation, NaN and out-of-range give INT_MIN.
__device__ __forceinline__ int host_trunc(float v) {
    if (!(v > -2147483648.0f && v < 2147483648.0f)) return INT_MIN;
    return __float2int_rz(v);
}

__device__ __forceinline__ float host_angle(const float* a, const float* b) {  // HPM.cpp:281-290
    const float dot = a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
    const float ang = (float)acos((double)dot);
    return ang != ang ? 0.0f : ang;
}

template <int MODE>
__global__ void __launch_bounds__(256) k_candidates(const __grid_constant__ ScanRun a) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= a.npix) return;
    const int r = q / a.W, c = q - r * a.W;
    uint32_t T = 0;
    const float ref_depth = a.depth[q];
    bool valid = a.mask[q] != 1 && ref_depth > 0.0f;
    if (MODE == 0 && valid && (ref_depth < a.cam.depth_min || ref_depth > a.cam.depth_max)) valid = false;
    if (valid) {
        const float3 X = sc_world_point(c, r, ref_depth, a.cam, a.centre);
        const float rn[3] = { a.normal[3 * (size_t)q], a.normal[3 * (size_t)q + 1], a.normal[3 * (size_t)q + 2] };
#pragma unroll 1
        for (int j = 0; j < a.n; ++j) {
            const ScanSource& vs = a.src[j];
            float pd;
            const float2 pt = sc_project(X, vs.cam, pd);
            const int sr = host_trunc(pt.y + 0.5f);
            const int scc = host_trunc(pt.x + 0.5f);
            if (!(scc >= 0 && scc < vs.W && sr >= 0 && sr < vs.H)) continue;
            const int p = sr * vs.W + scc;
            const float sd = vs.depth[p];
            if (!(sd > 0.0f)) continue;
            if (MODE == 0 && (sd < a.cam.depth_min || sd > a.cam.depth_max)) continue;
            const float3 tX = sc_world_point(scc, sr, sd, vs.cam, vs.centre);
            float proj;
            const float2 tp = sc_project(tX, a.cam, proj);
            const double dx = (double)(c - tp.x), dy = (double)(r - tp.y);
            const float reproj = (float)sqrt(dx * dx + dy * dy);
            const float rel = (float)(fabs((double)(proj - ref_depth)) / (double)ref_depth);
            if (!(reproj < 2.0f && rel < 0.01f)) continue;  // most misses end before the normals and the arc cosine
            const float ang = host_angle(rn, vs.normal + 3 * (size_t)p);
            if (!(ang < 0.174533f) || vs.mask[p] == 1) continue;
            const float idx = reproj + 200 * rel + ang * 10;
            T |= 1u << j;
            // exp(float) of the reference's host code: the float function
            a.wexp[(size_t)j * a.stride + q] = (float)exp((double)(-idx));
            a.pos[(size_t)j * a.stride + q] = p;
        }
    }
    a.test[q] = T;
    a.word[q] = T;
}

// The set bits of a word, kBatch at a time: a batch's gathers are in flight together (one bit after the
// other, k_update_eff spent its time waiting for two dependent gathers a bit).
constexpr int kBatch = 4;
struct Batch {
    int j[kBatch];  // -1 past the last
    __device__ __forceinline__ explicit Batch(uint32_t& bits) {
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            j[k] = __ffs(bits) - 1;
            bits &= bits - 1;
        }
    }
};

// Where source j's marks start.  (The lanes of a warp ask for different sources, which the constant
// memory of the parameters would serve one after the other.)
__device__ __forceinline__ size_t marks_of(const ScanRun& a, int j) {
    return (a.distinct ? j : a.src[j].slot) * a.mark_stride;
}

// A round's kernels run when the round before changed something.
__device__ __forceinline__ bool settled(const int* before) { return before && *before == 0; }

// Acceptance from the eff bits, the chunks' summaries, and the marks of accepted pixels on the
// positions they counted.  One block per chunk; pixels past the last have empty words.
__global__ void __launch_bounds__(kScanBlock) k_accept(const __grid_constant__ ScanRun a, const int* before,
                                                       uint32_t round) {
    __shared__ uint32_t ws[32];
    if (settled(before)) return;
    const int q = blockIdx.x * kScanBlock + threadIdx.x;
    uint32_t w = 0;
    if (q < a.npix) {
        const uint32_t e = a.word[q] & ~kAccepted;
        w = e;
        float d = 0.0f;
        for (uint32_t m = e; m;) {
            const Batch b(m);
            float x[kBatch];
#pragma unroll
            for (int k = 0; k < kBatch; ++k) x[k] = b.j[k] >= 0 ? a.wexp[(size_t)b.j[k] * a.stride + q] : 0.0f;
#pragma unroll
            for (int k = 0; k < kBatch; ++k)
                if (b.j[k] >= 0) d = (float)((double)d + (double)x[k]);
        }
        const int n = __popc(e);
        a.dyn[q] = d;
        if (n >= 1 && (double)d > 0.3 * n) {
            w |= kAccepted;
            const unsigned long long mark = (unsigned long long)~round << 32 | (uint32_t)q;
            for (uint32_t m = e; m;) {
                const Batch b(m);
                int p[kBatch];
#pragma unroll
                for (int k = 0; k < kBatch; ++k) p[k] = b.j[k] >= 0 ? a.pos[(size_t)b.j[k] * a.stride + q] : 0;
#pragma unroll
                for (int k = 0; k < kBatch; ++k)
                    if (b.j[k] >= 0) atomicMin(a.first_mark + marks_of(a, b.j[k]) + p[k], mark);
            }
        }
    }
    a.word[q] = w;
    const int lane = threadIdx.x & 31, words = a.stride / 32;
    const uint32_t any = __reduce_or_sync(0xffffffffu, w);
    for (int j = 0; j <= a.n; ++j) {
        const uint32_t b = __ballot_sync(0xffffffffu, w & (j < a.n ? 1u << j : kAccepted));
        if (lane == 0) a.map[(size_t)j * words + (q >> 5)] = b;
    }
    if (lane == 0) ws[threadIdx.x >> 5] = any;
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint32_t all = __reduce_or_sync(0xffffffffu, ws[threadIdx.x]);
        if (threadIdx.x == 0) a.chunk[blockIdx.x] = all;
    }
}

// The first chunk from `c` on whose summary has a bit of `m`, or one past the last.
__device__ __forceinline__ int next_chunk(const ScanRun& a, int c, uint32_t m) {
    const int chunks = a.stride / kScanBlock;
    for (; c < chunks; c += 4) {  // four loads in flight
        uint32_t v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = c + k < chunks ? a.chunk[c + k] & m : 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (v[k]) return c + k;
    }
    return chunks;
}

// The first pixel from `q` on with eff bit j (or accepted, when ALSO_ACCEPTED), or stride.
template <bool ALSO_ACCEPTED>
__device__ __forceinline__ int next_pixel(const ScanRun& a, int q, int j) {
    if (q >= a.stride) return a.stride;
    const int words = a.stride / 32;
    const uint32_t* eff = a.map + (size_t)j * words;
    const uint32_t* acc = a.map + (size_t)a.n * words;
    auto bits = [&](int w) { return ALSO_ACCEPTED ? eff[w] | acc[w] : eff[w]; };
    int w = q >> 5;
    uint32_t b = bits(w) & (0xffffffffu << (q & 31));
    while (!b && (++w & 31)) b = bits(w);  // to the end of the chunk: 32 words
    if (!b) {
        const int c = next_chunk(a, w >> 5, ALSO_ACCEPTED ? 1u << j | kAccepted : 1u << j);
        if (c * kScanBlock >= a.stride) return a.stride;
        w = c * 32;
        const int end = w + 32;
        for (b = bits(w); !b && w + 1 < end;) b = bits(++w);
        if (!b) return a.stride;
    }
    return w * 32 + __ffs(b) - 1;
}

// The last accepted pixel in [lo, hi], or -1.
__device__ __forceinline__ int last_accepted(const ScanRun& a, int lo, int hi) {
    const uint32_t* acc = a.map + (size_t)a.n * (a.stride / 32);
    int w = hi >> 5;
    const int w_lo = lo >> 5;
    uint32_t b = acc[w] & (0xffffffffu >> (31 - (hi & 31)));
    while (!b && w > w_lo) {
        if (!(w & 31)) {  // the chunk below: skip those without an accepted pixel
            int c = (w >> 5) - 1;
            while (c > (w_lo >> 5) && !(a.chunk[c] & kAccepted)) --c;
            w = c * 32 + 32;
        }
        b = acc[--w];
    }
    if (!b) return -1;
    const int q = w * 32 + 31 - __clz(b);
    return q >= lo ? q : -1;
}

// Pixels walked one by one, all sources of a pixel together, before the bitmaps are searched source by
// source: most intervals end within a few pixels.
constexpr int kWalk = 16;

// Marks of counted but not accepted pixels: by the next accepted pixel, unless a pixel up to it counts
// the source again.
__global__ void __launch_bounds__(256) k_mark_stale(const __grid_constant__ ScanRun a, const int* before,
                                                    uint32_t round) {
    if (settled(before)) return;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= a.npix) return;
    uint32_t m = a.word[q];
    if (m & kAccepted) return;
    const int walk = min(q + kWalk, a.npix - 1);
    int n = q;
    uint32_t w = 0;
    while (m && n < walk && !(w & kAccepted)) {
        w = a.word[++n];
        m &= ~w;  // counted again
    }
    for (; m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        int by = n;
        if (!(w & kAccepted)) {
            by = next_pixel<true>(a, n + 1, j);
            if (by >= a.npix || ((a.word[by] >> j) & 1u)) continue;
        }
        atomicMin(a.first_mark + marks_of(a, j) + a.pos[(size_t)j * a.stride + q],
                  (unsigned long long)~round << 32 | (uint32_t)by);
    }
}

// eff = T minus the pairs whose source pixel is marked before q.
__global__ void __launch_bounds__(256) k_update_eff(const __grid_constant__ ScanRun a, const int* before,
                                                    uint32_t round, int* __restrict__ changed) {
    if (settled(before)) return;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= a.npix) return;
    const uint32_t T = a.test[q];
    uint32_t e = T;
    for (uint32_t m = T; m;) {
        const Batch b(m);
        int p[kBatch];
        unsigned long long v[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) p[k] = b.j[k] >= 0 ? a.pos[(size_t)b.j[k] * a.stride + q] : 0;
#pragma unroll
        for (int k = 0; k < kBatch; ++k)
            v[k] = b.j[k] >= 0 ? a.first_mark[marks_of(a, b.j[k]) + p[k]] : 0ull;
#pragma unroll
        for (int k = 0; k < kBatch; ++k)
            if (b.j[k] >= 0 && (uint32_t)(v[k] >> 32) == ~round && (uint32_t)v[k] < (uint32_t)q) e &= ~(1u << b.j[k]);
    }
    const uint32_t w = a.word[q];
    if (e != (w & ~kAccepted)) {
        a.word[q] = e;  // the next round sets kAccepted
        *changed = 1;
    }
}

// The settled marks: the source pixels of all marked entries become used; with MODE 0 each also
// learns the last accepted pixel of its interval.
template <int MODE>
__global__ void __launch_bounds__(256) k_settle(const __grid_constant__ ScanRun a, uint32_t view) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= a.npix) return;
    const uint32_t own = a.word[q];
    uint32_t m = own & ~kAccepted;
    int last = own & kAccepted ? q : -1, n = q;  // last accepted pixel up to n
    auto settle = [&](uint32_t bits, int by) {  // the sources whose interval's marking pixel is known
        if (by < 0) return;
        for (; bits; bits &= bits - 1) {
            const int j = __ffs(bits) - 1;
            const int p = a.pos[(size_t)j * a.stride + q];
            a.src[j].mask[p] = 1;
            if (MODE == 0)
                atomicMax(a.last_mark + marks_of(a, j) + p, (unsigned long long)view << 32 | (uint32_t)by);
        }
    };
    const int walk = min(q + kWalk, a.npix - 1);
    while (m && n < walk && !(MODE == 1 && last >= 0)) {
        const uint32_t w = a.word[++n];
        settle(m & w, last);  // counted again: the interval ends before n
        m &= ~w;
        if (w & kAccepted) last = n;
    }
    for (; m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        int by = last;
        if (MODE == 0) {
            const int next = min(next_pixel<false>(a, n + 1, j), a.npix);
            if (next > n + 1) by = max(by, last_accepted(a, n + 1, next - 1));
        } else if (by < 0) {
            const int next = next_pixel<true>(a, n + 1, j);
            if (next < a.npix && !((a.word[next] >> j) & 1u)) by = next;
        }
        settle(1u << j, by);
    }
}

// Confidences of the sources' pixels marked in this view: grid row j for source j.
__global__ void __launch_bounds__(256) k_marked_conf(const __grid_constant__ ScanRun a, uint32_t view) {
    const ScanSource& vs = a.src[blockIdx.y];
    const int p = 4 * (blockIdx.x * blockDim.x + threadIdx.x), n = vs.W * vs.H;
    if (p >= n) return;
    // the marks of four pixels in two loads; mark_stride is a multiple of four
    const ulonglong2* marks = reinterpret_cast<const ulonglong2*>(a.last_mark + vs.slot * a.mark_stride + p);
    const ulonglong2 lo = marks[0], hi = marks[1];
    const unsigned long long v[4] = { lo.x, lo.y, hi.x, hi.y };
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (p + k < n && (uint32_t)(v[k] >> 32) == view) vs.cons[p + k] = a.dyn[(uint32_t)v[k]];
}

__global__ void __launch_bounds__(256) k_conf_own(const __grid_constant__ ScanRun a, float* __restrict__ out) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= a.npix) return;
    float v = a.cons[q];
    if (a.word[q] & kAccepted) {
        v = a.dyn[q];
        a.cons[q] = v;
    }
    out[q] = v;  // confidence.dmb of view i is written after its own scan (main.cpp:1091-1095)
}

// Exact sequential pass (the reference loop) over the precomputed candidates;
// used when the fixed point has not settled within Ctx::scan_rounds.
__global__ void k_sequential(const __grid_constant__ ScanRun a, uint32_t round) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    int used[31];
    for (int j = 0; j < a.n; ++j) used[j] = -1;
    for (int c = 0; c < a.stride / kScanBlock; ++c) a.chunk[c] = 0;
    for (int w = 0; w < (a.n + 1) * (a.stride / 32); ++w) a.map[w] = 0;
    for (int q = 0; q < a.npix; ++q) {
        const uint32_t T = a.test[q];
        uint32_t e = 0;
        float d = 0.0f;
        for (int j = 0; j < a.n; ++j) {
            if (!((T >> j) & 1u)) continue;
            const int p = a.pos[(size_t)j * a.stride + q];
            if ((uint32_t)(a.first_mark[a.src[j].slot * a.mark_stride + p] >> 32) == ~round) continue;
            used[j] = p;
            d = (float)((double)d + (double)a.wexp[(size_t)j * a.stride + q]);
            e |= 1u << j;
        }
        const int n = __popc(e);
        const bool ok = n >= 1 && (double)d > 0.3 * n;
        a.dyn[q] = d;
        a.word[q] = ok ? e | kAccepted : e;
        a.chunk[q / kScanBlock] |= a.word[q];
        for (int j = 0; j <= a.n; ++j)
            if (j < a.n ? (e >> j) & 1u : (uint32_t)ok) a.map[(size_t)j * (a.stride / 32) + (q >> 5)] |= 1u << (q & 31);
        if (ok)
            for (int j = 0; j < a.n; ++j)
                if (used[j] >= 0)
                    a.first_mark[a.src[j].slot * a.mark_stride + used[j]] = (unsigned long long)~round << 32 | (uint32_t)q;
    }
}

// Fusion output: accepted pixels outside the sky (RunFusion_Sky_Strict, main.cpp:805).
__device__ __forceinline__ bool fused(const ScanRun& a, int q) {
    if (q >= a.npix || !(a.word[q] & kAccepted)) return false;
    if (!a.sky) return true;
    const uint8_t* s = a.sky + 3 * (size_t)q;
    return (int)s[0] != 234 && (int)s[1] != 235 && (int)s[2] != 55;
}

// Compaction of the fused points in three launches over tiles of kScanBlock
// pixels: tile totals, an exclusive scan of the totals onto the points already
// emitted (one block), and each tile's own scan, which writes the points.
// Warp scans by shuffle, then a scan of the 32 warp totals.
__device__ __forceinline__ int32_t warp_inclusive_sum(int32_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Inclusive sum over a block of kScanBlock threads; ws[31] holds the block
// total when it returns.  The caller syncs before ws is written again.
__device__ __forceinline__ int32_t block_inclusive_sum(int32_t v, int32_t* ws) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    v = warp_inclusive_sum(v);
    if (lane == 31) ws[w] = v;
    __syncthreads();
    if (w == 0) ws[lane] = warp_inclusive_sum(ws[lane]);
    __syncthreads();
    return v + (w > 0 ? ws[w - 1] : 0);
}

__global__ void __launch_bounds__(kScanBlock) k_fuse_count(const __grid_constant__ ScanRun a,
                                                           int32_t* __restrict__ tile_sum) {
    __shared__ int32_t ws[32];
    const int n = __popc(__ballot_sync(0xffffffffu, fused(a, blockIdx.x * kScanBlock + threadIdx.x)));
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = n;
    __syncthreads();
    if (threadIdx.x < 32) {
        const int32_t v = warp_inclusive_sum(ws[threadIdx.x]);
        if (threadIdx.x == 31) tile_sum[blockIdx.x] = v;
    }
}

// exclusive scan of the tile totals in place (one block, chunks with a carry); emitted[0] = points before
// this view, emitted[1] = after it
__global__ void __launch_bounds__(kScanBlock) k_scan_tile_sums(int32_t* __restrict__ tile_sum, int ntiles,
                                                               long long* __restrict__ emitted) {
    __shared__ int32_t ws[32];
    int32_t carry = 0;
    for (int base = 0; base < ntiles; base += kScanBlock) {
        const int q = base + threadIdx.x;
        const int32_t v = q < ntiles ? tile_sum[q] : 0;
        const int32_t inc = block_inclusive_sum(v, ws);
        if (q < ntiles) tile_sum[q] = carry + inc - v;
        carry += ws[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        emitted[0] = emitted[1];
        emitted[1] += carry;
    }
}

__global__ void __launch_bounds__(kScanBlock) k_fuse_emit(const __grid_constant__ ScanRun a,
                                                          const int32_t* __restrict__ tile_off,
                                                          const long long* __restrict__ emitted,
                                                          hpm_point* __restrict__ out, int64_t capacity) {
    __shared__ int32_t ws[32];
    const int q = blockIdx.x * kScanBlock + threadIdx.x;
    const bool keep = fused(a, q);
    const int32_t inc = block_inclusive_sum(keep ? 1 : 0, ws);
    if (!keep) return;
    const int64_t k = emitted[0] + tile_off[blockIdx.x] + inc - 1;
    if (k >= capacity) return;
    const int r = q / a.W, c = q - r * a.W;
    const float3 X = sc_world_point(c, r, a.depth[q], a.cam, a.centre);
    hpm_point p;
    p.coord[0] = X.x; p.coord[1] = X.y; p.coord[2] = X.z;
    for (int d = 0; d < 3; ++d) {
        p.normal[d] = a.normal[3 * (size_t)q + d];
        p.color[d] = (float)a.color[3 * (size_t)q + d];
    }
    out[k] = p;
}

// ---------------------------------------------------------------- host driver

template <class T>
static cudaError_t ensure_dev(T*& p, size_t& cap, size_t n) {
    if (n <= cap && p) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
    cudaError_t e = cudaMalloc((void**)&p, std::max<size_t>(n, 1) * sizeof(T));
    if (e == cudaSuccess) cap = n;
    return e;
}

int Ctx::consistency_scan(int mode, int n_views, const int32_t* src_off, const int32_t* src_ids, int depth_kind,
                          const uint8_t* const* sky_host, hpm_point* out, int64_t capacity, int64_t* n_points,
                          int* max_iterations_used) {
    cudaSetDevice(device);
    if (n_views < 1 || n_views > HPM_MAX_VIEWS || !src_off || !src_ids)
        return fail(HPM_E_INVALID, "consistency scan: bad arguments");
    if (depth_kind != HPM_MAP_DEPTH && depth_kind != HPM_MAP_DEPTH_GEOM)
        return fail(HPM_E_INVALID, "consistency scan: depth kind must be DEPTH or DEPTH_GEOM");
    size_t max_pix = 0;
    int max_ngb = 0;
    for (int v = 0; v < n_views; ++v) {
        ViewState& vs = views[v];
        const DevMap& dm = vs.maps[depth_kind];
        const DevMap& nm = vs.maps[HPM_MAP_NORMAL];
        if (!dm.ptr || !nm.ptr || dm.w != nm.w || dm.h != nm.h)
            return fail(HPM_E_STATE, "view %d lacks depth/normal maps of one size", v);
        if (vs.w != dm.w || vs.h != dm.h)
            return fail(HPM_E_STATE, "view %d: camera size %dx%d differs from its maps %dx%d", v, vs.w, vs.h, dm.w, dm.h);
        const int ng = src_off[v + 1] - src_off[v];
        if (ng < 0 || ng > 31) return fail(HPM_E_INVALID, "view %d has %d sources (max 31)", v, ng);
        for (int k = src_off[v]; k < src_off[v + 1]; ++k)
            if (src_ids[k] < 0 || src_ids[k] >= n_views || src_ids[k] == v)
                return fail(HPM_E_INVALID, "view %d: invalid source id %d", v, src_ids[k]);
        max_ngb = std::max(max_ngb, ng);
        if (mode == 1 && (!vs.color || vs.color_w != dm.w || vs.color_h != dm.h))
            return fail(HPM_E_STATE, "view %d lacks a colour image of its map size", v);
        max_pix = std::max(max_pix, (size_t)dm.w * dm.h);
    }
    // per-view scan state, carved out of one allocation in 256-byte aligned pieces
    auto al = [](size_t bytes) { return (bytes + 255) & ~size_t(255); };
    struct State { uint8_t* mask; float* cons; const uint8_t* sky; };
    std::vector<State> hv(n_views);
    size_t state_bytes = 0;
    auto pixels = [&](int v) { return (size_t)views[v].w * views[v].h; };
    for (int v = 0; v < n_views; ++v)
        state_bytes += al(pixels(v)) + (mode == 0 ? al(4 * pixels(v)) : (sky_host && sky_host[v] ? al(3 * pixels(v)) : 0));
    cudaError_t e = ensure_dev(scan_state, scan_state_cap, state_bytes);
    if (e != cudaSuccess) return cuda_fail(e, "alloc scan state");
    uint8_t* cur = scan_state;
    auto carve = [&](size_t bytes) { uint8_t* p = cur; cur += al(bytes); return p; };
    for (int v = 0; v < n_views; ++v) {
        hv[v].mask = carve(pixels(v));
        hv[v].cons = mode == 0 ? reinterpret_cast<float*>(carve(4 * pixels(v))) : nullptr;
    }
    e = cudaMemsetAsync(scan_state, 0, cur - scan_state, stream);
    if (e != cudaSuccess) return cuda_fail(e, "clear scan state");
    for (int v = 0; v < n_views; ++v) {
        hv[v].sky = nullptr;
        if (mode == 1 && sky_host && sky_host[v]) {
            uint8_t* sky = carve(3 * pixels(v));
            e = cudaMemcpyAsync(sky, sky_host[v], 3 * pixels(v), cudaMemcpyHostToDevice, stream);
            if (e != cudaSuccess) return cuda_fail(e, "upload sky mask");
            hv[v].sky = sky;
        }
    }

    // work buffers, sized for the largest view and the most sources; the marks start as marked by no round
    const size_t ng = std::max(1, max_ngb);
    const size_t stride_max = (max_pix + kScanBlock - 1) / kScanBlock * kScanBlock;
    const size_t mark_stride = (max_pix + 3) & ~size_t(3);
    const size_t mark_bytes = al(8 * mark_stride * ng);
    const size_t wbytes = 2 * al(4 * stride_max * ng) + 3 * al(4 * stride_max) + al(4 * stride_max / kScanBlock) +
                          al(4 * stride_max / kScanBlock) + al(4 * (ng + 1) * (stride_max / 32)) +
                          (mode == 0 ? 2 : 1) * mark_bytes + al(64) +
                          al(4 * kMaxScanIterations);
    e = ensure_dev(scan_work, scan_work_cap, wbytes);
    if (e != cudaSuccess) return cuda_fail(e, "alloc scan work");
    cur = scan_work;
    ScanRun a{};
    a.pos = reinterpret_cast<int32_t*>(carve(4 * stride_max * ng));
    a.wexp = reinterpret_cast<float*>(carve(4 * stride_max * ng));
    a.test = reinterpret_cast<uint32_t*>(carve(4 * stride_max));
    a.word = reinterpret_cast<uint32_t*>(carve(4 * stride_max));
    a.dyn = reinterpret_cast<float*>(carve(4 * stride_max));
    a.chunk = reinterpret_cast<uint32_t*>(carve(4 * stride_max / kScanBlock));
    int32_t* tile_sum = reinterpret_cast<int32_t*>(carve(4 * stride_max / kScanBlock));
    a.map = reinterpret_cast<uint32_t*>(carve(4 * (ng + 1) * (stride_max / 32)));
    a.first_mark = reinterpret_cast<unsigned long long*>(carve(mark_bytes));
    a.last_mark = mode == 0 ? reinterpret_cast<unsigned long long*>(carve(mark_bytes)) : nullptr;
    a.mark_stride = mark_stride;
    long long* d_emitted = reinterpret_cast<long long*>(carve(64));
    int* d_changed = reinterpret_cast<int*>(carve(4 * kMaxScanIterations));  // one flag per round
    e = cudaMemsetAsync(a.first_mark, 0xff, mark_bytes, stream);
    if (e == cudaSuccess && mode == 0) e = cudaMemsetAsync(a.last_mark, 0, mark_bytes, stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_emitted, 0, 16, stream);
    if (e != cudaSuccess) return cuda_fail(e, "clear scan work");

    uint32_t round = 0;  // rounds of the whole scan, counted from 1: later ones win the atomicMin of the marks
    int expected = 4;    // rounds to launch before the first look at their change flags
    int max_iter = 0;
    for (int i = 0; i < n_views; ++i) {
        a.W = views[i].w;
        a.H = views[i].h;
        a.npix = a.W * a.H;
        a.stride = (a.npix + kScanBlock - 1) / kScanBlock * kScanBlock;
        a.n = src_off[i + 1] - src_off[i];
        a.cam = views[i].cam;
        camera_centre(a.cam, a.centre);
        a.depth = views[i].maps[depth_kind].ptr;
        a.normal = views[i].maps[HPM_MAP_NORMAL].ptr;
        a.color = views[i].color;
        a.sky = hv[i].sky;
        a.mask = hv[i].mask;
        a.cons = hv[i].cons;
        int max_sp = 1;
        a.distinct = true;
        for (int j = 0; j < a.n; ++j) {
            const int sid = src_ids[src_off[i] + j];
            ScanSource& s = a.src[j];
            s.cam = views[sid].cam;
            camera_centre(s.cam, s.centre);
            s.W = views[sid].w;
            s.H = views[sid].h;
            s.depth = views[sid].maps[depth_kind].ptr;
            s.normal = views[sid].maps[HPM_MAP_NORMAL].ptr;
            s.mask = hv[sid].mask;
            s.cons = hv[sid].cons;
            s.slot = (int)(std::find(src_ids + src_off[i], src_ids + src_off[i] + j, sid) - (src_ids + src_off[i]));
            a.distinct = a.distinct && s.slot == j;
            max_sp = std::max(max_sp, s.W * s.H);
        }
        const int blocks = (a.npix + 255) / 256;
        const int chunks = a.stride / kScanBlock;
        if (mode == 0) k_candidates<0><<<blocks, 256, 0, stream>>>(a);
        else k_candidates<1><<<blocks, 256, 0, stream>>>(a);
        ++launches;
        e = cudaMemsetAsync(d_changed, 0, 4 * kMaxScanIterations, stream);
        if (e != cudaSuccess) return cuda_fail(e, "clear change flags");
        int launched = 0, it = 0;
        bool converged = a.n == 0;
        while (!converged && launched < scan_rounds) {
            const int until = std::min(scan_rounds, launched + expected);
            const int from = launched;
            for (; launched < until; ++launched) {
                const int* before = launched ? d_changed + launched - 1 : nullptr;
                ++round;
                k_accept<<<chunks, kScanBlock, 0, stream>>>(a, before, round);
                k_mark_stale<<<blocks, 256, 0, stream>>>(a, before, round);
                k_update_eff<<<blocks, 256, 0, stream>>>(a, before, round, d_changed + launched);
                launches += 3;
            }
            int changed[kMaxScanIterations];
            e = cudaMemcpyAsync(changed + from, d_changed + from, 4 * (size_t)(launched - from), cudaMemcpyDeviceToHost,
                                stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
            if (e != cudaSuccess) return cuda_fail(e, "consistency iteration");
            for (int r = from; r < launched && !converged; ++r) {
                it = r + 1;
                converged = changed[r] == 0;
            }
            expected = converged ? expected : 2;
        }
        if (a.n == 0) {
            // no sources: nothing counted, nothing accepted (the words are the empty tests)
        } else if (!converged) {
            k_sequential<<<1, 1, 0, stream>>>(a, ++round);
            ++launches;
        } else {
            expected = std::min(16, std::max(2, it));
        }
        max_iter = std::max(max_iter, converged ? it : scan_rounds + 1);
        if (a.n > 0) {
            if (mode == 0) {
                k_settle<0><<<blocks, 256, 0, stream>>>(a, (uint32_t)i + 1);
                k_marked_conf<<<dim3((max_sp + 1023) / 1024, a.n), 256, 0, stream>>>(a, (uint32_t)i + 1);
                launches += 2;
            } else {
                k_settle<1><<<blocks, 256, 0, stream>>>(a, (uint32_t)i + 1);
                ++launches;
            }
        }
        if (mode == 0) {
            e = ensure_map(i, HPM_MAP_CONF, a.W, a.H);
            if (e != cudaSuccess) return cuda_fail(e, "alloc confidence map");
            k_conf_own<<<blocks, 256, 0, stream>>>(a, views[i].maps[HPM_MAP_CONF].ptr);
            ++launches;
        } else {
            k_fuse_count<<<chunks, kScanBlock, 0, stream>>>(a, tile_sum);
            k_scan_tile_sums<<<1, kScanBlock, 0, stream>>>(tile_sum, chunks, d_emitted);
            if (out) k_fuse_emit<<<chunks, kScanBlock, 0, stream>>>(a, tile_sum, d_emitted, out, capacity);
            launches += out ? 3 : 2;
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "consistency scan launch");
    }
    long long emitted[2] = { 0, 0 };
    e = cudaMemcpyAsync(emitted, d_emitted, sizeof(emitted), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return cuda_fail(e, "consistency scan");
    if (n_points) *n_points = emitted[1];
    if (max_iterations_used) *max_iterations_used = max_iter;
    return HPM_OK;
}

}  // namespace hpm
