// PatchMatch kernels of the plain FP32 path (sm_100a): random initialisation,
// red/black checkerboard propagation with the non-local sampling pattern, joint
// view selection and refinement, and the depth/normal export.
//
// Algorithm: HPM-MVS++ HPM.cu:567-842 (init, refinement), 843-1873 (standard
// propagation), 1875-2791 (mandatory consistency), 2793-2842 (schedule,
// export).  The kernels are laid out differently:
//   * one thread per pixel of the active colour, block 32 x 4 over (x, row
//     pair) so a warp covers a 32 x 2 strip (coherent texture reads);
//   * the pixel's reference patch (weights and weighted texels) lives in
//     registers and is built once per launch instead of once per NCC;
//   * images of whole grey levels are sampled from 8-bit textures with the same
//     bits as float ones (Ctx::bind_bytes), and their weights come from a table;
//   * NCCs whose view weight is zero are not evaluated (their product with the
//     zero weight is exactly 0 because the NCC is never NaN), and a reference
//     patch with variance < 1e-5 yields cost 2 for every hypothesis without
//     sampling (exactly the reference's result);
//   * a refinement candidate is dropped at the view where its partial cost
//     already rules it out.
//
// What bounds a half-sweep.  Three things compete on an SM: the texture data
// pipe (36 fetches per NCC; a quad of lanes that samples apart takes up to four
// passes), instruction fetch (the NCC is straight-line code, since its patch is
// in registers, and the warps stand at different places), and the latency of
// the serial parts around the NCCs.  Six half-sweeps of one run, ms, S = 10,
// before and after each change, all with the same bits:
//   code size 291 -> 130 KB, 124 since (loops and calls outside the NCC):
//                      1600x1200 mandatory 48.5 -> 42.0, prior 31.2 -> 22.8
//   8-bit textures:    800x600 photometric 13.4 -> 11.0 (2.2 -> 1.4 passes a quad)
//   pairs of samples in one instruction (f32x2):  mandatory 42.0 -> 39.0
//   weight table, candidate planes gathered at once:  mandatory 39.0 -> 37.5
//   candidates dropped early:  800x600 photometric 11.4 -> 11.0
//   the next 12 fetches issued before these are summed:  mandatory 37.3 -> 36.2
// Twelve warps per SM at 168 registers and sixteen at 128 (texels of the patch
// packed in bytes) ran alike; eight at 220 registers were 15-25 % slower, and
// blocks of 64 threads up to 15 % slower while the code was large.
// Arithmetic follows include/hpm_fp.h (IEEE fp32, explicit fused multiply-adds),
// which the CPU oracle shares, so the two differ only where the texture unit's
// filtered sample does (about 0.6 % of samples, by one ulp).
#include "hpm_device.cuh"
#include "pm_kernels.cuh"

#include <float.h>
#include <limits.h>

namespace hpm {


// Per-thread columns of shared memory of the initialisation: the costs of one
// hypothesis by view, and the same sorted.
template <int NS, int BLK>
struct InitScratch {
    float* base;  // smem + threadIdx linear
    static constexpr int kWords = 2 * NS;
    __device__ __forceinline__ float& ca(int d, int j) const { return base[(d * NS + j) * BLK]; }
};

// A source view's part of the geometric cost, in shared memory: in view selection every lane goes
// through its own selected views.
struct alignas(16) GeomView {
    float fwd_A[9], fwd_b[3], bwd_A[9], bwd_b[3];
    const float* depth;
    int w, h;
};
static_assert(sizeof(GeomView) == 112, "seven 16-byte loads");

// Per-thread scratch of a half-sweep, in blocks of at most BLK threads.  The cost rows of the eight
// directions are written once, an NCC apart, and read once, by view selection: they stream through the
// thread's local memory, so that shared memory (view weights, final costs, candidate positions) leaves
// the L1 to the textures and the registers alone bound the resident warps.  After view selection the
// rows' words hold the refinement's candidates and the state they are tested against, which would
// otherwise sit in registers across every NCC.
template <int NS, int BLK>
struct Scratch {
    float* base;   // smem + threadIdx linear
    float* rows;   // local memory, kRowWords
    float4* cand;  // local memory: plane_m of the eight directions' planes and their depth at the pixel
    const GeomView* views;  // shared memory, geometric modes only
    static constexpr int kWords = NS + 16;
    static constexpr int kRowWords = 8 * NS < 72 ? 72 : 8 * NS;  // at least a patch's texels and weights
    __device__ __forceinline__ float& ca(int d, int j) const { return rows[d * NS + j]; }
    __device__ __forceinline__ float4 held(int i) const {
        return make_float4(rows[4 * i], rows[4 * i + 1], rows[4 * i + 2], rows[4 * i + 3]);
    }
    __device__ __forceinline__ void hold(int i, float4 v) const {
        rows[4 * i] = v.x; rows[4 * i + 1] = v.y; rows[4 * i + 2] = v.z; rows[4 * i + 3] = v.w;
    }
    __device__ __forceinline__ float& vw(int j) const { return base[j * BLK]; }
    __device__ __forceinline__ float& fc(int d) const { return base[(NS + d) * BLK]; }
    __device__ __forceinline__ int& pos(int d) const { return reinterpret_cast<int*>(base)[(NS + 8 + d) * BLK]; }
};

constexpr int kWeightRows = 6;
static_assert(kWeightRows * 256 == kWeightTable, "RunArgs::weights");

constexpr int kSweepThreads = 128;
constexpr int kEvalThreads = 128;
constexpr int kSweepBlocks = 3;  // resident blocks per SM: at most 168 registers a thread

// Statistics of a pixel's reference patch (the view-independent part of the NCC).
struct RefStats {
    float mean;   // sum_ref / weight_sum
    float var;    // reference variance
    float inv_w;  // 1 / weight_sum
};

// Two floats in a register pair; one instruction works on both, each rounded as the scalar one.  The
// NCC takes two patch columns at a time, whose sums are separate, so pairing them changes no order.
using Pair = unsigned long long;

__device__ __forceinline__ Pair pair_of(float lo, float hi) {
    Pair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 halves(Pair a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) {
    Pair r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ Pair add2(Pair a, Pair b) {
    Pair r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ Pair mul2(Pair a, Pair b) {
    Pair r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// A pixel's reference patch in registers: the bilateral weights w_k and the weighted texels w_k r_k of
// samples k = 6 i + j (column-major), those of columns i and i + 1 (i even) in row j as a pair.
struct Patch {
    Pair w[kPatchSamples / 2], wr[kPatchSamples / 2];
    RefStats rs;
    __device__ __forceinline__ Pair w2(int i, int j) const { return w[3 * i + j]; }
    __device__ __forceinline__ Pair wr2(int i, int j) const { return wr[3 * i + j]; }
};

// The bilateral weight of a patch texel |dx|, |dy| = 5, 3 or 1 away and `d` grey levels off the centre.
__device__ __forceinline__ float bilateral_weight(int dx, int dy, float d, float two_ss, float two_sc) {
    const float sd = sqrtf((float)(dx * dx + dy * dy));
    return hpm_expf(-sd / two_ss - d / two_sc);
}

// Rows of the weight table: the six distances of a patch sample, by (|dx|, |dy|) in either order.
__host__ __device__ constexpr int weight_row(int dx, int dy) {
    const int a = dx < 0 ? -dx : dx, b = dy < 0 ? -dy : dy;
    const int hi = a > b ? a : b, lo = a > b ? b : a;
    return hi == 5 ? (lo - 1) / 2 + 3 : (hi == 3 ? (lo - 1) / 2 + 1 : 0);
}

#ifndef HPM_NS
// The weights of a reference of whole levels: kWeightRows x 256 values, one per distance and level
// difference (RunArgs::weights).
__global__ void k_weight_table(float two_ss, float two_sc, float* __restrict__ out) {
    const int row = blockIdx.x, d = threadIdx.x;
    const int hi = row < 1 ? 1 : (row < 3 ? 3 : 5), lo = row < 1 ? 1 : (row < 3 ? 2 * (row - 1) + 1 : 2 * (row - 3) + 1);
    out[row * 256 + d] = bilateral_weight(hi, lo, (float)d, two_ss, two_sc);
}
#endif

// The patch in two ways with the same bits.  A reference of whole levels reads bytes and takes its
// weights from the table: 36 loads of each, all in flight, instead of 36 exponentials and 72 divisions.
// Any other forms the weights: in a loop, through kPatchWords words of the thread's local memory, where
// code size counts (half-sweeps), and UNROLLED elsewhere: the 36 chains side by side take 13 us less
// (hpm_eval_costs of one pixel: 50 and 37 us a call, of 10,000: 88 and 74).
constexpr int kPatchWords = 2 * kPatchSamples;

template <bool UNROLLED>
__device__ __forceinline__ void build_patch(const RunArgs& a, int px, int py, Patch& P, float* tmp) {
    const int W = a.W, H = a.H;
    const int at = clampi(py, 0, H - 1) * W + clampi(px, 0, W - 1);
    float r[kPatchSamples], w[kPatchSamples];
    float center;
    if (a.whole_levels) {
        const int c = __ldg(a.ref_bytes + at);
        center = (float)c;
        int t[kPatchSamples];
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            const uint8_t* row = a.ref_bytes + (size_t)clampi(py - kPatchRadius + kPatchStep * j, 0, H - 1) * W;
#pragma unroll
            for (int i = 0; i < 6; ++i)
                t[i * 6 + j] = __ldg(row + clampi(px - kPatchRadius + kPatchStep * i, 0, W - 1));
        }
#pragma unroll
        for (int k = 0; k < kPatchSamples; ++k) {
            const int dx = -kPatchRadius + kPatchStep * (k / 6), dy = -kPatchRadius + kPatchStep * (k % 6);
            w[k] = __ldg(a.weights + weight_row(dx, dy) * 256 + abs(t[k] - c));
            // a byte as the low mantissa bits of 2^23, less 2^23: exact
            r[k] = __uint_as_float(0x4B000000u | (uint32_t)t[k]) - 8388608.0f;
        }
    } else {
        center = __ldg(a.ref_img + at);
        const float two_ss = 2.0f * a.prm.sigma_spatial * a.prm.sigma_spatial;
        const float two_sc = 2.0f * a.prm.sigma_color * a.prm.sigma_color;
        auto sample = [&](int k, float& texel, float& weight) {
            const int dx = -kPatchRadius + kPatchStep * (k / 6), dy = -kPatchRadius + kPatchStep * (k % 6);
            const float t = __ldg(a.ref_img + (size_t)clampi(py + dy, 0, H - 1) * W + clampi(px + dx, 0, W - 1));
            texel = t;
            weight = bilateral_weight(dx, dy, fabsf(t - center), two_ss, two_sc);
        };
        if (UNROLLED) {
#pragma unroll
            for (int k = 0; k < kPatchSamples; ++k) sample(k, r[k], w[k]);
        } else {
#pragma unroll 1
            for (int k = 0; k < kPatchSamples; ++k) sample(k, tmp[k], tmp[kPatchSamples + k]);
#pragma unroll
            for (int k = 0; k < kPatchSamples; ++k) {
                r[k] = tmp[k];
                w[k] = tmp[kPatchSamples + k];
            }
        }
    }
    // shifted moments (precision form): the patch relative to its centre texel; shift 0 is the plain arithmetic
    const float cs = a.ncc_shift ? center : 0.0f;
    float s_r = 0.f, s_rr = 0.f, s_w = 0.f;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        float r_r = 0.f, r_rr = 0.f, r_w = 0.f;
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            const int k = i * 6 + j;
            const float rs = r[k] - cs;
            r[k] = w[k] * rs;
            r_r += r[k];
            r_rr = hpm_fma(r[k], rs, r_rr);
            r_w += w[k];
        }
        s_r += r_r; s_rr += r_rr; s_w += r_w;
    }
#pragma unroll
    for (int q = 0; q < kPatchSamples / 2; ++q) {
        const int k = 12 * (q / 6) + q % 6;
        P.w[q] = pair_of(w[k], w[k + 6]);
        P.wr[q] = pair_of(r[k], r[k + 6]);
    }
    P.rs.inv_w = 1.0f / s_w;
    P.rs.mean = s_r * P.rs.inv_w;
    P.rs.var = s_rr * P.rs.inv_w - P.rs.mean * P.rs.mean;
}

// m = Kr^-T n / d of a camera-frame hypothesis: the view-independent part of
// its homographies (include/hpm_geometry.h).
struct PlaneM {
    float m[3];
};

__device__ __forceinline__ PlaneM plane_m(const RunArgs& a, float4 pl) {
    PlaneM r;
    hpm_plane_m(a.kinv, pl.x, pl.y, pl.z, pl.w, r.m);
    return r;
}

// One bilateral NCC (HPM.cu:375-448) with the patch in registers.  CNT: the
// counting build also counts the NCCs that sample the source (hyp_count[2]).
template <bool CNT>
__device__ __forceinline__ float ncc_view(const RunArgs& a, const Patch& P, int px, int py, const PlaneM& pm, int j) {
    const float cost_max = 2.0f;
    if (P.rs.var < 1e-5f) return cost_max;
    const hpm_camera& sc = a.cams[j + 1];
    float H[9];
    hpm_homography(a.basis[j + 1].A, a.basis[j + 1].b, pm.m, H);
    const int sw = sc.width, sh = sc.height;
    float iz_c;
    {
        const float fx = (float)px, fy = (float)py;
        const float cx = hpm_fma(H[0], fx, hpm_fma(H[1], fy, H[2]));
        const float cy = hpm_fma(H[3], fx, hpm_fma(H[4], fy, H[5]));
        const float cz = hpm_fma(H[6], fx, hpm_fma(H[7], fy, H[8]));
        iz_c = 1.0f / cz;
        const float ux = cx * iz_c, uy = cy * iz_c;
        if (ux >= sw || ux < 0.0f || uy >= sh || uy < 0.0f) return cost_max;
    }
    if (CNT) {  // one atomic per group of converged lanes
        unsigned lane;
        asm("mov.u32 %0, %%laneid;" : "=r"(lane));
        const unsigned m = __activemask();
        if (lane == (unsigned)(__ffs(m) - 1)) atomicAdd(a.hyp_count + 2, (unsigned long long)__popc(m));
    }
    const cudaTextureObject_t tex = a.tex[j + 1];
    float s_s = 0.f, s_ss = 0.f, s_rs = 0.f;
    // Every fetch is carried through RunArgs::tex_scale and tex_bias; taken off are the bias or, for
    // shifted moments, the patch's first sample.
    float vshift = -a.tex_bias;
    const Pair one = pair_of(1.0f, 1.0f), izc = pair_of(iz_c, iz_c);
    const Pair h0 = pair_of(H[0], H[0]), h3 = pair_of(H[3], H[3]), h6 = pair_of(-H[6], -H[6]);
    // Two patch columns make 12 fetches; the next two columns' are issued before the moments of these
    // are summed, so the texture unit has work while the sums run.  The summation order is the oracle's.
    float v[2][2][6];
    auto fetch = [&](int i0, float (&o)[2][6]) {
        const float x = (float)(px - kPatchRadius + kPatchStep * i0);
        const Pair xx = pair_of(x, x + (float)kPatchStep);
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const float y = (float)(py - kPatchRadius + kPatchStep * k);
            const float tx = hpm_fma(H[1], y, H[2]), ty = hpm_fma(H[4], y, H[5]), tz = hpm_fma(-H[7], y, -H[8]);
            const float2 qx = halves(fma2(h0, xx, pair_of(tx, tx)));
            const float2 qy = halves(fma2(h3, xx, pair_of(ty, ty)));
            const Pair nqz = fma2(h6, xx, pair_of(tz, tz));  // -q_z
            // hpm_recip_near(q_z, iz_c) of both
            Pair r = fma2(izc, fma2(nqz, izc, one), izc);
            r = fma2(r, fma2(nqz, r, one), r);
            const float2 iz = halves(r);
            o[0][k] = tex2D<float>(tex, hpm_fma(qx.x, iz.x, 0.5f), hpm_fma(qy.x, iz.x, 0.5f));
            o[1][k] = tex2D<float>(tex, hpm_fma(qx.y, iz.y, 0.5f), hpm_fma(qy.y, iz.y, 0.5f));
        }
    };
    fetch(0, v[0]);
#pragma unroll
    for (int i0 = 0; i0 < 6; i0 += 2) {
        const float (&vc)[2][6] = v[(i0 >> 1) & 1];
        if (i0 < 4) {
            fetch(i0 + 2, v[((i0 >> 1) + 1) & 1]);
            asm volatile("" ::: "memory");  // the compiler keeps these fetches ahead of the sums below
        }
        Pair r_s = 0, r_ss = 0, r_rs = 0;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            Pair vk = pair_of(vc[0][k], vc[1][k]);
            vk = fma2(vk, pair_of(a.tex_scale, a.tex_scale), pair_of(a.tex_bias, a.tex_bias));
            if (i0 == 0 && k == 0 && a.ncc_shift) vshift = -halves(vk).x;
            vk = add2(vk, pair_of(vshift, vshift));
            const Pair ws = mul2(P.w2(i0, k), vk);
            r_s = add2(r_s, ws);
            r_ss = fma2(ws, vk, r_ss);
            r_rs = fma2(P.wr2(i0, k), vk, r_rs);
        }
        const float2 c_s = halves(r_s), c_ss = halves(r_ss), c_rs = halves(r_rs);
        s_s += c_s.x; s_ss += c_ss.x; s_rs += c_rs.x;
        s_s += c_s.y; s_ss += c_ss.y; s_rs += c_rs.y;
    }
    s_s *= P.rs.inv_w; s_ss *= P.rs.inv_w; s_rs *= P.rs.inv_w;
    const float var_s = s_ss - s_s * s_s;
    if (var_s < a.var_s_min) return cost_max;
    const float cov = s_rs - P.rs.mean * s_s;
    const float vrs = sqrtf(P.rs.var * var_s);
    return fmaxf(0.0f, fminf(cost_max, 1.0f - cov / vrs));
}

// ---------------------------------------------------------------- init

template <int NS, int BLK, bool CNT>
__device__ __forceinline__ float initial_cost(const RunArgs& a, const Patch& P, int px, int py, float4 pl, uint32_t* sel_out,
                              const InitScratch<NS, BLK>& s) {
    const float cost_max = 2.0f;
    const int S = a.S;
    int valid = 0;
    if (CNT) atomicAdd(a.hyp_count, (unsigned long long)a.S);
    const PlaneM pm = plane_m(a, pl);
#pragma unroll 1
    for (int j = 0; j < S; ++j) {
        const float c = ncc_view<false>(a, P, px, py, pm, j);
        s.ca(0, j) = c;
        s.ca(1, j) = c;
        if (c < cost_max) ++valid;
    }
    // insertion sort of row 1 (HPM.cu:15-24)
    for (int i = 1; i < S; ++i) {
        const float t = s.ca(1, i);
        int k = i;
        for (; k >= 1 && t < s.ca(1, k - 1); --k) s.ca(1, k) = s.ca(1, k - 1);
        s.ca(1, k) = t;
    }
    uint32_t sel = 0;
    const int top_k = min(valid, a.prm.top_k);
    float result = cost_max;
    if (top_k > 0) {
        float cost = 0.0f;
        for (int i = 0; i < top_k; ++i) cost += s.ca(1, i);
        const float thr = s.ca(1, top_k - 1);
        for (int i = 0; i < S; ++i)
            if (s.ca(0, i) <= thr) sel |= (1u << i);
        result = cost / top_k;
    }
    *sel_out = sel;
    return result;
}

__device__ __forceinline__ float spatial_gauss(float x1, float y1, float x2, float y2, float sigma) {
    const float dx = x1 - x2, dy = y1 - y2;
    const float dis = dx * dx + dy * dy - 0.0f;
    return (float)exp(-1.0 * dis / (2 * sigma * sigma));
}

__device__ __forceinline__ float range_gauss(float x, float sigma) {
    return (float)exp(-1.0 * (x * x) / (2 * sigma * sigma));
}

template <int NS, int BLK, bool CNT>
__device__ __forceinline__ void init_pixel(const RunArgs& a, const InitScratch<NS, BLK>& s, int px, int py) {
    const int W = a.W, H = a.H;
    if (px >= W || py >= H) return;
    const int center = py * W + px;
    const hpm_camera& c0 = a.cams[0];
    const uint32_t mode = a.prm.mode;
    const bool geom = mode & HPM_MODE_GEOM, prior = mode & HPM_MODE_PRIOR, hier = mode & HPM_MODE_HIERARCHY;
    const bool ups = mode & HPM_MODE_UPSAMPLE, mand = mode & HPM_MODE_MAND;
    PixelRng rng;
    rng.init(a.seed, a.view_id, px, py, 0);

    if (!prior && !mand) a.texture[center] = texture_term(a.canny, W, H, px, py);

    // What the pixel starts from: the plane to store, and the hypothesis to cost against all sources,
    // if any.  Every mode meets in one costing loop, so the kernel carries one copy of the NCC.
    bool store = true, cost = true;
    float4 pl = a.planes[center];
    float pre_depth = 0.0f;  // upsample mode: offset of the pre-cost hypothesis
    if (!geom && !hier && !prior) {
        const float depth = rng.uniform() * (a.prm.depth_max - a.prm.depth_min) + a.prm.depth_min;
        pl = random_normal(c0, px, py, rng, depth);
        pl.w = depth;
    } else if (prior) {
        const bool sure = a.conf[center] > 0.3;
        if (a.pmask[center] > 0) {
            if (sure) {
                a.costs[center] = 0.1f;
                cost = false;
            } else if (a.costs[center] > 0.1f) {
                const float perturbation = 0.02f;
                const float4 pp = a.prior[center];
                float dp = pp.w;  // the prior's offset is used as a depth (HPM.cu:603-604)
                const float dmin_p = (1 - 3 * perturbation) * dp;
                const float dmax_p = (1 + 3 * perturbation) * dp;
                dp = rng.uniform() * (dmax_p - dmin_p) + dmin_p;
                pl = perturbed_normal(c0, px, py, pp, rng, (float)(3 * perturbation * 3.14159265358979323846));
                pl.w = dp;
                store = false;
                a.planes[center] = pl;
            }
        } else {
            cost = false;
            if (sure) a.costs[center] = 0.1f;
        }
    } else if (ups) {
        const int scols = a.prm.scaled_cols, srows = a.prm.scaled_rows;
        const float sc_f = (float)scols, sr_f = (float)srows;
        const float scale = (float)(1.0 * sc_f / W);
        const float sigmad = 0.50f, sigmar = 25.5f;
        const int image_scale = (int)fmaxf(W / sc_f, H / sr_f);
        const int nn = (image_scale * image_scale + 1) / 2;
        const float o_y = py * scale, o_x = px * scale;
        const float ref_pix = __ldg(a.ref_img + center);
        float nf = 0.0f;
        float n0 = 0.0f, n1 = 0.0f, n2 = 0.0f;
        for (int j = -nn; j <= nn; ++j) {
            int r_y = __float2int_rz(o_y + j);
            r_y = (r_y > 0 ? (r_y < sr_f ? r_y : srows - 1) : 0);
            const int r_ys = clampi(py + j, 0, H - 1);
#pragma unroll 1
            for (int i = -nn; i <= nn; ++i) {
                int r_x = __float2int_rz(o_x + i);
                r_x = (r_x > 0 ? (r_x < sc_f ? r_x : scols - 1) : 0);
                const int s_center = (int)(r_y * sc_f + r_x);
                const float4 sn = a.scaled[s_center];
                const float nb = __ldg(a.ref_img + (size_t)r_ys * W + clampi(px + i, 0, W - 1));
                const float tg = spatial_gauss(o_x, o_y, (float)r_x, (float)r_y, sigmad) *
                                 range_gauss(fabsf(ref_pix - nb), sigmar);
                nf += tg;
                n0 = n0 + sn.x * tg; n1 = n1 + sn.y * tg; n2 = n2 + sn.z * tg;
            }
        }
        float4 nt = make_float4(n0 / nf, n1 / nf, n2 / nf, 0.0f);
        normalize3(nt);
        pre_depth = pl.w;
        pl = rotate_to_cam(c0, nt);
        pl.w = pre_depth;
    } else {
        if (mand && !(a.conf[center] >= 0.3)) {
            if (texture_term(a.canny, W, H, px, py) > 0.5) a.conf[center] = 0.1f;
        }
        if (hier) pl = a.scaled[center];
        pl = rotate_to_cam(c0, pl);
    }
    if (store) {
        // pl.w is the depth here; the perturbed prior keeps its depth as the offset (HPM.cu:603-604)
        pl.w = distance_to_origin(c0, px, py, pl.w, pl);
        a.planes[center] = pl;
    }
    a.rng[center] = rng.draw;
    if (!cost) return;

    Patch P;
    build_patch<true>(a, px, py, P, nullptr);
    uint32_t sel = 0;
    // upsample mode costs the pre-cost plane first: zero normal, upsampled depth as offset (HPM.cu:689,
    // HPM.cpp:894-901)
#pragma unroll 1
    for (int h = ups ? 0 : 1; h < 2; ++h) {
        const float4 hyp = h ? pl : make_float4(0.f, 0.f, 0.f, pre_depth);
        const float c = initial_cost<NS, BLK, CNT>(a, P, px, py, hyp, &sel, s);
        (h ? a.costs : a.pre_costs)[center] = c;
    }
    a.sel[center] = sel;
}

// 32 x 4 blocks, 12 warps per SM: 1.10 ms per 1600x1200 geometric initialisation with one costing loop,
// byte textures and the weight table, against 1.50 with an inlined copy of the NCC per mode
template <int NS, int BLK, bool CNT>
__global__ void __launch_bounds__(BLK, kSweepBlocks) k_random_init(const __grid_constant__ RunArgs a) {
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const InitScratch<NS, BLK> s{ smem + tid };
    init_pixel<NS, BLK, CNT>(a, s, blockIdx.x * blockDim.x + threadIdx.x, blockIdx.y * blockDim.y + threadIdx.y);
}

// ---------------------------------------------------------------- batched launches
//
// The batching form: the runs of several reference views (one pass of the
// schedule over the views of a pyramid level, main.cpp:1253-1255) share one
// launch per stage.  Their RunArgs sit in device memory; block b of the launch
// is tile b - tile_start[k] of run k, the last run with tile_start[k] <= b.
// A tile is the block footprint of the single-view launch, so every pixel sees
// exactly the arithmetic of the per-view kernels.  With gridDim.x smaller than
// the tile count the launch is persistent: each block walks the tiles b,
// b + gridDim.x, ...  The per-view kernels launch one view at a time and wait
// for each launch (HPM.cu:2987-3035); here the tail of one view's grid overlaps
// the next view's tiles.

__device__ __forceinline__ int batch_run_of(const int* __restrict__ tile_start, int n, int b) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(tile_start + mid) <= b) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

template <int NS, int BLK, bool CNT>
__global__ void __launch_bounds__(BLK, kSweepBlocks) k_random_init_batch(const RunArgs* __restrict__ args,
                                                           const int* __restrict__ tile_start, int n) {
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const InitScratch<NS, BLK> s{ smem + tid };
    const int total = __ldg(tile_start + n);
    for (int b = __ldg(tile_start) + blockIdx.x; b < total; b += gridDim.x) {
        const int k = batch_run_of(tile_start, n, b);
        const RunArgs& a = args[k];
        const int t = b - __ldg(tile_start + k);
        const int tx = (a.W + blockDim.x - 1) / blockDim.x;
        init_pixel<NS, BLK, CNT>(a, s, (t % tx) * blockDim.x + threadIdx.x, (t / tx) * blockDim.y + threadIdx.y);
    }
}

// ---------------------------------------------------------------- propagation

// The lowest-cost position of a diagonal path: `start`, then up to seven more, steps (ax, ay) and
// (bx, by) in turn from (x, y), while inside the image.
static __device__ __noinline__ int v_path_best(const float* __restrict__ costs, int W, int H, int x, int y, int ax,
                                               int ay, int bx, int by, int start) {
    int best = start;
    float bc = costs[best];
    float c[7];
    int q[7];
    bool in = true;
#pragma unroll
    for (int i = 0; i < 7; ++i) {
        if (i % 2 == 0) { x += ax; y += ay; } else { x += bx; y += by; }
        in = in && x >= 0 && x < W && y < H && y >= 0;  // the path ends where it leaves the image
        q[i] = in ? y * W + x : start;
        c[i] = costs[q[i]];
    }
#pragma unroll
    for (int i = 0; i < 7; ++i)
        if (c[i] < bc) { bc = c[i]; best = q[i]; }
    return best;
}

// Non-local candidate positions of the eight directions (HPM.cu:1367-1608);
// returns the bitmask of valid directions and leaves the positions in scratch.
// Odd directions (up, down, left, right): the first candidate 5 px away, then up
// to 4 more every 2 px while inside the image (HPM.cu:1385-1475); the last
// keeps the maximum (HPM.cu:1464).  Even ones (left-up, right-up, right-down,
// left-down): a diagonal path from 5 or 6 px away.
template <int NS, int BLK>
__device__ __forceinline__ uint32_t direction_search(const RunArgs& a, int px, int py, const Scratch<NS, BLK>& s) {
    const int W = a.W, H = a.H;
    const float* __restrict__ costs = a.costs;
    uint32_t flags = 0;
    // one straight and one diagonal direction a turn, their loads in flight together
#pragma unroll 1
    for (int d = 0; d < 8; d += 2) {
        const int dx = d == 4 ? -1 : (d == 6 ? 1 : 0), dy = d == 0 ? -1 : (d == 2 ? 1 : 0);
        const int x = px + 5 * dx, y = py + 5 * dy;
        const bool straight = !(x < 0 || x >= W || y < 0 || y >= H);
        float far_cost[5];
        bool far_in[5];
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            const int xi = px + (5 + 2 * i) * dx, yi = py + (5 + 2 * i) * dy;
            far_in[i] = !(xi < 0 || xi >= W || yi < 0 || yi >= H);
            far_cost[i] = far_in[i] ? costs[yi * W + xi] : 0.0f;
        }
        const int sx = px + (d == 0 ? -5 : d == 2 ? 6 : d == 4 ? 5 : -6);
        const int sy = py + (d == 0 ? -6 : d == 2 ? -5 : d == 4 ? 6 : 5);
        if (!(sx < 0 || sx >= W || sy < 0 || sy >= H)) {
            // left-up: (-2, 0) (0, -2); right-up: (0, -2) (2, 0); right-down: (2, 0) (0, 2); left-down: (0, 2) (-2, 0)
            const bool x_first = d == 0 || d == 4;
            const int ex = d == 0 || d == 6 ? -2 : 2, ey = d == 0 || d == 2 ? -2 : 2;
            s.pos(d) = v_path_best(costs, W, H, sx, sy, x_first ? ex : 0, x_first ? 0 : ey, x_first ? 0 : ex,
                                   x_first ? ey : 0, sy * W + sx);
            flags |= 1u << d;
        }
        if (straight) {
            int best = 0;
            float bc = far_cost[0];
#pragma unroll
            for (int i = 1; i < 5; ++i)
                if (far_in[i] && (d == 6 ? (bc < far_cost[i]) : (far_cost[i] < bc))) { bc = far_cost[i]; best = i; }
            s.pos(d + 1) = (py + (5 + 2 * best) * dy) * W + px + (5 + 2 * best) * dx;
            flags |= 2u << d;
        }
    }
    return flags;
}

struct Selection {
    uint32_t temp_selected;
    float weight_norm;
};

// Joint view selection and the eight final costs (HPM.cu:1686-1771), from the
// cost rows of the directions; weights to scratch vw, final costs to fc.
template <int NS, int BLK>
__device__ __forceinline__ Selection view_selection(const RunArgs& a, int px, int py, int iter, uint32_t flags,
                                                    PixelRng& rng, const Scratch<NS, BLK>& s) {
    const int W = a.W, S = a.S;
    const int center = py * W + px;
    const bool geom = a.prm.mode & HPM_MODE_GEOM;
    const int nbr[4] = { center - W * 5, center + W * 5, center - 5, center + 5 };
    uint32_t near[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) near[i] = (flags & (1u << (2 * i + 1))) ? a.sel[nbr[i]] : 0u;
    const float cost_thr = (float)(0.8 * hpm_expf((float)(iter * iter) / (-90.0f)));
    float sum = 0.0f;
#pragma unroll 1
    for (int j = 0; j < S; ++j) {
        float prior = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (flags & (1u << (2 * i + 1))) prior += ((near[i] >> j) & 1u) ? 0.9f : 0.1f;
        float count = 0.0f, tmpw = 0.0f, prob = 0.0f;
        int count_false = 0;
        float c[8];
#pragma unroll
        for (int d = 0; d < 8; ++d) c[d] = s.ca(d, j);
#pragma unroll 4
        for (int d = 0; d < 8; ++d) {
            const float e = hpm_expf(c[d] * c[d] / (-0.18f));
            if (c[d] < cost_thr) { tmpw += e; count += 1.0f; }
            if (c[d] > 1.2f) ++count_false;
        }
        if (count > 2 && count_false < 3) prob = tmpw / count;
        else if (count_false < 3) prob = hpm_expf(cost_thr * cost_thr / (-0.32f));
        prob = prob * prior;
        s.vw(j) = prob;
        sum += prob;
    }
    // 15 draws from the cumulative distribution, counted in 4 bits per view: a draw takes the first
    // view whose sum is above it.  The sums do not fall, so that is the view numbered by how many are
    // not above it (no view when the probabilities are all zero and the sums NaN).
    float cum[NS];
    {
        const float inv = 1.0f / sum;
        float acc = 0.0f;
#pragma unroll
        for (int j = 0; j < NS; ++j)
            if (j < S) { acc += s.vw(j) * inv; cum[j] = acc; }
    }
    uint32_t hits[(NS + 7) / 8];
#pragma unroll
    for (int k = 0; k < (NS + 7) / 8; ++k) hits[k] = 0;
#pragma unroll 1
    for (int smp = 0; smp < 15; ++smp) {
        const float rp = rng.uniform() - FLT_EPSILON;
        int first = 0;
#pragma unroll
        for (int j = 0; j < NS; ++j)
            if (j < S && !(cum[j] > rp)) ++first;
#pragma unroll
        for (int k = 0; k < (NS + 7) / 8; ++k)
            if (first < S && (first >> 3) == k) hits[k] += 1u << (4 * (first & 7));
    }
    Selection o;
    o.temp_selected = 0; o.weight_norm = 0.0f;
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        const uint32_t n = (hits[j >> 3] >> (4 * (j & 7))) & 15u;
        const float w = (float)n;
        s.vw(j) = w;
        if (n > 0) {
            o.temp_selected |= 1u << j;
            o.weight_norm += w;
        }
    }
    // Final costs of the directions (HPM.cu:1752-1771): sums over the selected views in their order.
    // View after view, so that the eight directions' depth gathers of the geometric cost are in
    // flight together.
    float fc[8];
#pragma unroll
    for (int d = 0; d < 8; ++d) fc[d] = s.fc(d) = 0.0f;
    if (!geom) {
#pragma unroll 1
        for (int j = 0; j < S; ++j) {
            const float w = s.vw(j);
            if (!(w > 0)) continue;
#pragma unroll
            for (int d = 0; d < 8; ++d) fc[d] += w * s.ca(d, j);
        }
    } else {
#pragma unroll 1
        for (uint32_t m = o.temp_selected; m; m &= m - 1) {
            const int j = __ffs(m) - 1;
            const float w = s.vw(j);
            const GeomView v = s.views[j];
#pragma unroll 1
            for (int h = 0; h < 8; h += 4) {
                float sx[4], sy[4], sd[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float depth = (flags >> (h + k)) & 1u ? s.cand[h + k].w : 0.0f;
                    sd[k] = geom_source_depth(v.depth, v.w, v.h, v.fwd_A, v.fwd_b, depth, px, py, sx[k], sy[k]);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float g = (flags >> (h + k)) & 1u
                                        ? 0.2f * geom_back_cost(v.bwd_A, v.bwd_b, sx[k], sy[k], sd[k], px, py)
                                        : 0.1f * 3.0f;
                    s.fc(h + k) += w * (s.ca(h + k, j) + g);
                }
            }
        }
    }
#pragma unroll
    for (int d = 0; d < 8; ++d) s.fc(d) = (geom ? s.fc(d) : fc[d]) / o.weight_norm;
    return o;
}

constexpr float kPriorBeta = 0.18f;

// The prior's factor of the score: how near the hypothesis is to the prior plane.
static __device__ __noinline__ float prior_factor(float depth_now, float depth_prior, float4 pp, float4 pl, float texture,
                                              float two_dss, float two_ass) {
    const float gamma = 0.5f;
    const float dd = depth_now - depth_prior;
    const float nd = fabsf(pp.x - pl.x) + fabsf(pp.y - pl.y) + fabsf(pp.z - pl.z);
    return (float)(gamma * (1.2 - 0.2 * texture) + (double)(hpm_expf(-dd * dd / two_dss) * hpm_expf(-nd * nd / two_ass)));
}

static __device__ __noinline__ float prior_score(float final_cost, float depth_now, float depth_prior, float4 pp,
                                             float4 pl, float texture, float two_dss, float two_ass) {
    const float prior = prior_factor(depth_now, depth_prior, pp, pl, texture, two_dss, two_ass);
    return (float)(exp(-final_cost * final_cost / kPriorBeta * (1 + 0.2 * texture)) * (double)prior);
}

// Threshold of a good cost in round `it` of the extension (HPM.cu:1063-1126).
static __device__ __noinline__ float good_threshold(int iter, int it) {
    return (float)(0.8 * exp(-iter * iter * (3 - it) / 90.0));
}

// Margins of the refinement's rejection limits.  A candidate is accepted when its weighted mean cost
// is below the current one (or, under a prior, when its score is above the current one, which falls
// with the cost).  The terms of the sum are not negative and rounded addition and division are
// monotone, so a partial sum above the limit is a rejection; the margins cover the rounding of the
// limit itself (a few units of 2^-24, and the logarithm's), ten and a hundred times over.
constexpr float kLimitMargin = 1.000002f;
constexpr float kLogMargin = 1e-5f;

// One pixel of a black or red half-sweep: CheckerboardPropagation (HPM.cu:1347-1873)
// or, with MAND, CheckerboardPropagation_MandatoryConsistency (HPM.cu:1875-2791).
//
// The NCC work runs in one loop of 17 slots, each costing at most one
// hypothesis:
//   slot  0      the left-up direction's candidate, against all sources;
//   slots 1-3    the three rounds of its extension (HPM.cu:1063-1126);
//   slots 4-10   the candidates of directions 1-7;
//   slot  11     view selection, then the current plane against the selected views;
//   slots 12-16  the five PlaneHypothesisRefinement candidates (HPM.cu:765-841),
//                built from the state at entry and accepted greedily in order.
// The decisions between slots are the reference's, in its order, and the
// random draws happen in the same sequence.
template <int NS, int BLK, bool MAND, bool CNT>
__device__ __forceinline__ void sweep_pixel(const RunArgs& a, float* smem_column, const GeomView* views, int px,
                                            int pair, int color, int iter) {
    const int py = 2 * pair + ((px & 1) ^ color);
    const int W = a.W, H = a.H, S = a.S;
    if (px >= W || py >= H || pair >= a.cover_pairs) return;
    const int center = py * W + px;
    const hpm_camera& c0 = a.cams[0];
    const uint32_t mode = a.prm.mode;
    const bool prior = mode & HPM_MODE_PRIOR, hier = mode & HPM_MODE_HIERARCHY, geom = mode & HPM_MODE_GEOM;
    const float dmin = a.prm.depth_min, dmax = a.prm.depth_max;

    if (!MAND && prior) {
        if (a.conf[center] > 0.3) return;
        if (a.pmask[center] == 0) return;
    }
    float rows[Scratch<NS, BLK>::kRowWords];
    float4 cand[8];
    const Scratch<NS, BLK> s{ smem_column, rows, cand, views };
    Patch P;
    build_patch<false>(a, px, py, P, rows);
    const uint32_t all_views = (S >= 32) ? 0xffffffffu : ((1u << S) - 1u);

    const uint32_t flags = direction_search(a, px, py, s);
    auto candidate = [&](int at) {
        const float4 p = a.planes[at];
        const PlaneM m = plane_m(a, p);
        return make_float4(m.m[0], m.m[1], m.m[2], geom ? depth_from_plane(c0, p, px, py) : 0.0f);
    };
#pragma unroll 4
    for (int d = 0; d < 8; ++d)  // the gathers in flight together, not one at each slot's head
        if ((flags >> d) & 1u) cand[d] = candidate(s.pos(d));
    // `float cost_array[8][32] = { 2.0f }` (HPM.cu:1378): the row of a direction outside the image is
    // 0, but [0][0] is 2.
    if (flags != 0xffu) {
        for (int d = 0; d < 8; ++d)
            if (!((flags >> d) & 1u))
                for (int j = 0; j < S; ++j) s.ca(d, j) = d + j == 0 ? 2.0f : 0.0f;
    }

    // state carried across slots
    bool extending = flags & 1u;  // left-up extension still active
    bool refine = false;          // slots 12-16 run
    uint32_t selected = 0;        // views of the selection, and the sum of their weights
    float weight_norm = 0.0f;
    float cost_now = 0.0f, restricted_cost = 0.0f;
    const float depth_sigma = (dmax - dmin) / 64.0f;
    const float two_dss = 2 * depth_sigma * depth_sigma;
    const float angle_sigma = (float)(3.14159265358979323846 * (5.0f / 180.0f));
    const float two_ass = 2 * angle_sigma * angle_sigma;
    // words of the scratch rows after view selection: 0-4 the candidates (normal, depth), 5 the plane
    // of the pixel, 6 the prior plane, 7 (prior depth, texture, prior used)
    constexpr int kHeldNow = 5, kHeldPrior = 6, kHeldTerms = 7;
#pragma unroll 1
    for (int t = 0; t < 17; ++t) {
        bool run = false;
        float4 pl = make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t mask = all_views;
        int row = 0;
        float depth = 0.0f;       // slots 11-16: the hypothesis' depth at the pixel (geometric cost)
        float limit = INFINITY;   // slots 12-16: a weighted cost sum above it is rejected
        if (t == 0) {
            run = flags & 1u;
        } else if (t < 4) {
            // Extended propagation: only orientation 0 (left_up) is active because
            // `bool symbol_eight_orientations[10] = { true }` (HPM.cu:1612, 1063-1126).
            const int it = t - 1;
            if (extending) {
                const float good_thr = good_threshold(iter, it);
                int good = 0, bad = 0;
                for (int j = 0; j < S; ++j) {
                    const float c = s.ca(0, j);
                    if (c < good_thr) ++good;
                    if (c > 1.2f) ++bad;
                }
                if (good >= 1 && bad <= 2) {
                    extending = false;
                } else if (px > 4 + 8 * it && py > 5 + 8 * it) {
                    const int sx = px - 5 - 8 * it, sy = py - 6 - 8 * it;
                    int best = sy * W + sx;
                    best = v_path_best(a.costs, W, H, sx, sy, -2, 0, 0, -2, best);
                    const int prev = s.pos(0);
                    if (a.costs[best] > a.costs[prev]) {
                        best = prev;
                    } else if (best != prev) {
                        run = true;
                        cand[0] = candidate(best);
                    }
                    // best == prev recomputes the same row in the reference: identical values
                    if (run) s.pos(0) = best;
                }
            }
        } else if (t < 11) {
            row = t - 3;
            run = (flags >> row) & 1u;
        } else if (t == 11) {
            PixelRng rng;
            rng.init(a.seed, a.view_id, px, py, a.rng[center]);
            const Selection sel = view_selection(a, px, py, iter, flags, rng, s);
            a.rng[center] = rng.draw;
            selected = sel.temp_selected;
            weight_norm = sel.weight_norm;
            run = true;
            pl = a.planes[center];
            mask = selected;
            if (geom) depth = depth_from_plane(c0, pl, px, py);
        } else if (refine) {
            // candidates (depth, normal): (rand, entry) (entry, rand) (rand, rand) (entry, perturbed) (perturbed, entry)
            pl = s.held(t - 12);
            const float dc = pl.w;
            pl.w = distance_to_origin(c0, px, py, dc, pl);
            run = true;
            mask = selected;
            depth = depth_from_plane(c0, pl, px, py);
            const float4 terms = s.held(kHeldTerms);
            if (!(depth >= dmin && depth <= dmax)) {
                mask = 0;
            } else if (terms.z == 0.0f) {
                limit = cost_now * weight_norm * kLimitMargin;
            } else if (restricted_cost > 0.0f) {
                const float lead = logf(prior_factor(dc, terms.x, s.held(kHeldPrior), pl, terms.y, two_dss, two_ass) /
                                        restricted_cost) + kLogMargin;
                if (lead > 0.0f)
                    limit = sqrtf(lead * kPriorBeta / (1.0f + 0.2f * terms.y)) * weight_norm * kLimitMargin;
                else
                    mask = 0, limit = -1.0f;
            }
        }

        // The hypothesis against the views in `mask`: cost rows of the directions (slots 0-10,
        // ComputeMultiViewCostVector, HPM.cu:490-495), or the weighted cost sum over the selected
        // views (HPM.cu:1775-1786, 805-817).  The only place a half-sweep evaluates the NCC, so the
        // kernel carries one copy.  The loop runs over view indices, the same for every lane: a
        // variant in which each lane took its own k-th selected view ran three times slower on B200,
        // because texture fetches with different texture objects across a warp serialise.
        float wcost = 0.0f;
        if (run) {
            if (CNT) atomicAdd(a.hyp_count + 1, (unsigned long long)S);
            PlaneM pm;
            if (t < 11) {
                const float4 m = cand[row];
                pm.m[0] = m.x; pm.m[1] = m.y; pm.m[2] = m.z;
            } else {
                pm = plane_m(a, pl);
            }
#pragma unroll 1
            for (int j = 0; j < S; ++j) {
                if (!((mask >> j) & 1u)) continue;
                const bool weighted = t >= 11;
                const float c = ncc_view<CNT>(a, P, px, py, pm, j);
                if (!weighted) {
                    s.ca(row, j) = c;
                } else {
                    const float w = s.vw(j);
                    float sx = 0.0f, sy = 0.0f, sd = 0.0f;
                    if (geom)
                        sd = geom_source_depth(a.depth_src[j + 1], a.dsw[j + 1], a.dsh[j + 1], a.fwd[j + 1].A,
                                               a.fwd[j + 1].b, depth, px, py, sx, sy);
                    if (geom)
                        wcost += w * (c + 0.2f * geom_back_cost(a.bwd[j + 1].A, a.bwd[j + 1].b, sx, sy, sd, px, py));
                    else
                        wcost += w * c;
                    if (wcost > limit) mask = 0;
                }
            }
        }

        if (t == 11) {
            float4 cur = pl;
            if (!MAND || a.conf[center] >= 0.3) {
                int min_idx = 0;  // ties: the last (HPM.cu:41-52)
                float min_cost = s.fc(0);
#pragma unroll 1
                for (int d = 1; d < 8; ++d)
                    if (s.fc(d) <= min_cost) { min_cost = s.fc(d); min_idx = d; }
                const bool min_valid = flags & (1u << min_idx);
                cost_now = wcost / weight_norm;
                a.costs[center] = cost_now;
                const float cost_chk = cost_now;  // costs[center] as read by the NaN test
                float depth_now = depth_from_plane(c0, cur, px, py);
                float texture = 0.0f, depth_prior = 0.0f;
                float4 pp = make_float4(0.f, 0.f, 0.f, 0.f);
                float4 prior_pick = cur;  // prior mode: the maximum-score neighbour's plane, when valid
                bool has_pick = false;
                if (!MAND && prior) {
                    pp = a.prior[center];
                    depth_prior = depth_from_plane(c0, pp, px, py);
                    texture = texture_term(a.canny, W, H, px, py);
                    if (a.pmask[center] > 0) {
                        int max_idx = 0;  // ties: the last (HPM.cu:54-65)
                        float max_score = 0.0f;
#pragma unroll 1
                        for (int d = 0; d < 8; ++d) {
                            float score = 0.0f;
                            if (flags & (1u << d)) {
                                const float4 pd = a.planes[s.pos(d)];
                                const float dn = depth_from_plane(c0, pd, px, py);
                                score = prior_score(s.fc(d), dn, depth_prior, pp, pd, texture, two_dss, two_ass);
                            }
                            if (d == 0 || score >= max_score) { max_score = score; max_idx = d; }
                        }
                        const float rnow = prior_score(cost_now, depth_now, depth_prior, pp, cur, texture, two_dss,
                                                       two_ass);
                        if (flags & (1u << max_idx)) {
                            const float4 pd = a.planes[s.pos(max_idx)];
                            const float db = depth_from_plane(c0, pd, px, py);
                            prior_pick = pd;
                            has_pick = true;
                            if (db >= dmin && db <= dmax && max_score > rnow) {
                                // depth_now is left alone: HPM.cu:1815 shadows it in this block, so
                                // the refinement receives the pre-acceptance depth
                                cur = pd;
                                a.planes[center] = pd;
                                a.costs[center] = s.fc(max_idx);
                                restricted_cost = max_score;
                                a.sel[center] = selected;
                            }
                        }
                    } else if (min_valid) {
                        const float4 pd = a.planes[s.pos(min_idx)];
                        const float db = depth_from_plane(c0, pd, px, py);
                        if (db >= dmin && db <= dmax && min_cost < cost_now) {
                            depth_now = db;
                            cur = pd;
                            a.planes[center] = pd;
                            a.costs[center] = min_cost;
                        }
                    }
                }
                // plane_hypotheses_now (HPM.cu:1844, 2299) is assigned only when the neighbour
                // is accepted; the reference as compiled holds the minimum-cost neighbour's plane
                // whenever that direction is valid; prior mode never assigns it and holds the
                // maximum-score neighbour's plane when valid.  Otherwise it starts as the
                // pixel's current plane.
                float4 plane_now = (!MAND && prior && has_pick) ? prior_pick : cur;
                if ((MAND || !prior) && min_valid) {
                    const float4 pd = a.planes[s.pos(min_idx)];
                    const float db = depth_from_plane(c0, pd, px, py);
                    plane_now = pd;
                    if (db >= dmin && db <= dmax && min_cost < cost_now) {
                        depth_now = db; plane_now = pd; cost_now = min_cost;
                        a.sel[center] = selected;
                    }
                    if (cost_chk != cost_chk) {
                        if (!MAND) depth_now = db;
                        plane_now = pd; cost_now = min_cost;
                        a.sel[center] = selected;
                    }
                }
                // PlaneHypothesisRefinement's random draws (HPM.cu:765-799), before any candidate is costed
                refine = true;
                const bool use_prior = prior && a.pmask[center] > 0;
                const float perturbation = 0.02f;
                float4 plane_rand;
                float depth_rand;
                PixelRng rng;
                rng.init(a.seed, a.view_id, px, py, a.rng[center]);
                if (use_prior) {
                    depth_rand = rng.uniform() * 6 * depth_sigma + (depth_prior - 3 * depth_sigma);
                    plane_rand = perturbed_normal(c0, px, py, pp, rng, angle_sigma);
                } else {
                    depth_rand = rng.uniform() * (dmax - dmin) + dmin;
                    plane_rand = random_normal(c0, px, py, rng, depth_now);
                }
                const float dmin_p = (1 - perturbation) * depth_now;
                const float dmax_p = (1 + perturbation) * depth_now;
                const float depth_pert = rng.uniform() * (dmax_p - dmin_p) + dmin_p;
                const float4 plane_pert = perturbed_normal(c0, px, py, plane_now, rng,
                                                           (float)(perturbation * 3.14159265358979323846));
                a.rng[center] = rng.draw;
                s.hold(0, make_float4(plane_now.x, plane_now.y, plane_now.z, depth_rand));
                s.hold(1, make_float4(plane_rand.x, plane_rand.y, plane_rand.z, depth_now));
                s.hold(2, make_float4(plane_rand.x, plane_rand.y, plane_rand.z, depth_rand));
                s.hold(3, make_float4(plane_pert.x, plane_pert.y, plane_pert.z, depth_now));
                s.hold(4, make_float4(plane_now.x, plane_now.y, plane_now.z, depth_pert));
                s.hold(kHeldNow, plane_now);
                s.hold(kHeldPrior, pp);
                s.hold(kHeldTerms, make_float4(depth_prior, texture, use_prior ? 1.0f : 0.0f, 0.0f));
            } else {
                // mandatory consistency, unreliable pixel (HPM.cu:2684-2789)
                const float beta = 0.18f;
                const float mmc = __popc(selected) * 0.5f;
                // score of a cost under a confidence (HPM.cu:2691-2716)
                auto score_of = [&](float cost, float conf) {
                    const float gce = hpm_expf(-cost * cost / beta);
                    const float dm = fmaxf(0.0f, mmc - conf);
                    const float mce = (float)(0.5f + exp(-dm * dm / (mmc * mmc * 1.0)));
                    return (conf > 0) ? fmaxf(3.0f, mce) * gce : mce * gce;
                };
                float cost_u = wcost / weight_norm;
                const float cost_chk = cost_u;
                const float cc = a.conf[center];
                // the eight directions, then the pixel's own plane (d = 8)
                int max_idx = 0;  // ties: the last (HPM.cu:54-65)
                float max_score = 0.0f, max_cost = 0.0f, rnow = 0.0f;
#pragma unroll 1
                for (int d = 0; d < 9; ++d) {
                    const bool own = d == 8;
                    float score = 0.0f, cost = own ? cost_u : s.fc(d);
                    if (own || (flags & (1u << d))) {
                        const float cp = own ? cc : a.conf[s.pos(d)];
                        score = score_of(cost, cp);
                        if (!own && cp > 0) cost = (float)(cost * fmin((double)hpm_expf(-cp * 2), 0.35));
                    }
                    if (own) rnow = score;
                    else if (d == 0 || score >= max_score) { max_score = score; max_idx = d; max_cost = cost; }
                }
                if (cc < 0.3) cost_u = (float)(cost_u * exp(0.2 + cc * 2));
                else cost_u = cost_u * hpm_expf(-cc * 2);
                float4 pu = cur;  // HPM.cu:2761: the neighbour's plane whenever that direction is valid
                if (flags & (1u << max_idx)) {
                    const int pm = s.pos(max_idx);
                    const float4 pd = a.planes[pm];
                    pu = pd;
                    const float db = depth_from_plane(c0, pd, px, py);
                    if (db >= dmin && db <= dmax && max_score > rnow) {
                        pu = pd; cost_u = max_cost;
                        a.sel[center] = selected;
                        a.conf[center] = (float)(0.5 * a.conf[pm]);
                    }
                    if (cost_chk != cost_chk) {
                        pu = pd; cost_u = max_cost;
                        a.sel[center] = selected;
                        a.conf[center] = (float)(0.5 * a.conf[pm]);
                    }
                }
                a.costs[center] = cost_u;
                a.planes[center] = pu;
            }
        } else if (t >= 12 && refine) {
            // a sum cut short by its limit, or of no view (weight_norm 0: NaN), is rejected here
            const float tc = wcost / weight_norm;
            if (depth >= dmin && depth <= dmax) {
                const float4 terms = s.held(kHeldTerms);
                if (terms.z == 0.0f) {
                    if (tc < cost_now) {
                        s.hold(kHeldNow, pl);
                        cost_now = tc;
                    }
                } else if (limit >= 0.0f) {
                    const float rt = prior_score(tc, s.held(t - 12).w, terms.x, s.held(kHeldPrior), pl, terms.y,
                                                 two_dss, two_ass);
                    if (rt > restricted_cost) {
                        s.hold(kHeldNow, pl);
                        cost_now = tc;
                        restricted_cost = rt;
                    }
                }
            }
        }
    }

    if (refine && (MAND || !hier || cost_now < a.pre_costs[center] - 0.1f)) {
        a.costs[center] = cost_now;
        a.planes[center] = s.held(kHeldNow);
    }
}

// The views' geometry into shared memory, behind the threads' columns.  Every thread of the block calls it,
// before any returns: the geometric modes (a prior run may be one) end it with a barrier.
template <int NS, int BLK>
__device__ __forceinline__ GeomView* load_geom_views(const RunArgs& a, float* smem, int tid) {
    static_assert(Scratch<NS, BLK>::kWords * BLK % 4 == 0, "GeomView's alignment");
    GeomView* views = reinterpret_cast<GeomView*>(smem + Scratch<NS, BLK>::kWords * BLK);
    if (a.prm.mode & HPM_MODE_GEOM) {
        for (int j = tid; j < a.S; j += blockDim.x * blockDim.y) {
            GeomView v;
#pragma unroll
            for (int k = 0; k < 9; ++k) { v.fwd_A[k] = a.fwd[j + 1].A[k]; v.bwd_A[k] = a.bwd[j + 1].A[k]; }
#pragma unroll
            for (int k = 0; k < 3; ++k) { v.fwd_b[k] = a.fwd[j + 1].b[k]; v.bwd_b[k] = a.bwd[j + 1].b[k]; }
            v.depth = a.depth_src[j + 1];
            v.w = a.dsw[j + 1];
            v.h = a.dsh[j + 1];
            views[j] = v;
        }
        __syncthreads();
    }
    return views;
}

template <int NS, int BLK, bool MAND, bool CNT>
__global__ void __launch_bounds__(BLK, kSweepBlocks) k_half_sweep(const __grid_constant__ RunArgs a, int color, int iter,
                                                                    int first_pair, int last_pair) {
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const GeomView* views = load_geom_views<NS, BLK>(a, smem, tid);
    const int pair = first_pair + blockIdx.y * blockDim.y + threadIdx.y;
    if (pair >= last_pair) return;
    sweep_pixel<NS, BLK, MAND, CNT>(a, smem + tid, views, blockIdx.x * blockDim.x + threadIdx.x, pair, color, iter);
}

// Prior mode with work lists (RunArgs::active_px): thread x of a row pair takes the x-th pixel the
// sweep updates, so the pixels that return at once (confident, or outside the prior mask) leave
// whole warps idle instead of holding lanes of working ones.  Pixels of one colour read only the
// other colour's state, so the mapping does not change any result.
template <int NS, int BLK, bool CNT>
__global__ void __launch_bounds__(BLK, kSweepBlocks) k_half_sweep_listed(const __grid_constant__ RunArgs a,
                                                                         int color, int iter, int first_pair,
                                                                         int last_pair) {
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const GeomView* views = load_geom_views<NS, BLK>(a, smem, tid);
    const int pair = first_pair + blockIdx.y * blockDim.y + threadIdx.y;
    if (pair >= last_pair) return;
    const int k = color * a.cover_pairs + pair;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= a.active_n[k]) return;
    sweep_pixel<NS, BLK, false, CNT>(a, smem + tid, views, a.active_px[(size_t)k * a.W + x], pair, color, iter);
}

#ifndef HPM_NS
// The pixels a prior-mode half-sweep updates (CheckerboardPropagation returns at once where
// confidence > 0.3 or the prior mask is clear, HPM.cu:1352-1365): one warp per (row pair, colour)
// writes their columns in increasing order and their count.
__global__ void k_prior_active(const __grid_constant__ RunArgs a, int* __restrict__ out_px, int* __restrict__ out_n) {
    const int pair = blockIdx.x, color = blockIdx.y, lane = threadIdx.x;
    const int W = a.W, H = a.H;
    int* row = out_px + ((size_t)color * a.cover_pairs + pair) * W;
    int n = 0;
    for (int x0 = 0; x0 < W; x0 += 32) {
        const int px = x0 + lane;
        const int py = 2 * pair + ((px & 1) ^ color);
        bool act = false;
        if (px < W && py < H) {
            const int c = py * W + px;
            act = !(a.conf[c] > 0.3) && a.pmask[c] != 0;
        }
        const unsigned m = __ballot_sync(0xffffffffu, act);
        if (act) row[n + __popc(m & ((1u << lane) - 1u))] = px;
        n += __popc(m);
    }
    if (lane == 0) out_n[color * a.cover_pairs + pair] = n;
}

cudaError_t launch_prior_active(const RunArgs& a, int* px, int* n, cudaStream_t st) {
    if (a.cover_pairs <= 0) return cudaSuccess;
    k_prior_active<<<dim3(a.cover_pairs, 2), 32, 0, st>>>(a, px, n);
    return cudaGetLastError();
}
#endif

// The batched form of k_half_sweep_listed: tile t of run k maps to columns of that run's work lists.
template <int NS, int BLK, bool CNT>
__global__ void __launch_bounds__(BLK, kSweepBlocks)
    k_half_sweep_batch_listed(const RunArgs* __restrict__ args, const int* __restrict__ tile_start, int n,
                              int color, int iter) {
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const int total = __ldg(tile_start + n);
    for (int b = __ldg(tile_start) + blockIdx.x; b < total; b += gridDim.x) {
        const int k = batch_run_of(tile_start, n, b);
        const RunArgs& a = args[k];
        const int t = b - __ldg(tile_start + k);
        const int tx = (a.W + blockDim.x - 1) / blockDim.x;
        if (a.prm.mode & HPM_MODE_GEOM) __syncthreads();  // the tile before may still read its views
        const GeomView* views = load_geom_views<NS, BLK>(a, smem, tid);
        const int x = (t % tx) * blockDim.x + threadIdx.x;
        const int pair = (t / tx) * blockDim.y + threadIdx.y;
        if (pair >= a.cover_pairs) continue;
        const int r = color * a.cover_pairs + pair;
        if (x >= a.active_n[r]) continue;
        sweep_pixel<NS, BLK, false, CNT>(a, smem + tid, views, a.active_px[(size_t)r * a.W + x], pair, color, iter);
    }
}

template <int NS, int BLK, bool MAND, bool CNT>
__global__ void __launch_bounds__(BLK, kSweepBlocks)
    k_half_sweep_batch(const RunArgs* __restrict__ args, const int* __restrict__ tile_start, int n, int color,
                       int iter) {
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const int total = __ldg(tile_start + n);
    for (int b = __ldg(tile_start) + blockIdx.x; b < total; b += gridDim.x) {
        const int k = batch_run_of(tile_start, n, b);
        const RunArgs& a = args[k];
        const int t = b - __ldg(tile_start + k);
        const int tx = (a.W + blockDim.x - 1) / blockDim.x;
        if (a.prm.mode & HPM_MODE_GEOM) __syncthreads();  // the tile before may still read its views
        const GeomView* views = load_geom_views<NS, BLK>(a, smem, tid);
        sweep_pixel<NS, BLK, MAND, CNT>(a, smem + tid, views, (t % tx) * blockDim.x + threadIdx.x,
                                        (t / tx) * blockDim.y + threadIdx.y, color, iter);
    }
}

#ifndef HPM_NS
__global__ void k_export(const __grid_constant__ RunArgs a) {
    const int px = blockIdx.x * blockDim.x + threadIdx.x;
    const int py = blockIdx.y * blockDim.y + threadIdx.y;
    if (px >= a.W || py >= a.H) return;
    const int center = py * a.W + px;
    float4 pl = a.planes[center];
    pl.w = depth_from_plane(a.cams[0], pl, px, py);
    a.planes[center] = rotate_to_world(a.cams[0], pl);
}

// Thread x of grid row y costs pixel x against the views y, y + gridDim.y, ...  Three blocks to an SM: at
// the 183 registers of two, 100,000 pixels x 10 views took 614 us a call, with three 577.
__global__ void __launch_bounds__(kEvalThreads, kSweepBlocks)
    k_eval_costs(const __grid_constant__ RunArgs a, int n, const int32_t* __restrict__ px,
                 const float4* __restrict__ planes, float* __restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int x = px[2 * k], y = px[2 * k + 1];
    Patch P;
    build_patch<true>(a, x, y, P, nullptr);
    const float4 pl = planes[k];
    const PlaneM pm = plane_m(a, pl);
    for (int j = blockIdx.y; j < a.S; j += gridDim.y) out[(size_t)k * a.S + j] = ncc_view<false>(a, P, x, y, pm, j);
}
#endif

// ---------------------------------------------------------------- launchers

#ifndef HPM_NS
cudaError_t launch_weight_table(const hpm_params& prm, float* out, cudaStream_t st) {
    const float two_ss = 2.0f * prm.sigma_spatial * prm.sigma_spatial;
    const float two_sc = 2.0f * prm.sigma_color * prm.sigma_color;
    k_weight_table<<<kWeightRows, 256, 0, st>>>(two_ss, two_sc, out);
    return cudaGetLastError();
}
#endif

template <int NS, bool CNT>
cudaError_t init_impl(const RunArgs& a, cudaStream_t st) {
    constexpr int BLK = 128;
    const size_t shm = sizeof(float) * InitScratch<NS, BLK>::kWords * BLK;
    auto k = k_random_init<NS, BLK, CNT>;
    dim3 block(32, 4), grid((a.W + 31) / 32, (a.H + 3) / 4);
    k<<<grid, block, shm, st>>>(a);
    return cudaGetLastError();
}

template <int NS>
static constexpr size_t sweep_smem() {
    return sizeof(float) * Scratch<NS, kSweepThreads>::kWords * kSweepThreads + sizeof(GeomView) * NS;
}

static int blocks_of_four(const RunArgs& a) { return (a.W + 31) / 32 * ((a.cover_pairs + 3) / 4); }

static bool one_wave(int blocks) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return false;
    return blocks < kSweepBlocks * sms;
}

// Row pairs of a block, one warp each.  An image of less than one wave of four-warp blocks runs in
// two-warp blocks, which spread over the SMs more evenly: 320x240 has 320 blocks of four warps for
// 3 x 148 places, and its half-sweeps take 142 instead of 155 us (photometric, 4 sources), 297 instead
// of 313 (prior, 10 sources).  From 400x300 on (520 blocks) four warps are as fast or faster, since the
// warps of a block share what they fetch.
static int block_pairs(const RunArgs& a) { return one_wave(blocks_of_four(a)) ? 2 : 4; }

template <int NS, bool MAND, bool CNT>
cudaError_t sweep_impl(const RunArgs& a, int color, int iter, int first_pair, int last_pair, cudaStream_t st) {
    constexpr int BLK = kSweepThreads, BX = 32;
    const int across = (a.W + BX - 1) / BX;
    const int pairs = block_pairs(a);
    const dim3 block(BX, pairs), grid(across, (last_pair - first_pair + pairs - 1) / pairs);
    if (!MAND && a.active_px)
        k_half_sweep_listed<NS, BLK, CNT><<<grid, block, sweep_smem<NS>(), st>>>(a, color, iter, first_pair, last_pair);
    else
        k_half_sweep<NS, BLK, MAND, CNT><<<grid, block, sweep_smem<NS>(), st>>>(a, color, iter, first_pair, last_pair);
    return cudaGetLastError();
}

template <int NS, bool CNT>
cudaError_t init_batch_impl(const BatchLaunch& bl, cudaStream_t st) {
    constexpr int BLK = 128;
    const size_t shm = sizeof(float) * InitScratch<NS, BLK>::kWords * BLK;
    auto k = k_random_init_batch<NS, BLK, CNT>;
    const int grid = bl.grid_blocks > 0 && bl.grid_blocks < bl.tiles ? bl.grid_blocks : bl.tiles;
    k<<<grid, dim3(16, 8), shm, st>>>(bl.args, bl.tile_start, bl.n);
    return cudaGetLastError();
}

template <int NS, bool MAND, bool CNT>
cudaError_t sweep_batch_impl(const BatchLaunch& bl, int color, int iter, cudaStream_t st) {
    constexpr int BLK = kSweepThreads;
    auto k = (!MAND && bl.listed) ? k_half_sweep_batch_listed<NS, BLK, CNT>
                                  : k_half_sweep_batch<NS, BLK, MAND, CNT>;
    const int grid = bl.grid_blocks > 0 && bl.grid_blocks < bl.tiles ? bl.grid_blocks : bl.tiles;
    const int bx = (bl.bx > 0 && bl.bx <= BLK) ? bl.bx : 32;
    k<<<grid, dim3(bx, BLK / bx), sweep_smem<NS>(), st>>>(bl.args, bl.tile_start, bl.n, color, iter);
    return cudaGetLastError();
}

template <int NS, bool MAND>
int sweep_batch_occupancy() {
    constexpr int BLK = kSweepThreads;
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_half_sweep_batch<NS, BLK, MAND, false>, BLK,
                                                      sweep_smem<NS>()) != cudaSuccess)
        return 0;
    return blocks;
}

// The kernels are compiled once per source count they are specialised for, each in an object of its own
// (-DHPM_NS=4, 10, 16, 31); the object without HPM_NS holds the dispatch.
#define HPM_SWEEP_FORMS(linkage, NS)                                                        \
    linkage template cudaError_t init_impl<NS, false>(const RunArgs&, cudaStream_t);        \
    linkage template cudaError_t init_impl<NS, true>(const RunArgs&, cudaStream_t);         \
    linkage template cudaError_t init_batch_impl<NS, false>(const BatchLaunch&, cudaStream_t); \
    linkage template cudaError_t init_batch_impl<NS, true>(const BatchLaunch&, cudaStream_t);  \
    HPM_SWEEP_FORMS_OF(linkage, NS, false, false)                                           \
    HPM_SWEEP_FORMS_OF(linkage, NS, false, true)                                            \
    HPM_SWEEP_FORMS_OF(linkage, NS, true, false)                                            \
    HPM_SWEEP_FORMS_OF(linkage, NS, true, true)                                             \
    linkage template int sweep_batch_occupancy<NS, false>();                                \
    linkage template int sweep_batch_occupancy<NS, true>();
#define HPM_SWEEP_FORMS_OF(linkage, NS, MAND, CNT)                                                     \
    linkage template cudaError_t sweep_impl<NS, MAND, CNT>(const RunArgs&, int, int, int, int, cudaStream_t);    \
    linkage template cudaError_t sweep_batch_impl<NS, MAND, CNT>(const BatchLaunch&, int, int, cudaStream_t);

#ifdef HPM_NS
HPM_SWEEP_FORMS(, HPM_NS)
#else
HPM_SWEEP_FORMS(extern, 4)
HPM_SWEEP_FORMS(extern, 10)
HPM_SWEEP_FORMS(extern, 16)
HPM_SWEEP_FORMS(extern, 31)

// The kernel specialisation of a run: the source count rounded up to 4, 10, 16 or 31.
#define HPM_BY_SOURCES(s, fn, ...) \
    ((s) <= 4 ? fn<4, __VA_ARGS__>  \
              : (s) <= 10 ? fn<10, __VA_ARGS__> : (s) <= 16 ? fn<16, __VA_ARGS__> : fn<31, __VA_ARGS__>)

cudaError_t launch_random_init(const RunArgs& a, cudaStream_t st) {
    return a.hyp_count ? HPM_BY_SOURCES(a.S, init_impl, true)(a, st) : HPM_BY_SOURCES(a.S, init_impl, false)(a, st);
}

cudaError_t launch_half_sweep(const RunArgs& a, int color, int iter, int first_pair, int last_pair, cudaStream_t st) {
    const bool mand = a.prm.mode & HPM_MODE_MAND;
    if (last_pair <= first_pair) return cudaSuccess;
    if (a.hyp_count)
        return mand ? HPM_BY_SOURCES(a.S, sweep_impl, true, true)(a, color, iter, first_pair, last_pair, st)
                    : HPM_BY_SOURCES(a.S, sweep_impl, false, true)(a, color, iter, first_pair, last_pair, st);
    return mand ? HPM_BY_SOURCES(a.S, sweep_impl, true, false)(a, color, iter, first_pair, last_pair, st)
                : HPM_BY_SOURCES(a.S, sweep_impl, false, false)(a, color, iter, first_pair, last_pair, st);
}

cudaError_t launch_random_init_batch(const BatchLaunch& bl, cudaStream_t st) {
    return bl.count ? HPM_BY_SOURCES(bl.max_s, init_batch_impl, true)(bl, st)
                    : HPM_BY_SOURCES(bl.max_s, init_batch_impl, false)(bl, st);
}

cudaError_t launch_half_sweep_batch(const BatchLaunch& bl, int color, int iter, cudaStream_t st) {
    if (bl.count)
        return bl.mand ? HPM_BY_SOURCES(bl.max_s, sweep_batch_impl, true, true)(bl, color, iter, st)
                       : HPM_BY_SOURCES(bl.max_s, sweep_batch_impl, false, true)(bl, color, iter, st);
    return bl.mand ? HPM_BY_SOURCES(bl.max_s, sweep_batch_impl, true, false)(bl, color, iter, st)
                   : HPM_BY_SOURCES(bl.max_s, sweep_batch_impl, false, false)(bl, color, iter, st);
}

int half_sweep_batch_occupancy(int max_s, bool mand) {
    return mand ? HPM_BY_SOURCES(max_s, sweep_batch_occupancy, true)() : HPM_BY_SOURCES(max_s, sweep_batch_occupancy, false)();
}

bool half_sweep_one_wave(const RunArgs& a) { return one_wave(blocks_of_four(a)); }
int half_sweep_block_threads() { return kSweepThreads; }

cudaError_t launch_export(const RunArgs& a, cudaStream_t st) {
    dim3 block(32, 8), grid((a.W + 31) / 32, (a.H + 7) / 8);
    k_export<<<grid, block, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_eval_costs(const RunArgs& a, int n, const int32_t* px, const float4* planes, float* out,
                              cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    // A thread per pixel and view while they are resident together: one after the other, 31 views of one
    // pixel took 78 us a call and take 41, of 64 pixels 92 and 54.  Past that a thread goes through its
    // pixel's views, which share the patch (100,000 pixels x 31 views: 1200 us).
    const int blocks = (n + kEvalThreads - 1) / kEvalThreads;
    const bool apart = one_wave(blocks <= INT_MAX / HPM_MAX_SRC ? blocks * a.S : blocks);
    k_eval_costs<<<dim3(blocks, apart ? a.S : 1), kEvalThreads, 0, st>>>(a, n, px, planes, out);
    return cudaGetLastError();
}

#endif  // HPM_NS

}  // namespace hpm
