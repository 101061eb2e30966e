// PatchMatch run orchestration behind hpm_run_patchmatch / hpm_eval_costs:
// the device-resident replacement of HPM::CudaSpaceInitialization's reloads
// (HPM.cpp:741-906, 942-984), HPM::RunPatchMatch (HPM.cu:2987-3035) and the
// result hand-off of ProcessProblem (main.cpp:599-626).
#include "ctx.hpp"

#include <cuda_fp16.h>
#include "hpm_geometry.h"
#include "pm_kernels.cuh"
#include "aux_kernels.cuh"

#include <algorithm>
#include <cstring>

namespace hpm {

__global__ void k_pack_planes(const float* __restrict__ normal, const float* __restrict__ depth,
                              float4* __restrict__ planes, const float* __restrict__ cost_in,
                              float* __restrict__ cost_out, int n);
__global__ void k_pack_scaled(const float* __restrict__ normal, const float* __restrict__ w_src,
                              float4* __restrict__ out, int n);
__global__ void k_unpack_planes(const float4* __restrict__ planes, float* __restrict__ depth,
                                float* __restrict__ normal, int n);

template <class T>
static cudaError_t ensure_buf(T*& p, size_t& cap, size_t n) {
    if (n <= cap && p) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
    cudaError_t e = cudaMalloc((void**)&p, std::max<size_t>(n, 1) * sizeof(T));
    if (e == cudaSuccess) cap = n;
    return e;
}

__global__ void k_to_half(const float* __restrict__ src, int n, uint16_t* __restrict__ dst) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = __half_as_ushort(__float2half_rn(src[i]));
}

__global__ void k_to_u8(const float* __restrict__ src, int n, uint8_t* __restrict__ dst) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = (uint8_t)fminf(255.0f, fmaxf(0.0f, rintf(src[i])));
}

// Images for Ctx::bring_bytes, one to a grid row.
struct ByteCopies {
    const float* gray[HPM_MAX_SRC + 1];
    uint8_t* bytes[HPM_MAX_SRC + 1];
    int* whole[HPM_MAX_SRC + 1];  // cleared where a level is not a whole number 0..255; null: known to be
    int n[HPM_MAX_SRC + 1];
};

__global__ void k_bytes(const __grid_constant__ ByteCopies c) {
    const float* __restrict__ gray = c.gray[blockIdx.y];
    uint8_t* __restrict__ bytes = c.bytes[blockIdx.y];
    int* whole = c.whole[blockIdx.y];
    const int n = c.n[blockIdx.y];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float v = gray[i];
        if (whole && !(v >= 0.0f && v <= 255.0f && v == rintf(v))) *whole = 0;
        bytes[i] = (uint8_t)fminf(255.0f, fmaxf(0.0f, rintf(v)));
    }
}

bool Ctx::capturing() const {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone;
}

// A view's grey image has been replaced by one whose levels are whole (1) or not looked at (-1).  Once a
// capture holds such an upload, a replay may bring another image at any time without a call that the host
// sees, so the view stays on its float image (0), which every replay brings up to date.
void Ctx::new_image(int view, int whole_levels) {
    ViewState& v = views[view];
    v.captured = v.captured || capturing();
    v.whole_levels = v.captured ? 0 : whole_levels;
    v.bytes_current = v.bytes_bound = false;
    v.bytes_credit = 0;
}

static cudaError_t make_texture(cudaArray_t arr, int addr_mode, cudaTextureReadMode read, cudaTextureObject_t* tex) {
    cudaResourceDesc rd;
    memset(&rd, 0, sizeof(rd));
    rd.resType = cudaResourceTypeArray;
    rd.res.array.array = arr;
    cudaTextureDesc td;
    memset(&td, 0, sizeof(td));
    td.addressMode[0] = td.addressMode[1] = addr_mode == 1 ? cudaAddressModeWrap : cudaAddressModeClamp;
    td.filterMode = cudaFilterModeLinear;
    td.readMode = read;
    td.normalizedCoords = 0;
    return cudaCreateTextureObject(tex, &rd, &td, nullptr);
}

// 8-bit copies of a run's images of whole levels 0..255: bytes of the reference, and 8-bit textures of the
// sources that have float ones.  hpm_prepare_level makes them with the level's image; images from
// hpm_set_view are looked at once, for which the host waits.  The unit filters with weights of 1/256, so an F32
// fetch is a whole multiple N of 1/256 level, N <= 255 * 256, and an 8-bit fetch is N / 65280 rounded
// to a multiple of 1/65535: fetch * 65280 lies within 0.4999 of N, and rounding it to the nearest
// integer gives N, hence the F32 fetch times 256, for every N (tests/test_gpu_whole_levels.py).  A
// quarter of the bytes puts neighbouring samples of a warp on fewer lines.
//
// Not under stream capture: a replay reads the images of its time.  Not before the reference's runs have
// work for it either.  With S sources on B200, the copies take about 20 + 5.5 (S + 1) us and save a half-sweep
// 9 + 1.6 S us of its latency and (2 + S) / 16 ns a pixel, the initialisation 0.2 ns a pixel (0.125 here: an
// image with other levels gains nothing).  Runs on new images, float and bytes: 64x48, S = 2, one iteration
// 263 and 267 us, three 559 and 519; 160x120, S = 10, one iteration 762 and 715; 640x480, S = 10, none 1223
// and 1236, three 9.5 and 7.5 ms.
int Ctx::bring_bytes(int ref, const int32_t* srcs, int n_src, int n_half_sweeps) {
    if (capturing()) return HPM_OK;
    int todo[HPM_MAX_SRC + 1], n_todo = 0, n_copies = 0, max_px = 0;
    for (int j = -1; j < n_src; ++j) {
        const int view = j < 0 ? ref : srcs[j];
        const ViewState& v = views[view];
        if (v.whole_levels == 0 || (j >= 0 && v.arr_fmt != HPM_TEX_F32)) continue;
        if (v.bytes_current && (j < 0 || v.bytes_bound)) continue;
        if (std::find(todo, todo + n_todo, view) == todo + n_todo) todo[n_todo++] = view;
    }
    if (!n_todo) return HPM_OK;
    ViewState& rv = views[ref];
    const int64_t px = (int64_t)rv.w * rv.h;
    rv.bytes_credit += n_half_sweeps * (9000 + 1600 * n_src + px * (2 + n_src) / 16) + px / 8;  // in ns
    if (rv.bytes_credit <= 20000 + 5500 * n_todo) return HPM_OK;

    ByteCopies c;
    bool unknown = false;
    cudaError_t e = ensure_buf(level_flags, level_flags_cap, HPM_MAX_VIEWS);
    if (e != cudaSuccess) return cuda_fail(e, "alloc level flags");
    for (int k = 0; k < n_todo; ++k) {
        ViewState& v = views[todo[k]];
        if (v.bytes_current) continue;
        if (ensure_buf(v.bytes, v.bytes_cap, (size_t)v.w * v.h) != cudaSuccess) {
            no_bytes(todo[k]);
            continue;
        }
        c.gray[n_copies] = v.gray;
        c.bytes[n_copies] = v.bytes;
        c.n[n_copies] = v.w * v.h;
        c.whole[n_copies] = v.whole_levels < 0 ? level_flags + todo[k] : nullptr;
        unknown = unknown || v.whole_levels < 0;
        max_px = std::max(max_px, c.n[n_copies++]);
    }
    int flags[HPM_MAX_VIEWS];
    if (unknown && (e = cudaMemsetAsync(level_flags, 0xff, sizeof(flags), stream)) != cudaSuccess)
        return cuda_fail(e, "grey levels");
    if (n_copies) {
        k_bytes<<<dim3(std::min((max_px + 255) / 256, 1184), n_copies), 256, 0, stream>>>(c);
        ++launches;
    }
    if (unknown) {
        e = cudaMemcpyAsync(flags, level_flags, sizeof(flags), cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        if (e != cudaSuccess) return cuda_fail(e, "grey levels");
    }
    for (int k = 0; k < n_todo; ++k) {
        ViewState& v = views[todo[k]];
        if (v.whole_levels < 0) v.whole_levels = flags[todo[k]] ? 1 : 0;
        v.bytes_current = v.whole_levels == 1;
    }
    for (int j = 0; j < n_src; ++j) {
        const ViewState& v = views[srcs[j]];
        if (!v.bytes_current || v.bytes_bound || v.arr_fmt != HPM_TEX_F32) continue;
        const int rc = bind_bytes(srcs[j]);
        if (rc) return rc;
    }
    return HPM_OK;
}

// Where there is no memory for a copy, the view stays on its float image.
int Ctx::no_bytes(int view) {
    cudaGetLastError();
    ViewState& v = views[view];
    v.whole_levels = 0;
    v.bytes_current = v.bytes_bound = false;
    return HPM_OK;
}

// The 8-bit texture of a view whose bytes are current.
int Ctx::bind_bytes(int view) {
    ViewState& v = views[view];
    cudaError_t e = cudaSuccess;
    ByteArray* b = v.arr8;
    for (auto& other : v.arr8) {  // the one of this size, or the longest unused
        if (other.arr && other.w == v.w && other.h == v.h) { b = &other; break; }
        if (other.used < b->used) b = &other;
    }
    const bool sized = b->arr && b->w == v.w && b->h == v.h;
    if (b->tex && (!sized || b->mode != v.arr_mode)) {
        if ((e = cudaStreamSynchronize(stream)) != cudaSuccess) return cuda_fail(e, "byte image");  // runs may sample it
        cudaDestroyTextureObject(b->tex);
        b->tex = 0;
    }
    if (!sized) {
        if (b->arr) cudaFreeArray(b->arr);
        b->arr = nullptr;
        const cudaChannelFormatDesc fd = cudaCreateChannelDesc(8, 0, 0, 0, cudaChannelFormatKindUnsigned);
        if (cudaMallocArray(&b->arr, &fd, v.w, v.h) != cudaSuccess) {
            b->arr = nullptr;
            return no_bytes(view);
        }
        b->w = v.w; b->h = v.h;
    }
    if (!b->tex) {
        if (make_texture(b->arr, v.arr_mode, cudaReadModeNormalizedFloat, &b->tex) != cudaSuccess) {
            b->tex = 0;
            return no_bytes(view);
        }
        b->mode = v.arr_mode;
    }
    e = cudaMemcpy2DToArrayAsync(b->arr, 0, 0, v.bytes, (size_t)v.w, (size_t)v.w, v.h, cudaMemcpyDeviceToDevice, stream);
    if (e != cudaSuccess) return cuda_fail(e, "copy byte image to array");
    b->used = ++v.arr8_uses;
    v.tex8 = b->tex;
    v.bytes_bound = true;
    return HPM_OK;
}

int Ctx::bind_texture(int view) {
    ViewState& v = views[view];
    cudaError_t e;
    if (!v.arr || v.arr_w != v.w || v.arr_h != v.h || v.arr_mode != addr_mode || v.arr_fmt != tex_format) {
        if (v.tex) { cudaDestroyTextureObject(v.tex); v.tex = 0; }
        if (v.arr && (v.arr_w != v.w || v.arr_h != v.h || v.arr_fmt != tex_format)) {
            cudaFreeArray(v.arr);
            v.arr = nullptr;
        }
        if (!v.arr) {
            // float texels, or half texels: the 0..255 grey levels are exact, the filtered sample is
            // returned rounded to half precision
            cudaChannelFormatDesc fd = tex_format == HPM_TEX_F16
                                           ? cudaCreateChannelDesc(16, 0, 0, 0, cudaChannelFormatKindFloat)
                                           : (tex_format == HPM_TEX_U8
                                                  ? cudaCreateChannelDesc(8, 0, 0, 0, cudaChannelFormatKindUnsigned)
                                                  : cudaCreateChannelDesc(32, 0, 0, 0, cudaChannelFormatKindFloat));
            e = cudaMallocArray(&v.arr, &fd, v.w, v.h);
            if (e != cudaSuccess) return cuda_fail(e, "alloc image array");
            v.arr_w = v.w; v.arr_h = v.h;
            v.arr_fmt = tex_format;
        }
        e = make_texture(v.arr, addr_mode,
                         tex_format == HPM_TEX_U8 ? cudaReadModeNormalizedFloat : cudaReadModeElementType, &v.tex);
        if (e != cudaSuccess) return cuda_fail(e, "create texture");
        v.arr_mode = addr_mode;
    }
    if (tex_format == HPM_TEX_F16) {
        const size_t n = (size_t)v.w * v.h;
        e = ensure_buf(half_stage, half_stage_cap, n);
        if (e != cudaSuccess) return cuda_fail(e, "alloc half staging");
        k_to_half<<<(int)((n + 255) / 256), 256, 0, stream>>>(v.gray, (int)n, half_stage);
        ++launches;
        e = cudaMemcpy2DToArrayAsync(v.arr, 0, 0, half_stage, 2 * (size_t)v.w, 2 * (size_t)v.w, v.h,
                                     cudaMemcpyDeviceToDevice, stream);
    } else if (tex_format == HPM_TEX_U8) {
        const size_t n = (size_t)v.w * v.h;
        e = ensure_buf(half_stage, half_stage_cap, n);  // n bytes fit in the n half words
        if (e != cudaSuccess) return cuda_fail(e, "alloc byte staging");
        uint8_t* bytes = reinterpret_cast<uint8_t*>(half_stage);
        k_to_u8<<<(int)((n + 255) / 256), 256, 0, stream>>>(v.gray, (int)n, bytes);
        ++launches;
        e = cudaMemcpy2DToArrayAsync(v.arr, 0, 0, bytes, (size_t)v.w, (size_t)v.w, v.h, cudaMemcpyDeviceToDevice,
                                     stream);
    } else {
        e = cudaMemcpy2DToArrayAsync(v.arr, 0, 0, v.gray, sizeof(float) * v.w, sizeof(float) * v.w, v.h,
                                     cudaMemcpyDeviceToDevice, stream);
    }
    if (e != cudaSuccess) return cuda_fail(e, "copy image to array");
    return HPM_OK;
}

int Ctx::fill_run_args(int ref, const int32_t* srcs, int n_src, const hpm_params* params, RunArgs& a) {
    if (!params) return fail(HPM_E_INVALID, "null params");
    if (ref < 0 || ref >= HPM_MAX_VIEWS || views[ref].w == 0) return fail(HPM_E_STATE, "reference view %d not set", ref);
    if (n_src < 1 || n_src > HPM_MAX_SRC || !srcs) return fail(HPM_E_INVALID, "need 1..31 source views, got %d", n_src);
    if (params->patch_size != 11 || params->radius_increment != 2)
        return fail(HPM_E_INVALID, "patch_size 11 / radius_increment 2 required (got %d / %d)", params->patch_size,
                    params->radius_increment);
    if (params->num_images != n_src + 1)
        return fail(HPM_E_INVALID, "params.num_images (%d) != n_src + 1 (%d)", params->num_images, n_src + 1);
    memset(&a, 0, sizeof(a));
    const ViewState& rv = views[ref];
    a.cams[0] = rv.cam;
    for (int j = 0; j < n_src; ++j) {
        const int s = srcs[j];
        if (s < 0 || s >= HPM_MAX_VIEWS || views[s].w == 0) return fail(HPM_E_STATE, "source view %d not set", s);
        a.cams[j + 1] = views[s].cam;
        a.tex[j + 1] = views[s].tex;
        hpm_view_basis(&rv.cam, &views[s].cam, a.basis[j + 1].A, a.basis[j + 1].b);
        hpm_view_transfer(&rv.cam, &views[s].cam, a.fwd[j + 1].A, a.fwd[j + 1].b);
        hpm_view_transfer(&views[s].cam, &rv.cam, a.bwd[j + 1].A, a.bwd[j + 1].b);
    }
    hpm_ref_kinv(&rv.cam, a.kinv);
    // 8-bit textures return grey / 255; the NCC is scale-free, only the flat-source test scales
    a.var_s_min = tex_format == HPM_TEX_U8 ? 1e-5f / (255.0f * 255.0f) : 1e-5f;
    a.ncc_shift = ncc_mode == HPM_NCC_SHIFTED ? 1 : 0;
    a.tex_scale = 1.0f;
    a.ref_img = rv.gray;
    a.prm = *params;
    a.S = n_src;
    a.W = rv.w;
    a.H = rv.h;
    a.cover_pairs = covered_row_pairs(rv.h);
    a.view_id = (uint32_t)ref;
    a.hyp_count = (prof_flags & HPM_PROFILE_COUNT) ? prof_hyp : nullptr;
    return HPM_OK;
}

int Ctx::prepare_run(int ref, const int32_t* srcs, int n_src, const hpm_params* params, int texture_level,
                     uint64_t seed, RunArgs& a) {
    cudaSetDevice(device);
    if (ref < 0 || ref >= HPM_MAX_VIEWS || views[ref].w == 0) return fail(HPM_E_STATE, "reference view %d not set", ref);
    cudaError_t e = ensure_run((size_t)views[ref].w * views[ref].h);
    if (e != cudaSuccess) return cuda_fail(e, "alloc run buffers");
    RunBufs b;
    b.planes = planes; b.costs = costs; b.pre_costs = pre_costs; b.sel = sel; b.rng = rng; b.conf = conf;
    const int rc = prepare_run_into(ref, srcs, n_src, params, texture_level, seed, b, a);
    if (rc) return rc;
    return take_whole_levels(ref, srcs, weights, a);
}

// The hypothesis reload and run setup of one run (HPM.cpp:741-906, 942-984)
// into the run buffers `b`: fills `a` and issues the per-run copies and packing
// kernels on the context's stream.
int Ctx::prepare_run_into(int ref, const int32_t* srcs, int n_src, const hpm_params* params, int texture_level,
                          uint64_t seed, const RunBufs& b, RunArgs& a) {
    int rc = fill_run_args(ref, srcs, n_src, params, a);
    if (rc) return rc;
    if (texture_level < 0 || texture_level >= 8) return fail(HPM_E_INVALID, "texture_level must be 0..7");
    ViewState& rv = views[ref];
    const int W = rv.w, H = rv.h;
    const int n = W * H;
    const uint32_t mode = params->mode;
    const bool geom = mode & HPM_MODE_GEOM, prior = mode & HPM_MODE_PRIOR, hier = mode & HPM_MODE_HIERARCHY;
    const bool mand = mode & HPM_MODE_MAND, multi = mode & HPM_MODE_MULTIGEOM;
    if (mand && !geom) return fail(HPM_E_INVALID, "mandatory consistency requires the geometric mode");
    if (hier && geom && !prior)  // each would start the pixels from its own maps
        return fail(HPM_E_INVALID, "the hierarchy mode and the geometric mode exclude each other");
    if (!rv.canny || rv.canny_w != W || rv.canny_h != H) return fail(HPM_E_STATE, "view %d has no Canny map of its size", ref);
    cudaError_t e;
    float4* const planes = b.planes;
    float* const costs = b.costs;
    float* const conf = b.conf;
    a.seed = seed;
    a.planes = b.planes; a.costs = b.costs; a.pre_costs = b.pre_costs; a.sel = b.sel; a.rng = b.rng; a.conf = b.conf;
    a.canny = rv.canny;
    // selected_views starts at zero at every run (fresh allocation in the reference, HPM.cpp:782)
    e = cudaMemsetAsync(b.sel, 0, sizeof(uint32_t) * n, stream);
    if (e != cudaSuccess) return cuda_fail(e, "clear view masks");
    const int blocks = (n + 255) / 256;
    const int depth_kind = multi ? HPM_MAP_DEPTH_GEOM : HPM_MAP_DEPTH;
    auto map_ok = [&](int v, int kind, int w, int h) {
        const DevMap& m = views[v].maps[kind];
        return m.ptr && m.w == w && m.h == h;
    };

    if (geom || prior) {
        // hypotheses reload: normals.dmb + depths(_geom).dmb + costs.dmb (HPM.cpp:813-846, 942-962)
        if (!map_ok(ref, depth_kind, W, H) || !map_ok(ref, HPM_MAP_NORMAL, W, H) || !map_ok(ref, HPM_MAP_COST, W, H))
            return fail(HPM_E_STATE, "view %d lacks depth/normal/cost maps of size %dx%d", ref, W, H);
        k_pack_planes<<<blocks, 256, 0, stream>>>(rv.maps[HPM_MAP_NORMAL].ptr, rv.maps[depth_kind].ptr, planes,
                                                   rv.maps[HPM_MAP_COST].ptr, costs, n);
        ++launches;
    }
    if (geom) {
        for (int j = 0; j < n_src; ++j) {
            const ViewState& sv = views[srcs[j]];
            const DevMap& m = sv.maps[depth_kind];
            if (!m.ptr || m.w <= 0) return fail(HPM_E_STATE, "source view %d lacks its depth map", srcs[j]);
            a.depth_src[j + 1] = m.ptr;
            a.dsw[j + 1] = m.w;
            a.dsh[j + 1] = m.h;
        }
    }
    if (prior || mand) {
        if (!map_ok(ref, HPM_MAP_CONF, W, H)) return fail(HPM_E_STATE, "view %d lacks a confidence map", ref);
        e = cudaMemcpyAsync(conf, rv.maps[HPM_MAP_CONF].ptr, sizeof(float) * n, cudaMemcpyDeviceToDevice, stream);
        if (e != cudaSuccess) return cuda_fail(e, "copy confidences");
    }
    if (prior) {
        if (!rv.prior || rv.prior_w != W || rv.prior_h != H) return fail(HPM_E_STATE, "view %d has no prior", ref);
        a.prior = rv.prior;
        a.pmask = rv.pmask;
    }
    if (hier && !geom && !prior) {
        // HPM.cpp:849-905: fine depth from JBU, coarse normals and costs
        const DevMap& dm = rv.maps[HPM_MAP_DEPTH];
        const DevMap& nm = rv.maps[HPM_MAP_NORMAL];
        const DevMap& cm = rv.maps[HPM_MAP_COST];
        if (!dm.ptr || dm.w != W || dm.h != H) return fail(HPM_E_STATE, "hierarchy: view %d depth map is not %dx%d", ref, W, H);
        if (!nm.ptr || !cm.ptr || cm.w != nm.w || cm.h != nm.h)
            return fail(HPM_E_STATE, "hierarchy: view %d lacks coarse normal/cost maps", ref);
        // the reference compares the map width with the image rows (HPM.cpp:869)
        const bool upsample = (nm.w != H || nm.h != W);
        if (!upsample && (nm.w != W || nm.h != H))
            return fail(HPM_E_STATE, "hierarchy: non-upsampled maps must match the image size");
        const int ns = nm.w * nm.h;
        float4* sc = b.scaled;
        if (!sc) {
            e = ensure_buf(scaled, scaled_cap, (size_t)ns);
            if (e != cudaSuccess) return cuda_fail(e, "alloc scaled map");
            sc = scaled;
        }
        k_pack_scaled<<<(ns + 255) / 256, 256, 0, stream>>>(nm.ptr, upsample ? cm.ptr : dm.ptr, sc, ns);
        k_pack_planes<<<blocks, 256, 0, stream>>>(nullptr, dm.ptr, planes, nullptr, nullptr, n);
        launches += 2;
        a.scaled = sc;
        a.prm.scaled_cols = nm.w;
        a.prm.scaled_rows = nm.h;
        if (upsample) a.prm.mode |= HPM_MODE_UPSAMPLE;
        else a.prm.mode &= ~HPM_MODE_UPSAMPLE;
    } else {
        a.prm.mode &= ~HPM_MODE_UPSAMPLE;
    }
    if ((rc = bring_bytes(ref, srcs, n_src, 2 * std::max(0, params->max_iterations)))) return rc;
    const bool want_texture = !prior && !mand;
    if (want_texture) {
        e = ensure_map(ref, HPM_MAP_TEXTURE0 + texture_level, W, H);
        if (e != cudaSuccess) return cuda_fail(e, "alloc texture map");
        a.texture = rv.maps[HPM_MAP_TEXTURE0 + texture_level].ptr;
    }

    return HPM_OK;
}

// What a run gains from images of whole levels: the reference's bytes and weight table (pm_kernels.cu,
// build_patch), and the sources' 8-bit textures when every source has one.  A captured run takes neither:
// its replays have to see images that hpm_set_view brings later, whatever their levels.
int Ctx::take_whole_levels(int ref, const int32_t* srcs, float* weights, RunArgs& a) {
    if (capturing()) return HPM_OK;
    if (views[ref].bytes_current) {
        cudaError_t e = launch_weight_table(a.prm, weights, stream);
        if (e != cudaSuccess) return cuda_fail(e, "weight table");
        ++launches;
        a.whole_levels = 1;
        a.ref_bytes = views[ref].bytes;
        a.weights = weights;
    }
    for (int j = 0; j < a.S; ++j)
        if (!views[srcs[j]].bytes_bound) return HPM_OK;
    // fetches become multiples of 1/256 level, the moments of the source grow by powers of two
    for (int j = 0; j < a.S; ++j) a.tex[j + 1] = views[srcs[j]].tex8;
    a.tex_scale = 65280.0f;
    a.tex_bias = 12582912.0f;
    a.var_s_min *= 65536.0f;
    return HPM_OK;
}

int Ctx::record_start(int kind, TimedLaunch*& slot) {
    slot = nullptr;
    if (!(prof_flags & HPM_PROFILE_TIMING)) return HPM_OK;
    if (prof_used == prof_events.size()) {
        TimedLaunch t{};
        cudaError_t e = cudaEventCreate(&t.start);
        if (e == cudaSuccess) e = cudaEventCreate(&t.stop);
        if (e != cudaSuccess) return cuda_fail(e, "profiling event");
        prof_events.push_back(t);
    }
    slot = &prof_events[prof_used++];
    slot->kind = kind;
    slot->launches = 1;
    cudaError_t e = cudaEventRecord(slot->start, stream);
    return e == cudaSuccess ? HPM_OK : cuda_fail(e, "profiling event record");
}

int Ctx::launch_schedule(const RunArgs& a0, int n_half_sweeps) {
    cudaError_t e;
    TimedLaunch* t = nullptr;
    int rc = record_start(0, t);
    if (rc) return rc;
    if ((e = launch_random_init(a0, stream)) != cudaSuccess) return cuda_fail(e, "init launch");
    if (t) cudaEventRecord(t->stop, stream);
    ++launches;
    RunArgs a = a0;
    const uint32_t mode = a0.prm.mode;
    if ((mode & HPM_MODE_PRIOR) && !(mode & HPM_MODE_MAND) && n_half_sweeps > 0) {
        // confidences and the prior mask do not change during a prior-mode run: the pixels its
        // half-sweeps update are listed once, after the initialisation
        const size_t rows = 2 * (size_t)a0.cover_pairs;
        if ((e = ensure_buf(active_px, active_px_cap, rows * a0.W)) != cudaSuccess ||
            (e = ensure_buf(active_n, active_n_cap, rows)) != cudaSuccess)
            return cuda_fail(e, "alloc prior work lists");
        if ((e = launch_prior_active(a0, active_px, active_n, stream)) != cudaSuccess)
            return cuda_fail(e, "prior work lists");
        ++launches;
        a.active_px = active_px;
        a.active_n = active_n;
    }
    return launch_sweeps(a, n_half_sweeps);
}

bool Ctx::ensure_bands() {
    cudaError_t e = cudaSuccess;
    if (band_start) return true;
    if (capturing()) return false;
    for (int b = 0; b < kBands && e == cudaSuccess; ++b) {
        if (b && !band_stream[b]) e = cudaStreamCreateWithFlags(&band_stream[b], cudaStreamNonBlocking);
        for (auto& parity : band_done)
            if (e == cudaSuccess && !parity[b]) e = cudaEventCreateWithFlags(&parity[b], cudaEventDisableTiming);
    }
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&band_start, cudaEventDisableTiming);
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess;
}

// The half-sweeps of a run.  A half-sweep reads the other colour's state up to 28 rows above (the path
// of the left-up extension's third round) and 13 below, and writes its own colour's, so a band of 28
// rows or more can start half-sweep k + 1 when it and its two neighbours have finished half-sweep k.
// With four bands on streams of their own, one half-sweep's last, partly filled wave runs beside the
// next one's first, which six launches in a row cannot.  One half-sweep on B200, 10 sources, one launch
// and in bands: photometric 400x300 (520 blocks, 444 places) 92 and 85 us, 800x600 (1900 blocks) 281 and
// 255, 1600x1200 (7600) 1106 and 1077; mandatory 259 and 231 at 800x600; prior 157 and 131.  Three to
// eight bands differ by less than 3 %.  An image of one wave has no such tail: bands cost 320x240 (320
// blocks) 4 %, so it keeps one launch, as does a context without streams to spare.
int Ctx::launch_sweeps(const RunArgs& a, int n_half_sweeps) {
    constexpr int kBandPairs = 16;  // shortest band, in row pairs
    static_assert(2 * kBandPairs >= 28, "a half-sweep reaches no further than the neighbouring bands");
    cudaError_t e = cudaSuccess;
    TimedLaunch* t = nullptr;
    int rc = HPM_OK;
    const int pairs = std::min(a.cover_pairs, (a.H + 1) / 2);
    int bands = std::min(kBands, pairs / kBandPairs);
    if (n_half_sweeps < 2 || bands < 2 || half_sweep_one_wave(a) || !ensure_bands()) {
        for (int k = 0; k < n_half_sweeps; ++k) {
            if ((rc = record_start(1, t))) return rc;
            if ((e = launch_half_sweep(a, k & 1, k >> 1, 0, a.cover_pairs, stream)) != cudaSuccess)
                return cuda_fail(e, "half sweep");
            if (t) cudaEventRecord(t->stop, stream);
            ++launches;
        }
        return HPM_OK;
    }
    if ((rc = record_start(1, t))) return rc;
    if (t) t->launches = n_half_sweeps;  // timed together
    // whole blocks of four row pairs to each band, and kBandPairs or more
    auto first = [&](int b) { return b == bands ? a.cover_pairs : pairs * b / bands / 4 * 4; };
    auto of = [&](int b) { return b ? band_stream[b] : stream; };
    if ((e = cudaEventRecord(band_start, stream)) != cudaSuccess) return cuda_fail(e, "band start");
    int joined = 1;  // bands whose stream has been tied to the run
    for (; joined < bands && e == cudaSuccess; ++joined) e = cudaStreamWaitEvent(band_stream[joined], band_start, 0);
    for (int k = 0; k < n_half_sweeps && e == cudaSuccess; ++k) {
        const auto& before = band_done[(k + 1) & 1];
        for (int b = 0; b < bands && e == cudaSuccess; ++b) {
            if (k && b > 0) e = cudaStreamWaitEvent(of(b), before[b - 1], 0);
            if (k && b + 1 < bands && e == cudaSuccess) e = cudaStreamWaitEvent(of(b), before[b + 1], 0);
            if (e == cudaSuccess) e = launch_half_sweep(a, k & 1, k >> 1, first(b), first(b + 1), of(b));
            ++launches;
        }
        for (int b = 0; b < bands && e == cudaSuccess; ++b) e = cudaEventRecord(band_done[k & 1][b], of(b));
    }
    for (int b = 1; b < bands && e == cudaSuccess; ++b)
        e = cudaStreamWaitEvent(stream, band_done[(n_half_sweeps - 1) & 1][b], 0);
    if (e != cudaSuccess) {  // the other streams' work ends before the context goes on
        for (int b = 1; b < joined; ++b) cudaStreamSynchronize(band_stream[b]);
        return cuda_fail(e, "half sweeps");
    }
    if (t) cudaEventRecord(t->stop, stream);
    return HPM_OK;
}

int Ctx::profile_read(hpm_profile* out) {
    cudaSetDevice(device);
    memset(out, 0, sizeof(*out));
    cudaError_t e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return cuda_fail(e, "profile read");
    for (size_t i = 0; i < prof_used; ++i) {
        float ms = 0.0f;
        e = cudaEventElapsedTime(&ms, prof_events[i].start, prof_events[i].stop);
        if (e != cudaSuccess) return cuda_fail(e, "profiling event time");
        switch (prof_events[i].kind) {
        case HPM_STAGE_INIT: out->init_launches++; out->init_ms += ms; break;
        case HPM_STAGE_SWEEP: out->sweep_launches += prof_events[i].launches; out->sweep_ms += ms; break;
        case HPM_STAGE_CONFIDENCE: out->confidence_ms += ms; break;
        case HPM_STAGE_PRIOR: out->prior_ms += ms; break;
        case HPM_STAGE_JBU: out->jbu_ms += ms; break;
        case HPM_STAGE_LEVEL: out->level_ms += ms; break;
        default: out->fusion_ms += ms; break;
        }
    }
    prof_used = 0;
    if (prof_hyp) {
        unsigned long long h[3] = {0, 0, 0};
        e = cudaMemcpy(h, prof_hyp, sizeof(h), cudaMemcpyDeviceToHost);
        if (e == cudaSuccess) e = cudaMemset(prof_hyp, 0, sizeof(h));
        if (e != cudaSuccess) return cuda_fail(e, "hypothesis counters");
        out->init_view_evals = h[0];
        out->sweep_view_evals = h[1];
        out->sweep_sampled = h[2];
    }
    return HPM_OK;
}

int Ctx::run_patchmatch(int ref, const int32_t* srcs, int n_src, const hpm_params* params, int texture_level,
                        uint64_t seed) {
    RunArgs a;
    int rc = prepare_run(ref, srcs, n_src, params, texture_level, seed, a);
    if (rc) return rc;
    rc = launch_schedule(a, 2 * params->max_iterations);
    if (rc) return rc;
    return finish_run(ref, a, params->mode & HPM_MODE_GEOM);
}

// GetDepthandNormal (HPM.cu:2829-2842) and the hand-off of the run's results to
// the view's resident maps (ProcessProblem, main.cpp:599-626).
int Ctx::finish_run(int ref, const RunArgs& a, bool geom) {
    cudaError_t e;
    if ((e = launch_export(a, stream)) != cudaSuccess) return cuda_fail(e, "export launch");
    ++launches;
    ViewState& rv = views[ref];
    const int W = rv.w, H = rv.h;
    const int n = W * H;
    const int blocks = (n + 255) / 256;
    const int out_depth = geom ? HPM_MAP_DEPTH_GEOM : HPM_MAP_DEPTH;
    if ((e = ensure_map(ref, out_depth, W, H)) != cudaSuccess) return cuda_fail(e, "alloc depth map");
    if ((e = ensure_map(ref, HPM_MAP_NORMAL, W, H)) != cudaSuccess) return cuda_fail(e, "alloc normal map");
    if ((e = ensure_map(ref, HPM_MAP_COST, W, H)) != cudaSuccess) return cuda_fail(e, "alloc cost map");
    k_unpack_planes<<<blocks, 256, 0, stream>>>(a.planes, rv.maps[out_depth].ptr, rv.maps[HPM_MAP_NORMAL].ptr, n);
    ++launches;
    e = cudaMemcpyAsync(rv.maps[HPM_MAP_COST].ptr, a.costs, sizeof(float) * n, cudaMemcpyDeviceToDevice, stream);
    if (e != cudaSuccess) return cuda_fail(e, "store costs");
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "patchmatch run");
    return HPM_OK;
}

int Ctx::debug_run_partial(int ref, const int32_t* srcs, int n_src, const hpm_params* params, int texture_level,
                           uint64_t seed, int n_half_sweeps, float* planes_out, float* costs_out, uint32_t* sel_out,
                           uint32_t* draws_out) {
    if (n_half_sweeps < 0 || n_half_sweeps > 64) return fail(HPM_E_INVALID, "n_half_sweeps must be 0..64");
    RunArgs a;
    int rc = prepare_run(ref, srcs, n_src, params, texture_level, seed, a);
    if (rc) return rc;
    rc = launch_schedule(a, n_half_sweeps);
    if (rc) return rc;
    const size_t n = (size_t)a.W * a.H;
    cudaError_t e = cudaSuccess;
    if (planes_out) e = cudaMemcpyAsync(planes_out, planes, n * sizeof(float4), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess && costs_out) e = cudaMemcpyAsync(costs_out, costs, n * 4, cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess && sel_out) e = cudaMemcpyAsync(sel_out, sel, n * 4, cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess && draws_out) e = cudaMemcpyAsync(draws_out, rng, n * 4, cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return cuda_fail(e, "download run state");
    return HPM_OK;
}

__global__ void k_sample_view(cudaTextureObject_t tex, int n, const float2* __restrict__ xy, float* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = tex2D<float>(tex, xy[i].x, xy[i].y);
}

int Ctx::sample_view(int view, int n, const float* xy, float* out) {
    cudaSetDevice(device);
    if (view < 0 || view >= HPM_MAX_VIEWS || views[view].w == 0) return fail(HPM_E_STATE, "view %d not set", view);
    if (n < 0 || (n > 0 && (!xy || !out))) return fail(HPM_E_INVALID, "hpm_sample_view: bad arguments");
    if (n == 0) return HPM_OK;
    cudaError_t e = ensure_buf(scratch, scratch_cap, (size_t)n * 12 + 64);
    if (e != cudaSuccess) return cuda_fail(e, "alloc scratch");
    float2* d_xy = reinterpret_cast<float2*>(scratch);
    float* d_out = reinterpret_cast<float*>(scratch + (size_t)n * 8);
    e = cudaMemcpyAsync(d_xy, xy, (size_t)n * 8, cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess) return cuda_fail(e, "upload coordinates");
    k_sample_view<<<(n + 255) / 256, 256, 0, stream>>>(views[view].tex, n, d_xy, d_out);
    ++launches;
    e = cudaMemcpyAsync(out, d_out, (size_t)n * 4, cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return cuda_fail(e, "download samples");
    return HPM_OK;
}

// RunJBU (HPM.cpp:1266-1319): the coarser depths_geom map of a view upsampled to
// the view's current image size into its depths map; nothing happens when the
// integer scale is 1 (HPM.cpp:1272-1275).
int Ctx::jbu_view(int view, int* applied) {
    cudaSetDevice(device);
    if (applied) *applied = 0;
    if (view < 0 || view >= HPM_MAX_VIEWS || views[view].w == 0) return fail(HPM_E_STATE, "view %d not set", view);
    ViewState& v = views[view];
    const DevMap& src = v.maps[HPM_MAP_DEPTH_GEOM];
    if (!src.ptr || src.w <= 0) return fail(HPM_E_STATE, "view %d has no depths_geom map", view);
    const int scale = std::max(v.h / src.h, v.w / src.w);
    if (scale == 1) return HPM_OK;
    if (src.w * 1LL * src.h > (long long)v.w * v.h) return fail(HPM_E_STATE, "JBU source larger than the image");
    // the source map must survive while the output is written: stage it in scratch
    const size_t ns = (size_t)src.w * src.h;
    cudaError_t e = ensure_buf(scratch, scratch_cap, ns * 4 + 256);
    if (e != cudaSuccess) return cuda_fail(e, "alloc scratch");
    float* d_src = reinterpret_cast<float*>(scratch);
    const int sw = src.w, sh = src.h;
    e = cudaMemcpyAsync(d_src, src.ptr, ns * 4, cudaMemcpyDeviceToDevice, stream);
    if (e != cudaSuccess) return cuda_fail(e, "stage JBU source");
    e = ensure_map(view, HPM_MAP_DEPTH, v.w, v.h);
    if (e != cudaSuccess) return cuda_fail(e, "alloc depth map");
    e = launch_jbu(v.gray, v.w, v.h, d_src, sw, sh, v.maps[HPM_MAP_DEPTH].ptr, stream);
    if (e != cudaSuccess) return cuda_fail(e, "JBU launch");
    ++launches;
    if (applied) *applied = 1;
    return HPM_OK;
}

cudaError_t Ctx::ensure_scratch(size_t bytes) { return ensure_buf(scratch, scratch_cap, bytes); }

int Ctx::eval_costs(int ref, const int32_t* srcs, int n_src, const hpm_params* params, int n, const int32_t* px,
                    const float* planes_h, float* out) {
    cudaSetDevice(device);
    if (n < 0 || (n > 0 && (!px || !planes_h || !out))) return fail(HPM_E_INVALID, "hpm_eval_costs: bad arguments");
    RunArgs a;
    int rc = fill_run_args(ref, srcs, n_src, params, a);
    if (rc) return rc;
    if (n == 0) return HPM_OK;
    for (int k = 0; k < n; ++k)
        if (px[2 * k] < 0 || px[2 * k] >= a.W || px[2 * k + 1] < 0 || px[2 * k + 1] >= a.H)
            return fail(HPM_E_INVALID, "pixel %d outside the reference image", k);
    const size_t bytes = (size_t)n * (8 + 16) + (size_t)n * n_src * 4 + 64;
    cudaError_t e = ensure_buf(scratch, scratch_cap, bytes);
    if (e != cudaSuccess) return cuda_fail(e, "alloc scratch");
    float4* d_planes = reinterpret_cast<float4*>(scratch);
    int32_t* d_px = reinterpret_cast<int32_t*>(scratch + (size_t)n * 16);
    float* d_out = reinterpret_cast<float*>(scratch + (size_t)n * 24);
    e = cudaMemcpyAsync(d_planes, planes_h, (size_t)n * 16, cudaMemcpyHostToDevice, stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_px, px, (size_t)n * 8, cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess) return cuda_fail(e, "upload hypotheses");
    if ((e = launch_eval_costs(a, n, d_px, d_planes, d_out, stream)) != cudaSuccess) return cuda_fail(e, "eval launch");
    ++launches;
    e = cudaMemcpyAsync(out, d_out, (size_t)n * n_src * 4, cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return cuda_fail(e, "download costs");
    return HPM_OK;
}

}  // namespace hpm
