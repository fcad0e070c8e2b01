// k_deferred.cu -- the deferred renderer: a march pass that records every
// contributing view sample, then shading passes that evaluate the sun term for
// those samples in full warps (exact cone, or the MLP surrogate) and
// accumulate each pixel's colour.
//
// Phase A (k_march): one thread per pixel, one warp per 8x4 pixel tile.  The
// warp marches its rays in lockstep over the view steps; at every step the
// lanes whose sample has alpha > 0 append (voxel position, w = T*alpha,
// light G, lane) to the warp's region of the sample buffer (capacity 32 *
// view_steps), in (step, lane) order.  The pixel's alpha 1 - T is final after
// this pass (one float per pixel; the shading passes write the RGBA image).
// Exact shading (k_shade_exact): one warp per region, 32 samples at a time,
// then each pixel sums its own samples in step order (shuffle broadcast),
// exactly the order of the fused kernel.
// MLP shading: the march also lays the samples out in a flat order (each
// CTA's MARCH_WARPS regions reserve one contiguous range, padded to whole 32-sample
// chunks); a persistent tensor-core kernel (k_shade_mlp_tc) walks that order
// in 128-sample tiles, computing features, running the network and writing
// each sample's contribution to the compact per-slot array; k_accumulate then
// sums each pixel's contributions in step order.
#include <algorithm>

#include "cg_internal.h"
#include "cg_mlp.cuh"
#include "cg_sample.cuh"

namespace {

// pixel of lane `lane` in region `region` (k_march's mapping)
__device__ __forceinline__ void region_pixel(int region, int lane, int tiles_x, int& px,
                                             int& py) {
    const int blk = region >> 3, w = region & 7;
    px = (blk % tiles_x) * 16 + (w & 1) * 8 + (lane & 7);
    py = (blk / tiles_x) * 16 + (w >> 1) * 4 + (lane >> 3);
}

__device__ __forceinline__ bool pixel_ray(const CamDesc& cam, const VolDesc& vd, int px, int py,
                                          float3& d, float& tin, float& tout) {
    float ndx = (2.f * ((float)px + 0.5f) / (float)cam.W - 1.f) * cam.tanh * cam.aspect;
    float ndy = (1.f - 2.f * ((float)py + 0.5f) / (float)cam.H) * cam.tanh;
    float dx = cam.f[0] + ndx * cam.s[0] + ndy * cam.u[0];
    float dy = cam.f[1] + ndx * cam.s[1] + ndy * cam.u[1];
    float dz = cam.f[2] + ndx * cam.s[2] + ndy * cam.u[2];
    float inv = rsqrtf(dx * dx + dy * dy + dz * dz);
    d = make_float3(dx * inv, dy * inv, dz * inv);
    float dd[3] = {d.x, d.y, d.z};
    float tmin = -1e30f, tmax = 1e30f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float lo = vd.wmin[a], hi = vd.wmin[a] + vd.range[a];
        if (dd[a] == 0.f) {
            if (cam.eye[a] < lo || cam.eye[a] > hi) return false;
            continue;
        }
        float iv = 1.f / dd[a];
        float t0 = (lo - cam.eye[a]) * iv, t1 = (hi - cam.eye[a]) * iv;
        tmin = fmaxf(tmin, fminf(t0, t1));
        tmax = fminf(tmax, fmaxf(t0, t1));
    }
    tin = fmaxf(tmin, 0.f);
    tout = tmax;
    return tout > tin;
}

// Warps per CTA (8 / MARCH_WARPS CTAs share a 16x16 pixel block): a CTA waits
// for its slowest warp before it lays out its samples, so smaller CTAs waste
// fewer warp slots (1080p surrogate march, us: 8 warps 113, 4 109, 2 108, 1 116).
constexpr int MARCH_WARPS = 4;
// Steps whose brick flags are fetched together in the surrogate's march (four
// 109 us, eight 107).
constexpr int MARCH_FLAGS = 8;

// HW: view samples and noise filtered by the texture unit (surrogate renderer).
template <int FMT, bool HW>
__global__ void __launch_bounds__(32 * MARCH_WARPS, 32 / MARCH_WARPS)
    k_march(VolDesc vd, CamDesc cam, TraceParams tp, SampleBuf sb, float4* dst,
            unsigned long long* status) {
    // the shading pass may be scheduled once every march CTA has started: its
    // CTAs stage their network while the last wave of the march runs (and read
    // the samples and the status only once the march has completed)
    grid_dep_trigger();
    if (HW && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 4) status[threadIdx.x] = 0ull;
    constexpr int SHARE = 8 / MARCH_WARPS;
    const int lane = threadIdx.x & 31;
    const int region = (int)((blockIdx.y * (gridDim.x / SHARE) + blockIdx.x / SHARE) * 8 +
                             (blockIdx.x % SHARE) * MARCH_WARPS + (threadIdx.x >> 5));
    int px, py;
    region_pixel(region, lane, (int)(gridDim.x / SHARE), px, py);
    const bool valid = px < cam.W && py < cam.H;
    float3 d = make_float3(0.f, 0.f, 0.f);
    float tin = 0.f, tout = 0.f;
    bool live = valid && pixel_ray(cam, vd, px, py, d, tin, tout);
    const int Nv = tp.view_steps;
    const float dt = (tout - tin) / (float)Nv;
    const float D = (float)vd.D;
    const float vsx = D / vd.range[0], vsy = D / vd.range[1], vsz = D / vd.range[2];
    const float pixk = cam.tanh / (float)cam.H * vsx;
    // the pixel cone spans less than one voxel before t_lod1: lod is exactly 0
    const float t_lod1 = 0.5f / pixk;
    float T = 1.f;
    unsigned cnt = 0, nsteps = 0;
    float4* pw = sb.pos_w + (size_t)region * sb.capacity;
    float2* gl = sb.light_lane + (size_t)region * sb.capacity;
    // this lane's sampled steps: when every sample has lod 0, steps outside the
    // occupied box read 0 and are skipped (the warp starts at its first one)
    int kb = 0, ke = Nv;
    const bool lod0 = tin + ((float)(Nv - 1) + 0.5f) * dt < t_lod1;
    if (live && lod0) {
        int k0, k1;
        cgs::occupied_steps(vd, cam.eye, d, tin, dt, Nv, k0, k1);
        kb = k0;
        ke = k1 + 1;
        if (kb >= ke) live = false;
    }
    const int wkb = __reduce_min_sync(0xffffffffu, live ? kb : Nv);
    // records the samples of one step (those of lanes with `emit`)
    auto record = [&](bool emit, float v0, float v1, float v2, float w, float G) {
        const unsigned ballot = __ballot_sync(0xffffffffu, emit);
        if (emit) {
            const unsigned slot = cnt + __popc(ballot & ((1u << lane) - 1u));
            if (CG_IN_BOUNDS((size_t)region * sb.capacity + slot, sb.nslots)) {
                pw[slot] = make_float4(v0, v1, v2, w);
                gl[slot] = make_float2(G, __int_as_float(lane));
            }
        }
        // step table: where this step's samples start and which lanes emitted
        if (ballot) {
            if (lane == 0) sb.steps[(size_t)region * Nv + nsteps] = make_uint2(cnt, ballot);
            nsteps++;
        }
        cnt += __popc(ballot);
        return ballot;
    };
    if (HW && __all_sync(0xffffffffu, !live || lod0)) {
        // Every live lane's samples have lod 0 (the common case): level 0 is
        // sampled directly.  The march waits for its loads (one step at a time:
        // flag, then density, then noise; long scoreboard 4.1 of 12 stall cycles
        // per issue, issue 66 %), so they go out together: the brick flags of
        // MARCH_FLAGS steps (their coordinates are linear in k, off by a
        // rounding at most, which a flag that also covers the neighbouring
        // bricks allows), then, for the steps at which some lane's flag is set,
        // both textures of two steps at a time.  256^3 at 1080p: 145 -> 107 us.
        const float o = tin + 0.5f * dt;
        const float v0a[3] = {(cam.eye[0] + o * d.x - vd.wmin[0]) * vsx,
                              (cam.eye[1] + o * d.y - vd.wmin[1]) * vsy,
                              (cam.eye[2] + o * d.z - vd.wmin[2]) * vsz};
        const float dva[3] = {dt * d.x * vsx, dt * d.y * vsy, dt * d.z * vsz};
        cgs::OccRay fine;
        fine.set(vd, 0, v0a, dva, (float)(1 << vd.occ_shift), -0.5f);
        struct Fetch {
            float v0, v1, v2, nz;
            float2 rg;
        };
        auto fetch = [&](int k, bool on, Fetch& f) {
            f.rg = make_float2(0.f, 0.f);
            f.v0 = f.v1 = f.v2 = f.nz = 0.f;
            if (!on) return;
            const float t = tin + ((float)k + 0.5f) * dt;
            const float p0 = cam.eye[0] + t * d.x, p1 = cam.eye[1] + t * d.y,
                        p2 = cam.eye[2] + t * d.z;
            f.v0 = (p0 - vd.wmin[0]) * vsx;
            f.v1 = (p1 - vd.wmin[1]) * vsy;
            f.v2 = (p2 - vd.wmin[2]) * vsz;
            f.rg = tex3D<float2>((cudaTextureObject_t)vd.tex[0], f.v0, f.v1, f.v2);
            f.nz = cgs::fbm_volume(tp, p0, p1, p2);
        };
        auto resolve = [&](const Fetch& f) {
            bool emit = false;
            float w = 0.f;
            const float rho = f.rg.x * f.nz;
            if (live && f.rg.x > 0.f && rho > 0.f) {
                const float alpha = 1.f - __expf(-tp.sigma * rho * dt);
                w = T * alpha;
                emit = true;
                T *= 1.f - alpha;
                if (T < tp.cutoff) live = false;
            }
            record(emit, f.v0, f.v1, f.v2, w, f.rg.y);
        };
        for (int k = wkb; k < Nv; k += MARCH_FLAGS) {
            if (live && k >= ke) live = false;
            if (!__any_sync(0xffffffffu, live)) break;
            unsigned m = 0u;
#pragma unroll
            for (int j = 0; j < MARCH_FLAGS; ++j)
                m |= (fine.at((float)(k + j)) && k + j >= kb && k + j < ke ? 1u : 0u) << j;
            if (!live) m = 0u;
            unsigned any = __reduce_or_sync(0xffffffffu, m);
            while (any) {
                const int j0 = __ffs(any) - 1;
                any &= any - 1u;
                const int j1 = any ? __ffs(any) - 1 : MARCH_FLAGS;
                any &= any - 1u;
                Fetch f0, f1;
                fetch(k + j0, (m >> j0) & 1u, f0);
                fetch(k + j1, (m >> j1) & 1u, f1);
                resolve(f0);
                if (j1 < MARCH_FLAGS) resolve(f1);
            }
        }
    } else {
        for (int k = wkb; k < Nv; ++k) {
            if (live && k >= ke) live = false;
            if (!__any_sync(0xffffffffu, live)) break;
            bool emit = false;
            float v0 = 0.f, v1 = 0.f, v2 = 0.f, w = 0.f, G = 0.f;
            if (live && k >= kb) {
                float t = tin + ((float)k + 0.5f) * dt;
                float p0 = cam.eye[0] + t * d.x, p1 = cam.eye[1] + t * d.y, p2 = cam.eye[2] + t * d.z;
                v0 = (p0 - vd.wmin[0]) * vsx;
                v1 = (p1 - vd.wmin[1]) * vsy;
                v2 = (p2 - vd.wmin[2]) * vsz;
                float lod = t < t_lod1 ? 0.f : log2f(fmaxf(1.f, 2.f * t * pixk));
                const float2 rg = HW ? cgs::quad_hw<true>(vd, v0, v1, v2, lod)
                                     : cgs::quad<FMT, true, true, true>(vd, v0, v1, v2, lod);
                if (rg.x > 0.f) {
                    float rho = rg.x * (HW ? cgs::fbm_volume(tp, p0, p1, p2)
                                           : cgs::fbm(tp, p0, p1, p2));
                    if (rho > 0.f) {
                        float alpha = 1.f - (HW ? __expf(-tp.sigma * rho * dt) : expf(-tp.sigma * rho * dt));
                        w = T * alpha;
                        G = rg.y;
                        emit = true;
                        T *= 1.f - alpha;
                        if (T < tp.cutoff) live = false;
                    }
                }
            }
            record(emit, v0, v1, v2, w, G);
        }
    }
    if (lane == 0) {
        sb.count[region] = cnt;
        sb.nsteps[region] = nsteps;
    }
    if (HW && cnt == 0u) {
        // no sample in the region (nine tenths of a 1080p view): its pixels are
        // done, and the accumulate pass neither reads nor writes them
        if (valid)
            dst[(size_t)py * cam.W + px] = make_float4(
                0.f * tp.sun_color[0], 0.f * tp.sun_color[1], 0.f * tp.sun_color[2], 1.f - T);
    } else {
        if (HW && lane == 0) sb.busy[atomicAdd(sb.n_busy, 1u)] = (unsigned)region;
        if (valid) sb.alpha[(size_t)py * cam.W + px] = 1.f - T;
    }
    // Flat order for the shading pass: the CTA's regions take one contiguous
    // range (reserved with one atomic, padded to whole 32-sample chunks), and
    // every flat row records its sample's slot.
    __shared__ unsigned s_cnt[MARCH_WARPS], s_base, s_tot;
    const int w = threadIdx.x >> 5;
    if (lane == 0) s_cnt[w] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned tot = 0;
        for (int k = 0; k < MARCH_WARPS; ++k) tot += s_cnt[k];
        s_tot = tot;
        s_base = tot ? atomicAdd(sb.flat_total, (tot + 31u) & ~31u) : 0u;
    }
    __syncthreads();
    unsigned o0 = s_base;
    for (int k = 0; k < w; ++k) o0 += s_cnt[k];
    const unsigned slot0 = (unsigned)region * (unsigned)sb.capacity;
    for (unsigned j = lane; j < cnt; j += 32u) sb.slot_of[o0 + j] = slot0 + j;
    if (w == MARCH_WARPS - 1) {
        const unsigned end = s_base + s_tot, pad_end = s_base + ((s_tot + 31u) & ~31u);
        if (end + lane < pad_end) sb.slot_of[end + lane] = CG_NO_SLOT;
    }
}

// Sum of each lane's contributions over one chunk of up to 32 samples:
// sample j (held by lane j) belongs to pixel lane lj; pixels accumulate in j
// order with Neumaier compensation.
__device__ __forceinline__ void scatter_chunk(float c, int lj, int m, float& acc, float& comp) {
    const int lane = threadIdx.x & 31;
    for (int j = 0; j < m; ++j) {
        float cj = __shfl_sync(0xffffffffu, c, j);
        int pj = __shfl_sync(0xffffffffu, lj, j);
        if (pj == lane) cgs::neumaier(acc, comp, cj);
    }
}

// The pixel's colour C * sun colour with the alpha the march left in
// `alpha`, stored to `dst` (a device image or the caller's page-locked host
// image).
__device__ __forceinline__ void write_rgb(const float* alpha, float4* dst, const CamDesc& cam,
                                          int px, int py, float C, const TraceParams& tp) {
    if (px < cam.W && py < cam.H) {
        const size_t i = (size_t)py * cam.W + px;
        dst[i] = make_float4(C * tp.sun_color[0], C * tp.sun_color[1], C * tp.sun_color[2],
                             alpha[i]);
    }
}

template <int FMT>
__global__ void __launch_bounds__(128)
    k_shade_exact(const __grid_constant__ VolDesc vd, const __grid_constant__ CamDesc cam,
                  const __grid_constant__ TraceParams tp, const __grid_constant__ ConeSchedule cs,
                  SampleBuf sb, int regions, int tiles_x, float4* out) {
    const int region = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (region >= regions) return;
    const int lane = threadIdx.x & 31;
    const unsigned n = sb.count[region];
    const float4* pw = sb.pos_w + (size_t)region * sb.capacity;
    const float2* gl = sb.light_lane + (size_t)region * sb.capacity;
    float acc = 0.f, comp = 0.f;
    for (unsigned base = 0; base < n; base += 32) {
        const unsigned i = base + lane;
        float c = 0.f;
        int lj = -1;
        if (i < n) {
            float4 s = pw[i];
            float2 g = gl[i];
            float tau = cgs::sun_cone<FMT>(vd, cs, s.x, s.y, s.z, tp.sun[0], tp.sun[1], tp.sun[2]);
            float L = expf(-tp.sigma * tau) * (tp.ambient + (1.f - tp.ambient) * g.x);
            c = s.w * L;
            lj = __float_as_int(g.y);
        }
        scatter_chunk(c, lj, (int)min(32u, n - base), acc, comp);
    }
    int px, py;
    region_pixel(region, lane, tiles_x, px, py);
    write_rgb(sb.alpha, out, cam, px, py, acc + comp, tp);
}

// Per busy region (one with samples; one warp each): each pixel sums the
// contributions of its own samples in step order, locating them through the
// march's step table (base slot, ballot).  A grid of warps walks the march's
// list, so the regions without samples cost nothing here (1080p: 26 -> 19 us).
__global__ void __launch_bounds__(128) k_accumulate(CamDesc cam, TraceParams tp, SampleBuf sb,
                                                    int tiles_x, int view_steps, float4* dst) {
    grid_dep_wait();  // the contributions of the shading pass
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const unsigned nb = *sb.n_busy;
    for (unsigned i = blockIdx.x * 4u + (threadIdx.x >> 5); i < nb; i += gridDim.x * 4u) {
        const int region = (int)sb.busy[i];
        const unsigned ns = sb.nsteps[region];
        const uint2* steps = sb.steps + (size_t)region * view_steps;
        const float* cw = sb.contrib + (size_t)region * sb.capacity;
        float acc = 0.f, comp = 0.f;
        // the step table in coalesced chunks of 32 entries (lane e holds entry
        // e), broadcast by shuffles; eight steps' contributions are fetched
        // before any is summed, and the sums run in step order
        for (unsigned base = 0; base < ns; base += 32u) {
            const unsigned m = min(32u, ns - base);
            const uint2 st_l = lane < (int)m ? steps[base + lane] : make_uint2(0u, 0u);
            for (unsigned e0 = 0; e0 < m; e0 += 8u) {
                float v[8];
                unsigned have = 0u;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int src = (int)(e0 + q) & 31;
                    const unsigned sx = __shfl_sync(0xffffffffu, st_l.x, src);
                    const unsigned sy = __shfl_sync(0xffffffffu, st_l.y, src);
                    v[q] = 0.f;
                    // entries past m are (0, 0): no lane emitted there
                    if (e0 + q < m && ((sy >> lane) & 1u) &&
                        CG_IN_BOUNDS((size_t)region * sb.capacity + sx + __popc(sy & below),
                                     sb.nslots)) {
                        v[q] = cw[sx + __popc(sy & below)];
                        have |= 1u << q;
                    }
                }
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if ((have >> q) & 1u) cgs::neumaier(acc, comp, v[q]);
            }
        }
        int px, py;
        region_pixel(region, lane, tiles_x, px, py);
        write_rgb(sb.alpha, dst, cam, px, py, acc + comp, tp);
    }
}

// First sample of every region in region order (off[regions] = their number):
// one CTA, each thread a contiguous piece of the counts.
__global__ void __launch_bounds__(1024) k_sample_offsets(const unsigned* count, int regions,
                                                         unsigned long long* off) {
    __shared__ unsigned long long s_warp[32];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int per = (regions + 1023) / 1024;
    const int a = min(regions, t * per), b = min(regions, a + per);
    unsigned long long sum = 0ull;
#pragma unroll 8
    for (int r = a; r < b; ++r) sum += count[r];
    unsigned long long x = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[w] = x;
    __syncthreads();
    if (w == 0) {
        unsigned long long v = s_warp[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
        }
        s_warp[lane] = v;
    }
    __syncthreads();
    unsigned long long at = x - sum + (w ? s_warp[w - 1] : 0ull);
#pragma unroll 8
    for (int r = a; r < b; ++r) {
        off[r] = at;
        at += count[r];
    }
    if (t == 1023) off[regions] = at;
}

// Samples [lo, lo + n) of that order, packed: a warp per region, bound by the
// read of 16 bytes a sample.
__global__ void __launch_bounds__(256) k_gather_samples(SampleBuf sb, const unsigned long long* off,
                                                        int regions, unsigned long long lo,
                                                        unsigned n, float* positions,
                                                        float* weights) {
    const int region = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (region >= regions) return;
    const unsigned long long a = off[region], b = off[region + 1];
    if (b <= lo || a >= lo + n) return;
    const float4* pw = sb.pos_w + (size_t)region * sb.capacity;
    const unsigned long long end = min(b, lo + n);
    for (unsigned long long i = max(a, lo) + lane; i < end; i += 32) {
        if (!CG_IN_BOUNDS((size_t)region * sb.capacity + (i - a), sb.nslots)) continue;
        const float4 s = pw[i - a];
        const size_t o = (size_t)(i - lo);
        positions[3 * o] = s.x;
        positions[3 * o + 1] = s.y;
        positions[3 * o + 2] = s.z;
        weights[o] = s.w;
    }
}

}  // namespace

static int regions_of(const CamDesc& cam) { return ((cam.W + 15) / 16) * ((cam.H + 15) / 16) * 8; }

static dim3 march_grid(const CamDesc& cam) {
    return dim3((cam.W + 15) / 16 * (8 / MARCH_WARPS), (cam.H + 15) / 16);
}

cudaError_t launch_march(VolDesc vd, CamDesc cam, TraceParams tp, SampleBuf sb, cudaStream_t st) {
    // the flat-order reservation counter starts from zero on every launch
    cudaError_t e = cudaMemsetAsync(sb.flat_total, 0, sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    constexpr int threads = 32 * MARCH_WARPS;
    if (vd.fmt == 0)
        k_march<0, false><<<march_grid(cam), threads, 0, st>>>(vd, cam, tp, sb, nullptr, nullptr);
    else
        k_march<1, false><<<march_grid(cam), threads, 0, st>>>(vd, cam, tp, sb, nullptr, nullptr);
    return cudaGetLastError();
}

cudaError_t launch_march_mlp(VolDesc vd, CamDesc cam, TraceParams tp, SampleBuf sb, float4* dst,
                             unsigned long long* status, cudaStream_t st) {
    // the flat-order reservation counter and the busy count start from zero
    cudaError_t e = cudaMemsetAsync(sb.flat_total, 0, 2 * sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    k_march<0, true><<<march_grid(cam), 32 * MARCH_WARPS, 0, st>>>(vd, cam, tp, sb, dst, status);
    return cudaGetLastError();
}

cudaError_t launch_sample_offsets(const SampleBuf& sb, int regions, unsigned long long* off,
                                  cudaStream_t st) {
    k_sample_offsets<<<1, 1024, 0, st>>>(sb.count, regions, off);
    return cudaGetLastError();
}

cudaError_t launch_gather_samples(const SampleBuf& sb, const unsigned long long* off, int regions,
                                  unsigned long long lo, unsigned n, float* positions,
                                  float* weights, cudaStream_t st) {
    k_gather_samples<<<(regions + 7) / 8, 256, 0, st>>>(sb, off, regions, lo, n, positions,
                                                        weights);
    return cudaGetLastError();
}

cudaError_t launch_shade_exact(VolDesc vd, CamDesc cam, TraceParams tp, SampleBuf sb,
                               float4* out, cudaStream_t st) {
    ConeSchedule cs = make_cone_schedule(vd, tp);
    const int regions = regions_of(cam), tiles_x = (cam.W + 15) / 16;
    const int blocks = (regions + 3) / 4;
    if (vd.fmt == 0)
        k_shade_exact<0><<<blocks, 128, 0, st>>>(vd, cam, tp, cs, sb, regions, tiles_x, out);
    else
        k_shade_exact<1><<<blocks, 128, 0, st>>>(vd, cam, tp, cs, sb, regions, tiles_x, out);
    return cudaGetLastError();
}

cudaError_t launch_accumulate(CamDesc cam, TraceParams tp, SampleBuf sb, float4* dst,
                              cudaStream_t st) {
    // at most twelve CTAs per SM (152 SMs), which take the busy regions in turn
    const int tiles_x = (cam.W + 15) / 16;
    const int blocks = std::min((regions_of(cam) + 3) / 4, 152 * 12);
    return launch_dependent(k_accumulate, dim3(blocks), dim3(128), 0, st, cam, tp, sb, tiles_x,
                            (int)tp.view_steps, dst);
}

CG_OOB_TU(k_deferred)
