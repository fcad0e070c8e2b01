// k_trace.cu -- per-pixel view march with the exact sun cone (one thread per
// pixel), and the traceCone evaluator.
#include "cg_internal.h"
#include "cg_sample.cuh"

namespace {

// 16x16 pixel tile per 256-thread CTA; each warp owns an 8x4 sub-tile so that
// its rays stay spatially coherent.
__device__ __forceinline__ void tile_pixel(int& px, int& py) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    px = blockIdx.x * 16 + (w & 1) * 8 + (lane & 7);
    py = blockIdx.y * 16 + (w >> 1) * 4 + (lane >> 3);
}

// Ray through the pixel centre and its slab interval against the world box.
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

// Counts (STATS only): [0] view samples evaluated, [1] sun cones, [2] sun-cone
// samples, [3] pixels whose ray met the box.  The counting variant is used
// once, untimed, to derive the algorithmic bytes of a frame.
template <bool STATS>
__device__ __forceinline__ void bump(unsigned long long* stats, int i, unsigned v) {
    if (STATS && v) atomicAdd(stats + i, (unsigned long long)v);
}

template <int FMT, bool STATS>
__global__ void __launch_bounds__(256)
    k_trace_fused(const __grid_constant__ VolDesc vd, const __grid_constant__ CamDesc cam,
                  const __grid_constant__ TraceParams tp, const __grid_constant__ ConeSchedule cs,
                  float4* out, unsigned long long* stats) {
    int px, py;
    tile_pixel(px, py);
    if (px >= cam.W || py >= cam.H) return;
    float3 d;
    float tin, tout;
    float4 res = make_float4(0.f, 0.f, 0.f, 0.f);
    unsigned n_view = 0, n_cone = 0, n_sun = 0, n_hit = 0;
    if (pixel_ray(cam, vd, px, py, d, tin, tout)) {
        n_hit = 1;
        const int Nv = tp.view_steps;
        const float dt = (tout - tin) / (float)Nv;
        const float D = (float)vd.D;
        const float vsx = D / vd.range[0], vsy = D / vd.range[1], vsz = D / vd.range[2];
        const float pixk = cam.tanh / (float)cam.H * vsx;
        // when every sample has lod 0, steps outside the occupied box read 0
        int kbeg = 0, kend = Nv;
        const float tlast = tin + ((float)(Nv - 1) + 0.5f) * dt;
        if (2.f * tlast * pixk <= 1.f) {
            int k0, k1;
            cgs::occupied_steps(vd, cam.eye, d, tin, dt, Nv, k0, k1);
            kbeg = k0;
            kend = k1 + 1;
        }
        float T = 1.f, C = 0.f, Cc = 0.f;
        for (int k = kbeg; k < kend; ++k) {
            float t = tin + ((float)k + 0.5f) * dt;
            float p0 = cam.eye[0] + t * d.x, p1 = cam.eye[1] + t * d.y, p2 = cam.eye[2] + t * d.z;
            float v0 = (p0 - vd.wmin[0]) * vsx, v1 = (p1 - vd.wmin[1]) * vsy,
                  v2 = (p2 - vd.wmin[2]) * vsz;
            float lod = log2f(fmaxf(1.f, 2.f * t * pixk));
            float2 rg = cgs::quad<FMT, true, true, true>(vd, v0, v1, v2, lod);
            n_view++;
            if (!(rg.x > 0.f)) continue;
            float rho = rg.x * cgs::fbm(tp, p0, p1, p2);
            if (!(rho > 0.f)) continue;
            float alpha = 1.f - expf(-tp.sigma * rho * dt);
            float tau = cgs::sun_cone<FMT>(vd, cs, v0, v1, v2, tp.sun[0], tp.sun[1], tp.sun[2]);
            if (STATS) {
                n_cone++;
                n_sun += cgs::cone_samples(vd, cs, v0, v1, v2, tp.sun[0], tp.sun[1], tp.sun[2]);
            }
            float Ts = expf(-tp.sigma * tau);
            float L = Ts * (tp.ambient + (1.f - tp.ambient) * rg.y);
            cgs::neumaier(C, Cc, T * alpha * L);
            T *= 1.f - alpha;
            if (T < tp.cutoff) break;
        }
        C += Cc;
        res = make_float4(C * tp.sun_color[0], C * tp.sun_color[1], C * tp.sun_color[2], 1.f - T);
    }
    out[(size_t)py * cam.W + px] = res;
    bump<STATS>(stats, 0, n_view);
    bump<STATS>(stats, 1, n_cone);
    bump<STATS>(stats, 2, n_sun);
    bump<STATS>(stats, 3, n_hit);
}

// Step i of the reference cone (the light channel, clamp to edge, weight i).
template <int FMT>
__device__ __forceinline__ float quad_split_ref(const VolDesc& vd, const ConeSchedule& cs, int i,
                                                float x, float y, float z) {
    return cgs::quad_split<FMT, true, false, false>(vd, x, y, z, cs.st[i].l0, cs.st[i].frac).y *
           cs.st[i].w;
}

// One lane's share of a sun cone traced by the whole warp: the weighted
// samples of cone steps lane, lane + 32 (steps that lie beyond the box's
// widened bounds contribute nothing: along the ray they come after the step
// at which the serial cone stops, and none comes back inside).
template <int FMT>
__device__ __forceinline__ float cone_part(const VolDesc& vd, const ConeSchedule& cs, float vx,
                                           float vy, float vz, float sx, float sy, float sz,
                                           int lane) {
    float part = 0.f;
    const float D = (float)vd.D, E = cs.edge;
#pragma unroll
    for (int r = 0; r < CG_MAX_SUN_STEPS / 32; ++r) {
        const int i = lane + 32 * r;
        if (i >= cs.steps) break;
        const float h = cs.st[i].h;
        const float x = vx + h * sx, y = vy + h * sy, z = vz + h * sz;
        if (cs.quads) {
            const ConeStep& s = cs.st[i];
            float a = cgs::tri_quads<FMT>(vd, s.sc0, s.off0, s.p0, x, y, z);
            if (s.frac > 0.f) {
                const float b = cgs::tri_quads<FMT>(vd, s.sc1, s.off1, s.p1, x, y, z);
                a = a + s.frac * (b - a);
            }
            part += a * s.w;
        } else if (cs.mode == 1) {
            part += quad_split_ref<FMT>(vd, cs, i, x, y, z);
        } else if (!(x < -E || y < -E || z < -E || x > D + E || y > D + E || z > D + E)) {
            part += cgs::quad_split<FMT, false, true, true>(vd, x, y, z, cs.st[i].l0,
                                                            cs.st[i].frac)
                        .x *
                    cs.st[i].w;
        }
    }
    return part;
}

// The fused trace with warp-cooperative sun cones: the warp marches its 32
// rays (an 8x4 tile) in lockstep over the view steps; at a step where at most
// coop_max lanes' samples contribute, the warp traces each of those samples'
// cones in turn, its lanes over the cone steps, the weighted samples summed
// by a shuffle tree; at a step with more, every contributing lane traces its
// own cone as k_trace_fused does.  Samples, opacities and the compositing
// order are k_trace_fused's; only the order in which a cooperative cone's
// terms are added differs.
// Threads of a CTA (256 / COOP_THREADS of them share a 16x16 pixel block) and the
// warps an SM is to hold.  FP32 volumes, 1080p over 256^3, us: 256 threads and 32
// warps 641, 128 and 32 626, 128 and 28 621 (72 registers, hardly a spill; a CTA lives
// as long as its slowest warp), 128 and 24 635, 64 and 32 740.  Half-precision
// volumes would gain as much (4K over 512^3 3907 -> 3791) and keep the larger CTAs
// so that the surrogate stays the faster one next to a cone of half the steps.
template <int FMT>
constexpr int COOP_THREADS = FMT == 0 ? 128 : 256;
template <int FMT>
constexpr int COOP_WARPS = FMT == 0 ? 28 : 32;

template <int FMT>
__global__ void __launch_bounds__(COOP_THREADS<FMT>, COOP_WARPS<FMT> * 32 / COOP_THREADS<FMT>)
    k_trace_coop(const __grid_constant__ VolDesc vd, const __grid_constant__ CamDesc cam,
                 const __grid_constant__ TraceParams tp,
                 const __grid_constant__ ConeSchedule cone, float4* out, int coop_max) {
    // the schedule in shared memory: a cooperative cone's lanes read
    // different steps, which the constant bank would serve one by one
    __shared__ ConeSchedule cs;
    for (int i = threadIdx.x; i < (int)(sizeof(ConeSchedule) / 16); i += blockDim.x)
        reinterpret_cast<uint4*>(&cs)[i] = reinterpret_cast<const uint4*>(&cone)[i];
    __syncthreads();
    constexpr int SHARE = 256 / COOP_THREADS<FMT>;
    const int lane = threadIdx.x & 31;
    const int w = (int)(blockIdx.x % SHARE) * (8 / SHARE) + (int)(threadIdx.x >> 5);
    const int px = (int)(blockIdx.x / SHARE) * 16 + (w & 1) * 8 + (lane & 7);
    const int py = (int)blockIdx.y * 16 + (w >> 1) * 4 + (lane >> 3);
    const bool valid = px < cam.W && py < cam.H;
    float3 d = make_float3(0.f, 0.f, 0.f);
    float tin = 0.f, tout = 0.f;
    const bool hit = valid && pixel_ray(cam, vd, px, py, d, tin, tout);
    bool live = hit;
    const int Nv = tp.view_steps;
    const float dt = (tout - tin) / (float)Nv;
    const float D = (float)vd.D;
    const float vsx = D / vd.range[0], vsy = D / vd.range[1], vsz = D / vd.range[2];
    const float pixk = cam.tanh / (float)cam.H * vsx;
    int kbeg = 0, kend = Nv;
    bool lod0 = true;
    if (live) {
        const float tlast = tin + ((float)(Nv - 1) + 0.5f) * dt;
        lod0 = 2.f * tlast * pixk <= 1.f;
        if (lod0) {
            int k0, k1;
            cgs::occupied_steps(vd, cam.eye, d, tin, dt, Nv, k0, k1);
            kbeg = k0;
            kend = k1 + 1;
        }
        if (kbeg >= kend) live = false;
    }
    float T = 1.f, C = 0.f, Cc = 0.f;
    const int wk0 = __reduce_min_sync(0xffffffffu, live ? kbeg : Nv);
    // SKIP: every lane's samples have lod 0 (the common case), so a step reads 0
    // where its brick is unoccupied: the flags of eight steps are fetched together
    // (linear in k, off by a rounding at most, which the flags allow: they cover
    // the bricks around), and only the steps at which some lane has one are taken.
    // FP32 volumes only, as COOP_THREADS (1080p over 256^3 621 -> 590 us).
    const bool skip = FMT == 0 && __all_sync(0xffffffffu, !live || lod0);
    cgs::OccRay bricks;
    if (skip) {
        const float o = tin + 0.5f * dt;
        const float v0a[3] = {(cam.eye[0] + o * d.x - vd.wmin[0]) * vsx,
                              (cam.eye[1] + o * d.y - vd.wmin[1]) * vsy,
                              (cam.eye[2] + o * d.z - vd.wmin[2]) * vsz};
        const float dva[3] = {dt * d.x * vsx, dt * d.y * vsy, dt * d.z * vsz};
        bricks.set(vd, 0, v0a, dva, (float)(1 << vd.occ_shift), -0.5f);
    }
    unsigned mine = 0u, any = 0u;  // flags of the steps of the chunk at kc: this lane's, the warp's
    int kc = wk0 - 8;
    for (int k = wk0;; ++k) {
        if (skip) {
            while (!any) {
                kc += 8;
                if (live && kc >= kend) live = false;
                if (kc >= Nv || !__any_sync(0xffffffffu, live)) break;
                mine = 0u;
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    mine |= (bricks.at((float)(kc + j)) && kc + j >= kbeg && kc + j < kend ? 1u : 0u)
                            << j;
                if (!live) mine = 0u;
                any = __reduce_or_sync(0xffffffffu, mine);
            }
            if (!any) break;
            k = kc + __ffs(any) - 1;
            any &= any - 1u;
        } else {
            if (live && k >= kend) live = false;
            if (k >= Nv || !__any_sync(0xffffffffu, live)) break;
        }
        bool emit = false;
        float v0 = 0.f, v1 = 0.f, v2 = 0.f, alpha = 0.f, G = 0.f;
        if (live && (skip ? (mine >> (k - kc)) & 1u : k >= kbeg)) {
            const float t = tin + ((float)k + 0.5f) * dt;
            const float p0 = cam.eye[0] + t * d.x, p1 = cam.eye[1] + t * d.y,
                        p2 = cam.eye[2] + t * d.z;
            v0 = (p0 - vd.wmin[0]) * vsx;
            v1 = (p1 - vd.wmin[1]) * vsy;
            v2 = (p2 - vd.wmin[2]) * vsz;
            const float2 rg =
                skip ? cgs::tri<FMT, true, true, false>(vd, 0, v0, v1, v2)
                     : cgs::quad<FMT, true, true, true>(vd, v0, v1, v2,
                                                        log2f(fmaxf(1.f, 2.f * t * pixk)));
            if (rg.x > 0.f) {
                const float rho = rg.x * cgs::fbm(tp, p0, p1, p2);
                if (rho > 0.f) {
                    alpha = 1.f - expf(-tp.sigma * rho * dt);
                    G = rg.y;
                    emit = true;
                }
            }
        }
        const unsigned ballot = __ballot_sync(0xffffffffu, emit);
        if (!ballot) continue;
        float tau = 0.f;
        if (__popc(ballot) <= coop_max) {
            for (unsigned b = ballot; b; b &= b - 1u) {
                const int j = __ffs(b) - 1;
                const float x0 = __shfl_sync(0xffffffffu, v0, j);
                const float x1 = __shfl_sync(0xffffffffu, v1, j);
                const float x2 = __shfl_sync(0xffffffffu, v2, j);
                float part = cone_part<FMT>(vd, cs, x0, x1, x2, tp.sun[0], tp.sun[1], tp.sun[2],
                                            lane);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
                if (lane == j) tau = part;
            }
        } else if (emit) {
            tau = cgs::sun_cone<FMT>(vd, cs, v0, v1, v2, tp.sun[0], tp.sun[1], tp.sun[2]);
        }
        if (emit) {
            const float Ts = expf(-tp.sigma * tau);
            const float L = Ts * (tp.ambient + (1.f - tp.ambient) * G);
            cgs::neumaier(C, Cc, T * alpha * L);
            T *= 1.f - alpha;
            if (T < tp.cutoff) live = false;
        }
    }
    C += Cc;
    if (valid)
        out[(size_t)py * cam.W + px] =
            hit ? make_float4(C * tp.sun_color[0], C * tp.sun_color[1], C * tp.sun_color[2],
                              1.f - T)
                : make_float4(0.f, 0.f, 0.f, 0.f);
}

template <int FMT>
__global__ void k_trace_cones(const __grid_constant__ VolDesc vd,
                              const __grid_constant__ TraceParams tp,
                              const __grid_constant__ ConeSchedule cs, const float* pos, int n,
                              float* out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
    // a caller's position may be a NaN, which the pyramid's own walk carries
    // through only where it samples something
    if (cs.quads && !isnan(x + y + z))
        out[i] = cgs::cone_quads<FMT, false>(vd, cs, x, y, z, tp.sun[0], tp.sun[1], tp.sun[2]);
    else
        out[i] = cgs::cone_general<FMT>(vd, cs, x, y, z, tp.sun[0], tp.sun[1], tp.sun[2]);
}

}  // namespace

// Cone schedule in FP64 on the host (see ConeSchedule).
ConeSchedule make_cone_schedule(const VolDesc& vd, const TraceParams& tp) {
    ConeSchedule cs{};
    cs.steps = tp.sun_steps;
    cs.mode = tp.cone_mode;
    cs.edge = (float)vd.D / (float)vd.dims[vd.L - 1];
    const double vw = (double)vd.range[0] / (double)vd.D;
    double h = tp.h0;
    const double maxl = (double)(vd.L - 1);
    for (int i = 0; i < tp.sun_steps && i < CG_MAX_SUN_STEPS; ++i) {
        double r, lod, w;
        if (tp.cone_mode == 1) {
            r = h * (double)tp.tan_half;
            double rr = 2.0 * r > 1.0 ? 2.0 * r : 1.0;
            lod = log2(rr) + (double)tp.lod_offset;
            w = (double)(i + 1) / ((double)tp.sun_steps * (double)tp.down_scaling);
        } else {
            r = h * (double)tp.tan_half;
            if (r < (double)tp.rmin) r = (double)tp.rmin;
            double rr = 2.0 * r > 1.0 ? 2.0 * r : 1.0;
            lod = log2(rr) + (double)tp.lod_offset;
            w = r * vw;
        }
        if (!(lod > 0.0)) lod = 0.0;
        if (lod > maxl) lod = maxl;
        int l0 = (int)floor(lod);
        cs.st[i].h = (float)h;
        cs.st[i].w = (float)w;
        cs.st[i].l0 = l0;
        cs.st[i].frac = (float)(lod - (double)l0);
        h += r;
    }
    // density quads: every level the cone reads must have them.  reach: half a
    // texel of the coarsest level read, plus a voxel for the rounding of the
    // distance to the box
    bool quads = tp.cone_mode != 1 && vd.quad != nullptr && tp.sun_steps > 0;
    for (int i = 0; i < cs.steps && quads; ++i) quads = cs.st[i].l0 >= vd.quad_base;
    cs.quads = quads ? 1 : 0;
    if (quads) {
        for (int i = 0; i < cs.steps; ++i) {
            ConeStep& s = cs.st[i];
            const int l1 = s.l0 + 1 < vd.L ? s.l0 + 1 : vd.L - 1;
            s.sc0 = vd.lsc[s.l0];
            s.off0 = vd.quad_off[s.l0];
            s.p0 = vd.quad_p[s.l0];
            s.sc1 = vd.lsc[l1];
            s.off1 = vd.quad_off[l1];
            s.p1 = vd.quad_p[l1];
            const float half = 0.5f * (float)vd.D / (float)vd.dims[s.frac > 0.f ? l1 : s.l0];
            if (half + 1.f > cs.reach) cs.reach = half + 1.f;
        }
        // (positions within flat_reach of the box stay in the padded quads)
        cs.flat_reach = 0.5f / cs.st[0].sc0 + 1.f;
        if (cs.st[0].sc0 <= 0.75f && cs.st[0].h >= 0.f)
            while (cs.flat < cs.steps && cs.st[cs.flat].l0 == cs.st[0].l0 &&
                   cs.st[cs.flat].frac == 0.f)
                ++cs.flat;
        cs.flat &= ~1;
        if (cs.steps & 1) {
            cs.st[cs.steps] = cs.st[cs.steps - 1];
            cs.st[cs.steps].w = 0.f;
        }
    }
    return cs;
}

template <int FMT>
static void coop(dim3 blocks16, const VolDesc& vd, const CamDesc& cam, const TraceParams& tp,
                 const ConeSchedule& cs, float4* out, cudaStream_t st) {
    constexpr int T = COOP_THREADS<FMT>;
    k_trace_coop<FMT><<<dim3(blocks16.x * (256 / T), blocks16.y), T, 0, st>>>(vd, cam, tp, cs, out,
                                                                             tp.cone_lanes);
}

cudaError_t launch_trace_fused(VolDesc vd, CamDesc cam, TraceParams tp, float4* out,
                               unsigned long long* stats, cudaStream_t st) {
    ConeSchedule cs = make_cone_schedule(vd, tp);
    dim3 grd((cam.W + 15) / 16, (cam.H + 15) / 16);
    if (!stats && tp.cone_lanes > 0) {
        if (vd.fmt == 0)
            coop<0>(grd, vd, cam, tp, cs, out, st);
        else
            coop<1>(grd, vd, cam, tp, cs, out, st);
    } else if (stats) {
        if (vd.fmt == 0)
            k_trace_fused<0, true><<<grd, 256, 0, st>>>(vd, cam, tp, cs, out, stats);
        else
            k_trace_fused<1, true><<<grd, 256, 0, st>>>(vd, cam, tp, cs, out, stats);
    } else {
        if (vd.fmt == 0)
            k_trace_fused<0, false><<<grd, 256, 0, st>>>(vd, cam, tp, cs, out, nullptr);
        else
            k_trace_fused<1, false><<<grd, 256, 0, st>>>(vd, cam, tp, cs, out, nullptr);
    }
    return cudaGetLastError();
}

namespace {
// Lattice values of every tabulated octave (one thread per entry).
__global__ void k_noise_table(TraceParams tp, float* tab, int total) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    int o = 0;
    while (o + 1 < tp.noise_octaves && i >= tp.nt.off[o + 1]) ++o;
    int r = i - tp.nt.off[o];
    const int dx = tp.nt.dim[o][0], dy = tp.nt.dim[o][1];
    int tx = r % dx, ty = (r / dx) % dy, tz = r / (dx * dy);
    tab[i] = cgs::lattice(tp.nt.lo[o][0] + tx, tp.nt.lo[o][1] + ty, tp.nt.lo[o][2] + tz,
                          cgs::octave_key(tp.noise_seed, o));
}
}  // namespace

cudaError_t launch_noise_table(TraceParams tp, float* tab, int total, cudaStream_t st) {
    if (total <= 0) return cudaSuccess;
    k_noise_table<<<(total + 255) / 256, 256, 0, st>>>(tp, tab, total);
    return cudaGetLastError();
}

cudaError_t launch_trace_cones(VolDesc vd, TraceParams tp, const float* pos, int n, float* out,
                               cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    ConeSchedule cs = make_cone_schedule(vd, tp);
    if (cs.mode == 1) return launch_reference_cones(vd, tp, cs, pos, n, out, st);
    int blocks = (n + 127) / 128;
    if (vd.fmt == 0)
        k_trace_cones<0><<<blocks, 128, 0, st>>>(vd, tp, cs, pos, n, out);
    else
        k_trace_cones<1><<<blocks, 128, 0, st>>>(vd, tp, cs, pos, n, out);
    return cudaGetLastError();
}

CG_OOB_TU(k_trace)
