// fluid.cu -- the particle entry points of cupar:: (src/ParticleGPU.cuh:11-21):
// integrator stages, periodic wrap, density, equation of state, the SDPD
// pair force, wall repulsion, body force and the no-slip wall velocity.
//
// These are the FP32 kernels behind the drop-in boundary: one kernel per
// entry point on the caller's arrays (float3/float4, slot order), no state
// kept from one call to the next.  The neighbour passes sweep the 27 cubes of
// the caller's begin/end table, one block per cube (sweep.cuh); the others run
// one thread per slot.  Particle type is decided from the original id in
// d_sortpart (src/Particle.cu:432-435).
//
// The formulas (pinned because GPUCell's kernel bodies are absent):
//   density   rho_i = m (W(0) + sum_j W_ij), j over Bound2, fluid, membrane;
//             Bound2 keeps rho = DenInit (src/ParticleGPU.cuh:13 comment)
//   EOS       P_i = c_i^2 (rho_i - rho0), c = SoundSpeed1 (fluid, Bound2) or
//             SoundSpeed2 (membrane)
//   SDPD      Espanol & Revenga (2003), with d = rho/m:
//             f_i = sum_j (P_i/d_i^2 + P_j/d_j^2) F_ij r_ij
//                   - F_ij/(d_i d_j) [A v_ij + B e_ij (e_ij . v_ij)]
//                   + q_ij [sqrt(A) xi_ij + (sqrt(A+B) - sqrt(A)) e_ij (e_ij . xi_ij)]
//             A = 5 eta/3 - zeta, B = 5 (zeta + eta/3),
//             q_ij = sqrt(2 kT F_ij / (d_i d_j dt)), xi_ij the Philox pair noise
//   repulsion Monaghan (1994): f_i += D [(r0/r)^12 - (r0/r)^4] r_ij / r^2 from
//             Bound1 within r0 = rc/3, D = SoundSpeed1^2
//   walls     Adami, Hu & Adams (2012): v_w = 2 v_presc - sum_f v_f W / sum_f W,
//             v_presc = the wall's VelHalf (zero unless the caller sets it)
//   integrator Groot & Warren (1997) modified velocity-Verlet with lambda = VVsigma
#include "gc_internal.cuh"
#include "sweep.cuh"

namespace {

// K2 -- r += dt v + dt^2/2 F/m for fluid and membrane particles.
__global__ void k_update_coor(int n, GcParams p, const int* __restrict__ sortpart, const float3* __restrict__ force,
                              float3* __restrict__ coor, const float4* __restrict__ velrhop, unsigned* flags) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (!is_mobile((unsigned)sortpart[i], p)) return;
    float3 x = coor[i], f = force[i];
    float4 v = velrhop[i];
    float h = 0.5f * p.dt * p.dt * p.inv_mass;
    x.x += p.dt * v.x + h * f.x;
    x.y += p.dt * v.y + h * f.y;
    x.z += p.dt * v.z + h * f.z;
    if (!(isfinite(x.x) && isfinite(x.y) && isfinite(x.z))) raise_flag(flags, GC_FLAG_NONFINITE);
    coor[i] = x;
}

// K3 -- wrap moving particles into the box on periodic axes and count the
// crossings (+1 for a crossing of the upper face) so that membranes can be
// unwrapped as x + nThroBound * L.
__global__ void k_periodic(int n, GcParams p, const int* __restrict__ sortpart, float3* __restrict__ coor,
                           int3* __restrict__ nthro, const float* __restrict__ bbox, unsigned* flags) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (!is_mobile((unsigned)sortpart[i], p)) return;
    float3 x = coor[i];
    int3 t = nthro[i];
    float* xs[3] = {&x.x, &x.y, &x.z};
    int* ts[3] = {&t.x, &t.y, &t.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (!(p.g.pmask & (1 << a))) continue;
        float lo = bbox[2 * a], hi = bbox[2 * a + 1], L = hi - lo;
        float v = *xs[a];
        if (v >= hi) { v -= L; *ts[a] += 1; }
        else if (v < lo) { v += L; *ts[a] -= 1; }
        // less than half an ulp below lo, v + L rounds to hi itself: a position like any other
        if (v > hi || v < lo) raise_flag(flags, GC_FLAG_NONFINITE);
        *xs[a] = v;
    }
    coor[i] = x;
    nthro[i] = t;
}

// K8 -- kernel-sum density of fluid and membrane particles.
struct DensityOp {
    float4* velrhop;
    static constexpr int kBlocks = 8;   // resident blocks the registers are cut to
    struct Extra {};
    struct Self { unsigned id; };
    struct Acc { float sum; };
    __device__ float cut2(const GcParams& p) const { return p.rc2; }
    __device__ bool active(unsigned id, const GcParams& p) const { return is_mobile(id, p); }
    __device__ bool keep(unsigned id, const GcParams& p) const { return is_sdpd(id, p); }
    __device__ void idle(int) const {}
    __device__ void begin(Acc& a, Self& s, int, unsigned id, bool, const GcParams&) const {
        a.sum = 0.f;
        s.id = id;
    }
    __device__ void stage(Extra&, int, int, const GcParams&) const {}
    __device__ void pair(Acc& a, const Self& s, const Extra&, int, unsigned idj, float3, float r2, const GcParams& p) const {
        if (idj != s.id) a.sum += wendland_w(sqrtf(r2), p);
    }
    __device__ void reduce(Acc& a) const { a.sum = gcsweep::lane_sum(a.sum); }
    __device__ void finish(const Acc& a, const Self&, int i, const GcParams& p) const {
        velrhop[i].w = p.mass * (p.w0 + a.sum);
    }
};

// K9 -- predictor: VelHalf = v + dt/2 F/m, v <- v + lambda dt F/m.
__global__ void k_predict(int n, GcParams p, const int* __restrict__ sortpart, float4* __restrict__ velrhop,
                          float3* __restrict__ velhalf, const float3* __restrict__ force) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (!is_mobile((unsigned)sortpart[i], p)) return;
    float4 v = velrhop[i];
    float3 f = force[i];
    float h = 0.5f * p.dt * p.inv_mass, l = p.lambda * p.dt * p.inv_mass;
    velhalf[i] = f3(v.x + h * f.x, v.y + h * f.y, v.z + h * f.z);
    v.x += l * f.x;
    v.y += l * f.y;
    v.z += l * f.z;
    velrhop[i] = v;
}

// K10 -- no-slip velocity of Bound2 wall particles.
struct Bound2VelOp {
    float4* velrhop;
    const float3* velhalf;
    static constexpr int kBlocks = 6;   // resident blocks the registers are cut to
    struct Extra { float3 v[gcsweep::kCap]; };
    struct Self {};
    struct Acc { float3 num; float den; };
    __device__ float cut2(const GcParams& p) const { return p.rc2; }
    __device__ bool active(unsigned id, const GcParams& p) const { return ptype(id, p) == PT_B2; }
    __device__ bool keep(unsigned id, const GcParams& p) const { return is_mobile(id, p); }
    __device__ void idle(int) const {}
    __device__ void begin(Acc& a, Self&, int, unsigned, bool, const GcParams&) const {
        a.num = f3(0.f, 0.f, 0.f);
        a.den = 0.f;
    }
    __device__ void stage(Extra& e, int q, int j, const GcParams&) const {
        const float4 v = velrhop[j];
        e.v[q] = f3(v.x, v.y, v.z);
    }
    __device__ void pair(Acc& a, const Self&, const Extra& e, int q, unsigned, float3, float r2, const GcParams& p) const {
        const float w = wendland_w(sqrtf(r2), p);
        a.num += w * e.v[q];
        a.den += w;
    }
    __device__ void reduce(Acc& a) const {
        a.num = f3(gcsweep::lane_sum(a.num.x), gcsweep::lane_sum(a.num.y), gcsweep::lane_sum(a.num.z));
        a.den = gcsweep::lane_sum(a.den);
    }
    __device__ void finish(const Acc& a, const Self&, int i, const GcParams&) const {
        const float3 vw = velhalf ? velhalf[i] : f3(0.f, 0.f, 0.f);
        float4 v = velrhop[i];
        if (a.den > 0.f) {
            const float inv = 1.f / a.den;
            v.x = 2.f * vw.x - a.num.x * inv;
            v.y = 2.f * vw.y - a.num.y * inv;
            v.z = 2.f * vw.z - a.num.z * inv;
        } else {
            v.x = vw.x; v.y = vw.y; v.z = vw.z;
        }
        velrhop[i] = v;   // walls only: no other block stages this slot's velocity
    }
};

// K11 -- equation of state.
__global__ void k_eos(int n, GcParams p, const int* __restrict__ sortpart, const float4* __restrict__ velrhop,
                      float* __restrict__ press) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int t = ptype((unsigned)sortpart[i], p);
    float rho = velrhop[i].w;
    float P = 0.f;
    if (t == PT_MEMB) P = p.c2sq * (rho - p.rho0);
    else if (t != PT_B1) P = p.c1sq * (rho - p.rho0);
    press[i] = P;
}

// K12 -- SDPD pair force; writes the force of every slot (zero for walls).
// A candidate's velocity, d and P/d^2 are staged with its position.  The
// pair terms are gathered into one coefficient along d = x_i - x_j (pressure
// and the e e^T parts of the viscous and random forces, e = d/r), one along
// v_ij and one along xi_ij, as in the fused step.  Roots and divisions are the
// correctly rounded ones, here and in the other sweeps: with rsqrt.approx and
// a product of two reciprocals a million-particle step took 0.18 ms less (3.06
// of 3.24), but a pair near the cut-off, where F goes as (1 - r/rc)^3, was off
// by twice as much.
template <bool NOISE>
struct SdpdOp {
    const float4* velrhop;
    const float* press;
    float3* force;
    static constexpr int kBlocks = 6;   // resident blocks the registers are cut to
    struct Extra { float4 v[gcsweep::kCap]; float pt[gcsweep::kCap]; };
    struct Self { float3 v; float d, pt; unsigned id; };
    struct Acc { float3 f; };
    __device__ float cut2(const GcParams& p) const { return p.rc2; }
    __device__ bool active(unsigned id, const GcParams& p) const { return is_mobile(id, p); }
    __device__ bool keep(unsigned id, const GcParams& p) const { return is_sdpd(id, p); }
    __device__ void idle(int i) const { force[i] = f3(0.f, 0.f, 0.f); }
    __device__ void begin(Acc& a, Self& s, int i, unsigned id, bool act, const GcParams& p) const {
        a.f = f3(0.f, 0.f, 0.f);
        if (!act) return;
        const float4 v = velrhop[i];
        const float d = v.w * p.inv_mass;
        s.v = f3(v.x, v.y, v.z);
        s.d = d;
        s.pt = press[i] / (d * d);
        s.id = id;
    }
    __device__ void stage(Extra& e, int q, int j, const GcParams& p) const {
        const float4 v = velrhop[j];
        const float d = v.w * p.inv_mass;
        e.v[q] = make_float4(v.x, v.y, v.z, d);
        e.pt[q] = press[j] / (d * d);
    }
    __device__ void pair(Acc& a, const Self& s, const Extra& e, int q, unsigned idj, float3 d, float r2,
                         const GcParams& p) const {
        if (r2 <= 0.f || idj == s.id) return;   // coincident particles exert no force
        const float4 vj = e.v[q];
        const float r = sqrtf(r2), inv_r = 1.f / r;
        const float F = wendland_f(r, p);
        const float3 vij = f3(s.v.x - vj.x, s.v.y - vj.y, s.v.z - vj.z);
        const float fdd = F / (s.d * vj.w);
        float cd = (s.pt + e.pt[q]) * F - (fdd * p.visB) * (dot3(d, vij) * inv_r) * inv_r;
        a.f += (-fdd * p.visA) * vij;
        if constexpr (NOISE) {
            // a pair at the cut-off can give F a rounding-sized negative value: no noise then
            float n = fdd > 0.f ? sqrtf(p.noise_pref * fdd) : 0.f;
            n = s.id < idj ? n : -n;   // the pair sign of xi_ij
            const float3 xi = pair_noise_unsigned(s.id, idj, p);
            cd += (n * (p.sqrtAB - p.sqrtA)) * (dot3(d, xi) * inv_r) * inv_r;
            a.f += (n * p.sqrtA) * xi;
        }
        a.f += cd * d;
    }
    __device__ void reduce(Acc& a) const {
        a.f = f3(gcsweep::lane_sum(a.f.x), gcsweep::lane_sum(a.f.y), gcsweep::lane_sum(a.f.z));
    }
    __device__ void finish(const Acc& a, const Self&, int i, const GcParams&) const { force[i] = a.f; }
};

// K13 -- repulsion of fluid and membrane particles by Bound1 walls.
struct RepulsionOp {
    float3* force;
    static constexpr int kBlocks = 8;   // resident blocks the registers are cut to
    struct Extra {};
    struct Self {};
    struct Acc { float3 f; };
    __device__ float cut2(const GcParams& p) const { return p.rep_r0sq; }
    __device__ bool active(unsigned id, const GcParams& p) const { return is_mobile(id, p); }
    __device__ bool keep(unsigned id, const GcParams& p) const { return ptype(id, p) == PT_B1; }
    __device__ void idle(int) const {}
    __device__ void begin(Acc& a, Self&, int, unsigned, bool, const GcParams&) const { a.f = f3(0.f, 0.f, 0.f); }
    __device__ void stage(Extra&, int, int, const GcParams&) const {}
    __device__ void pair(Acc& a, const Self&, const Extra&, int, unsigned, float3 d, float r2, const GcParams& p) const {
        if (r2 <= 0.f) return;
        const float q2 = p.rep_r0sq / r2, q4 = q2 * q2, q12 = q4 * q4 * q4;
        a.f += (p.rep_D * (q12 - q4) / r2) * d;
    }
    __device__ void reduce(Acc& a) const {
        a.f = f3(gcsweep::lane_sum(a.f.x), gcsweep::lane_sum(a.f.y), gcsweep::lane_sum(a.f.z));
    }
    __device__ void finish(const Acc& a, const Self&, int i, const GcParams&) const {
        if (a.f.x != 0.f || a.f.y != 0.f || a.f.z != 0.f) force[i] += a.f;
    }
};

template <class Op>
int launch_sweep(const Op& op, int n, const GcParams& p, const float* coor, const int* sortpart, const int* bec,
                 cudaStream_t st, const char* what) {
    const int K = p.g.ncells, per = gcsweep::cubes_per_block(n, K);
    gcsweep::k_sweep<<<gc_blocks(K, per), gcsweep::kBlock, 0, st>>>(K, p, op, (const float3*)coor, sortpart,
                                                                    (const int2*)bec);
    GC_CHECK_LAUNCH(what);
    return GC_OK;
}

// K14 -- body force in x on fluid and membrane particles.
__global__ void k_ext(int n, GcParams p, const int* __restrict__ sortpart, float3* __restrict__ force) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (!is_mobile((unsigned)sortpart[i], p)) return;
    force[i].x += p.gx;
}

// K19 -- corrector: v = VelHalf + dt/2 F/m.
__global__ void k_correct(int n, GcParams p, const int* __restrict__ sortpart, const float3* __restrict__ force,
                          const float3* __restrict__ velhalf, float4* __restrict__ velrhop, unsigned* flags) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (!is_mobile((unsigned)sortpart[i], p)) return;
    float3 f = force[i], h = velhalf[i];
    float4 v = velrhop[i];
    float s = 0.5f * p.dt * p.inv_mass;
    v.x = h.x + s * f.x;
    v.y = h.y + s * f.y;
    v.z = h.z + s * f.z;
    if (!(isfinite(v.x) && isfinite(v.y) && isfinite(v.z))) raise_flag(flags, GC_FLAG_NONFINITE);
    velrhop[i] = v;
}

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Number and id checksum of every slot's neighbours: the pairs that the other
// sweeps evaluate.
struct NeighborOp {
    int* count;
    unsigned long long* hash;
    static constexpr int kBlocks = 8;   // resident blocks the registers are cut to
    struct Extra {};
    struct Self { unsigned id; };
    struct Acc { int cnt; unsigned long long h; };
    __device__ float cut2(const GcParams& p) const { return p.rc2; }
    __device__ bool active(unsigned, const GcParams&) const { return true; }
    __device__ bool keep(unsigned, const GcParams&) const { return true; }
    __device__ void idle(int) const {}
    __device__ void begin(Acc& a, Self& s, int, unsigned id, bool, const GcParams&) const {
        a.cnt = 0;
        a.h = 0;
        s.id = id;
    }
    __device__ void stage(Extra&, int, int, const GcParams&) const {}
    __device__ void pair(Acc& a, const Self& s, const Extra&, int, unsigned idj, float3, float, const GcParams&) const {
        if (idj == s.id) return;
        ++a.cnt;
        a.h += mix64((unsigned long long)idj);
    }
    __device__ void reduce(Acc& a) const {
#pragma unroll
        for (int o = gcsweep::kLanes / 2; o; o >>= 1) {
            a.cnt += __shfl_xor_sync(0xffffffffu, a.cnt, o, gcsweep::kLanes);
            a.h += __shfl_xor_sync(0xffffffffu, a.h, o, gcsweep::kLanes);
        }
    }
    __device__ void finish(const Acc& a, const Self&, int i, const GcParams&) const {
        count[i] = a.cnt;
        hash[i] = a.h;
    }
};

}  // namespace

#define GC_PRE(name, need_grid)                                            \
    GcState& s = gc_state();                                               \
    if (n < 0) return gc_fail(GC_EINVAL, name ": n < 0");                  \
    GcParams p;                                                            \
    GC_TRY(gc_make_params(&p, need_grid));                                 \
    if ((unsigned)n != p.nT)                                               \
        return gc_fail(GC_EINVAL, name ": n = %d but nTotalPar = %u", n, p.nT); \
    if (n == 0) return GC_OK;                                              \
    const int nb = gc_blocks(n, SDPDSIZE);                                 \
    (void)nb

extern "C" {

int gc_cupar_UpdateFluidCoor(int n, int* d_sortpart, float* d_totalforce, float* d_totalcoor, float* d_velrhop) {
    GcState& s0 = gc_state();
    s0.ref.sortpart = d_sortpart;
    s0.ref.force = d_totalforce;
    s0.ref.coor = d_totalcoor;
    s0.ref.velrhop = d_velrhop;
    s0.step += 1;   // first call of every step (src/Particle.cu:1312)
    // With the fused engine, every step after the first is run whole at
    // SetFluidExtForce (which carries DriveOn); the other calls of the step
    // only record their buffers.
    s0.in_fused_step = s0.engine_mode == 1 && s0.plain_steps >= 1;
    if (s0.in_fused_step) return GC_OK;
    s0.plain_steps += 1;
    GC_PRE("UpdateFluidCoor", false);
    k_update_coor<<<nb, SDPDSIZE, 0, s.stream>>>(n, p, d_sortpart, (const float3*)d_totalforce, (float3*)d_totalcoor,
                                                (const float4*)d_velrhop, gc_flags_ptr());
    GC_CHECK_LAUNCH("UpdateFluidCoor");
    return GC_OK;
}

int gc_cupar_AppFluidPeriodicBC(int n, int* d_sortpart, float* d_totalcoor, int* d_nthrobound, float* d_bboxsdpd) {
    gc_state().ref.nthro = d_nthrobound;
    gc_state().ref.bbox = d_bboxsdpd;
    if (gc_state().in_fused_step) return GC_OK;
    GC_PRE("AppFluidPeriodicBC", false);
    p.g.pmask = s.periodic_mask;
    k_periodic<<<nb, SDPDSIZE, 0, s.stream>>>(n, p, d_sortpart, (float3*)d_totalcoor, (int3*)d_nthrobound, d_bboxsdpd,
                                             gc_flags_ptr());
    GC_CHECK_LAUNCH("AppFluidPeriodicBC");
    return GC_OK;
}

int gc_cupar_CalFluidDen(int n, float* d_totalcoor, float* d_velrhop, int* d_cc, int* d_ncube, float* d_outerregion,
                         int* d_sortpart, int* d_beginendcube) {
    if (gc_state().in_fused_step) return GC_OK;
    (void)d_cc; (void)d_ncube; (void)d_outerregion;
    GC_PRE("CalFluidDen", true);
    return launch_sweep(DensityOp{(float4*)d_velrhop}, n, p, d_totalcoor, d_sortpart, d_beginendcube, s.stream,
                        "CalFluidDen");
}

int gc_cupar_PredictFluidVel(int n, int* d_sortpart, float* d_velrhop, float* d_velhalf, float* d_totalforce) {
    gc_state().ref.velhalf = d_velhalf;
    if (gc_state().in_fused_step) return GC_OK;
    GC_PRE("PredictFluidVel", false);
    s.velhalf_ptr = d_velhalf;
    k_predict<<<nb, SDPDSIZE, 0, s.stream>>>(n, p, d_sortpart, (float4*)d_velrhop, (float3*)d_velhalf,
                                            (const float3*)d_totalforce);
    GC_CHECK_LAUNCH("PredictFluidVel");
    return GC_OK;
}

int gc_cupar_CalBound2Vel(int n, float* d_totalcoor, float* d_velrhop, int* d_cc, int* d_ncube, float* d_outerregion,
                          int* d_sortpart, int* d_beginendcube) {
    if (gc_state().in_fused_step) return GC_OK;
    (void)d_cc; (void)d_ncube; (void)d_outerregion;
    GC_PRE("CalBound2Vel", true);
    if (p.nF == p.nB2) return GC_OK;   // no Bound2 particles
    // The prescribed wall velocity lives in the wall's VelHalf, which the
    // reference sets to zero (src/Particle.cu:513-515).  The reference passes
    // no VelHalf here, so it is taken from the pointer the caller gave to
    // the latest PredictFluidVel / CorrectFliudVel (both precede every
    // CalBound2Vel in src/Particle.cu:1316-1327); without one the walls are
    // at rest.
    return launch_sweep(Bound2VelOp{(float4*)d_velrhop, (const float3*)s.velhalf_ptr}, n, p, d_totalcoor, d_sortpart,
                        d_beginendcube, s.stream, "CalBound2Vel");
}

int gc_cupar_EOS(int n, int* d_sortpart, float* d_velrhop, float* d_press) {
    gc_state().ref.press = d_press;
    if (gc_state().in_fused_step) return GC_OK;
    GC_PRE("EOS", false);
    k_eos<<<nb, SDPDSIZE, 0, s.stream>>>(n, p, d_sortpart, (const float4*)d_velrhop, d_press);
    GC_CHECK_LAUNCH("EOS");
    return GC_OK;
}

int gc_cupar_CalFluidSDPDForce(int n, float* h_sdpdforce, float* d_totalcoor, float* d_velrhop, int* d_cc,
                               int* d_ncube, int* d_sortpart, float* d_outerregion, int* d_beginendcube,
                               float* d_totalforce, float* d_press) {
    if (gc_state().in_fused_step) return GC_OK;
    (void)h_sdpdforce; (void)d_cc; (void)d_ncube; (void)d_outerregion;
    GC_PRE("CalFluidSDPDForce", true);
    const float4* vr = (const float4*)d_velrhop;
    float3* fo = (float3*)d_totalforce;
    if (p.noise_pref > 0.f)
        return launch_sweep(SdpdOp<true>{vr, d_press, fo}, n, p, d_totalcoor, d_sortpart, d_beginendcube, s.stream,
                            "CalFluidSDPDForce");
    return launch_sweep(SdpdOp<false>{vr, d_press, fo}, n, p, d_totalcoor, d_sortpart, d_beginendcube, s.stream,
                        "CalFluidSDPDForce");
}

int gc_cupar_CalFluidRepForce(int n, float* d_totalcoor, int* d_cc, int* d_ncube, int* d_sortpart,
                              float* d_outerregion, int* d_beginendcube, float* d_totalforce) {
    if (gc_state().in_fused_step) return GC_OK;
    (void)d_cc; (void)d_ncube; (void)d_outerregion;
    GC_PRE("CalFluidRepForce", true);
    if (p.nB2 == 0) return GC_OK;   // no Bound1 particles
    return launch_sweep(RepulsionOp{(float3*)d_totalforce}, n, p, d_totalcoor, d_sortpart, d_beginendcube, s.stream,
                        "CalFluidRepForce");
}

int gc_cupar_SetFluidExtForce(int driveon, int n, int* d_sortpart, float* d_totalforce) {
    if (gc_state().in_fused_step) return gc_engine_step(driveon);
    GC_PRE("SetFluidExtForce", false);
    if (!driveon || p.gx == 0.f) return GC_OK;
    k_ext<<<nb, SDPDSIZE, 0, s.stream>>>(n, p, d_sortpart, (float3*)d_totalforce);
    GC_CHECK_LAUNCH("SetFluidExtForce");
    return GC_OK;
}

int gc_cupar_CorrectFliudVel(int n, int* d_sortpart, float* d_totalforce, float* d_velhalf, float* d_velrhop,
                             float* d_totalcoor, int* d_cc, int* d_ncube, float* d_outerregion, int* d_beginendcube) {
    gc_state().ref.velhalf = d_velhalf;
    if (gc_state().in_fused_step) return GC_OK;
    (void)d_totalcoor; (void)d_cc; (void)d_ncube; (void)d_outerregion; (void)d_beginendcube;
    GC_PRE("CorrectFliudVel", false);
    s.velhalf_ptr = d_velhalf;
    k_correct<<<nb, SDPDSIZE, 0, s.stream>>>(n, p, d_sortpart, (const float3*)d_totalforce, (const float3*)d_velhalf,
                                            (float4*)d_velrhop, gc_flags_ptr());
    GC_CHECK_LAUNCH("CorrectFliudVel");
    return GC_OK;
}

int gc_debug_neighbor_stats(int n, float* d_totalcoor, int* d_sortpart, int* d_beginendcube, int* d_count,
                            unsigned long long* d_hash) {
    GC_PRE("debug_neighbor_stats", true);
    return launch_sweep(NeighborOp{d_count, d_hash}, n, p, d_totalcoor, d_sortpart, d_beginendcube, s.stream,
                        "debug_neighbor_stats");
}

}  // extern "C"

