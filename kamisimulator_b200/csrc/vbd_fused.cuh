// vbd_fused.cuh -- the fused step kernel: one warp per tile, all substeps and iterations of one
// KamiSimulator step in registers.
//
// Per substep every slot folds its step-constant terms into a few coefficients, so that an
// iteration only touches the iterated state (dx, q, d3 = q e_x q*):
//   position block (cosseratItr, YarnBall/sim/cosserat.cu:112-161, 246-285), with the segment
//   constraint c = (e + dx_next - dx)/l - d3 expanded,
//     f  = F0 + ddN dx_next + ddP dx_prev - (a + s) dx - kkN d3_i + kkP d3_{i-1}
//     F0 = a y + ddN e_i - ddP e_{i-1},  kk = kStretch / l,  dd = kk / l,  s = (ddN + ddP)(1 + damping/h)
//   (ddN/kkN are zero for a vertex without a next segment, ddP/kkP are the previous slot's),
//   then dx += (f - mean f) accel/s + mean f accel/(s + 3a)   (the exact inverse of a 1 1^T + s I),
//   evaluated as dx + f isA + mean f isD with isA = accel/s, isD = accel/(s + 3a) - isA;
//   orientation (quaternionLambdaItr, cosserat.cu:290-337) with V = -2 kk (e_i + dx_next - dx).
// Missing neighbours enter as zero coefficients, so the iteration loop has no data-dependent branches.
// Sums of two products are written with fmaf, so that each kernel built from this file rounds them as
// written, whatever the compiler would contract.
#pragma once
#include "vbd_math.cuh"

namespace kami {

// PTX rsqrt.approx.ftz.f32: rsqrtf's approximation without the input scaling that the non-ftz form
// adds for subnormal inputs.  Every input here is a normal float, where the two give the same result.
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float rsqrt_nonneg(float x) { return rsqrt_ftz(fmaxf(x, 1e-30f)); }

// The Hamilton product of qmul (vbd_common.cuh) as FMA chains: the same product in 16 instead of
// 20 instructions, rounded differently.  qmul_conj_fma(l, r) = l * conj(r).
__device__ __forceinline__ float4 qmul_fma(float4 l, float4 r) {
    return make_float4(fmaf(l.w, r.x, fmaf(r.w, l.x, fmaf(l.y, r.z, -r.y * l.z))),
                       fmaf(l.w, r.y, fmaf(r.w, l.y, fmaf(l.z, r.x, -r.z * l.x))),
                       fmaf(l.w, r.z, fmaf(r.w, l.z, fmaf(l.x, r.y, -r.x * l.y))),
                       fmaf(l.w, r.w, -fmaf(l.x, r.x, fmaf(l.y, r.y, l.z * r.z))));
}
__device__ __forceinline__ float4 qmul_conj_fma(float4 l, float4 r) {
    return qmul_fma(l, make_float4(-r.x, -r.y, -r.z, r.w));
}

// ---- packed FP32x2 updates (sm_100 FFMA2 / FADD2 / FMUL2) -----------------------------------------
// A paired FP32 instruction does two operations in one issue slot; an operand may be negated, in one half
// or both, or be one half used twice, at no cost, but exchanged halves cost a move.  So a vector keeps y and
// z in one register pair and a quaternion (y, z) and (x, w): a scalar coefficient is a half used twice, and
// the few products that need exchanged halves are scalar instructions.
//
// What bounds an iteration is the register file: three-operand FMAs on distinct registers run at 1.5
// cycles a scheduler (3 packed), multiplications and additions at 1 (2), measured on loops of each.  That
// sum is about 180 cycles a row of 32 slots and iteration, against 115 issue slots and 115 cycles of the FMA
// pipe; the scalar updates before took 175 issue slots and 212 cycles.  Hence the signs of the two
// quaternion products applied once to the result, missing neighbours kept out by the shuffle's source
// lane, and predicated results instead of selects.  Packing two slots of a colour instead (four slots a
// lane, or two tiles a warp) took 91 issue slots but the same register reads, and twice the registers: 101
// us for 10,000 x 64, 20 iterations, against 89 here (99 before).
//
// Rounding.  On single tiles every sum below runs in the order, with the contractions, that this step's
// trajectories have always had, so a groom moves to the same bits: an FP32 velocity is dx / h, and another
// rounding of the iterations comes back in it 1e-5 to 1e-4 large on short strands over a few substeps.
// That order differs between a tile of 2 and of 4 slots a lane, and in the host frame (FROM_E, Y_FIRST,
// WZ_FIRST and the force in fused_step_body).  Groups of tiles (SHORT) take shorter sums and sqrt.approx, in
// every kernel that steps them, a host frame and a recorded step among them: 10.3 ms instead of 10.7 for 6,000
// strands of 100-300 vertices, 42 substeps of 32 iterations, paired (10.9 with the longer sums in scalar
// instructions, 10.2 with these); against 64 bits their positions and orientations err as with the longer sums
// (2.7e-7 and 1.6e-6 relative).  The scalar form of the step (vbd_scalar.cuh) takes the same sums, slot by slot.
struct V3 {
    float x;
    float2 yz;
};
struct Q4 {
    float2 yz, xw;
};
__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, neg2(b)); }
__device__ __forceinline__ V3 v3(float3 a) { return {a.x, make_float2(a.y, a.z)}; }
__device__ __forceinline__ float3 f3(V3 a) { return f3(a.x, a.yz.x, a.yz.y); }
__device__ __forceinline__ Q4 q4(float4 a) { return {make_float2(a.y, a.z), make_float2(a.x, a.w)}; }
__device__ __forceinline__ float4 f4(Q4 a) { return make_float4(a.xw.x, a.yz.x, a.yz.y, a.xw.y); }
__device__ __forceinline__ float4 f4(V3 a) { return make_float4(a.x, a.yz.x, a.yz.y, 0.f); }
__device__ __forceinline__ V3 shfl(V3 a, int lane) {
    return {__shfl_sync(0xffffffffu, a.x, lane),
            make_float2(__shfl_sync(0xffffffffu, a.yz.x, lane), __shfl_sync(0xffffffffu, a.yz.y, lane))};
}
__device__ __forceinline__ Q4 shfl(Q4 a, int lane) {
    return {make_float2(__shfl_sync(0xffffffffu, a.yz.x, lane), __shfl_sync(0xffffffffu, a.yz.y, lane)),
            make_float2(__shfl_sync(0xffffffffu, a.xw.x, lane), __shfl_sync(0xffffffffu, a.xw.y, lane))};
}
template <bool Y_FIRST>
__device__ __forceinline__ float norm2(V3 a) {
    const float t = Y_FIRST ? fmaf(a.yz.x, a.yz.x, __fmul_rn(a.x, a.x)) : fmaf(a.x, a.x, __fmul_rn(a.yz.x, a.yz.x));
    return fmaf(a.yz.y, a.yz.y, t);
}
__device__ __forceinline__ float norm2(Q4 a) {
    return fmaf(a.xw.y, a.xw.y, fmaf(a.yz.y, a.yz.y, fmaf(a.xw.x, a.xw.x, __fmul_rn(a.yz.x, a.yz.x))));
}

__device__ __forceinline__ float short_norm2(Q4 a) {
    const float2 t = fma2(a.yz, a.yz, mul2(a.xw, a.xw));
    return t.x + t.y;
}
// PTX sqrt.approx.ftz.f32 (0 for 0 and for squares of lengths below 1e-19).
__device__ __forceinline__ float sqrt_ftz(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// l r  and  l conj(r): the products that need halves exchanged are written as scalars (an exchanged or
// partly negated pair costs a move and a negation in every iteration)
__device__ __forceinline__ Q4 qmul(Q4 l, Q4 r) {
    const float lx = l.xw.x, ly = l.yz.x, lz = l.yz.y, rx = r.xw.x, ry = r.yz.x, rz = r.yz.y;
    float2 yz = make_float2(fmaf(lz, rx, __fmul_rn(-rz, lx)), fmaf(lx, ry, __fmul_rn(-rx, ly)));
    yz = fma2(both(r.xw.y), l.yz, yz);
    const float2 t = mul2(both(lz), r.yz);
    const float x = fmaf(r.xw.y, lx, fmaf(ly, rz, -t.x));
    const float w = fmaf(lx, rx, fmaf(ly, ry, t.y));
    return {fma2(both(l.xw.y), r.yz, yz), fma2(both(l.xw.y), r.xw, make_float2(x, -w))};
}
__device__ __forceinline__ Q4 qmul_conj(Q4 l, Q4 r) {
    const float lx = l.xw.x, ly = l.yz.x, lz = l.yz.y, rx = r.xw.x, ry = r.yz.x, rz = r.yz.y;
    float2 yz = make_float2(fmaf(-lz, rx, __fmul_rn(rz, lx)), fmaf(-lx, ry, __fmul_rn(rx, ly)));
    yz = fma2(both(r.xw.y), l.yz, yz);
    const float2 t = mul2(both(lz), r.yz);
    const float x = fmaf(r.xw.y, lx, fmaf(-ly, rz, t.x));
    const float w = fmaf(lx, rx, fmaf(ly, ry, t.y));
    return {fma2(both(-l.xw.y), r.yz, yz), make_float2(fmaf(-l.xw.y, rx, x), fmaf(l.xw.y, r.xw.y, w))};
}

// Half the material axis, d3 / 2 = q e_x q* / 2 (d3_of, vbd_common.cuh); the position update's
// coefficient carries the other factor of two.
// SHORT: of a unit quaternion.  It is taken only after an update, which leaves one (a segment that has a next
// vertex is always updated); the axis of an orientation set from outside is the full one.
template <bool X_FIRST, bool WZ_FIRST, bool SHORT = false>
__device__ __forceinline__ V3 half_axis(Q4 q) {
    if (SHORT) {  // (1/2 - y^2 - z^2, x y + w z, x z - w y)
        const float2 t = mul2(both(q.xw.x), q.yz);
        return {fmaf(-q.yz.y, q.yz.y, fmaf(-q.yz.x, q.yz.x, 0.5f)),
                make_float2(fmaf(q.xw.y, q.yz.y, t.x), fmaf(-q.xw.y, q.yz.x, t.y))};
    }
    const float x = q.xw.x, y = q.yz.x, z = q.yz.y, w = q.xw.y;
    const float xw = X_FIRST ? fmaf(x, x, __fmul_rn(w, w)) : fmaf(w, w, __fmul_rn(x, x));
    const float d = 0.5f * fmaf(-z, z, fmaf(-y, y, xw));
    if (WZ_FIRST) return {d, make_float2(fmaf(w, z, __fmul_rn(x, y)), fmaf(x, z, __fmul_rn(-w, y)))};
    return {d, fma2(both(x), q.yz, make_float2(__fmul_rn(w, z), __fmul_rn(-w, y)))};
}

// A vertex's folded coefficients for one substep (see the file comment); zeros for a vertex that does not
// move.  The order of the force's sum differs between the slots of a lane.
enum ForceOrder { CHAINED, HALF_CHAINED, SEPARATE };
struct VertexFold {
    float3 F0;
    float as_, isA, isD;
};
template <ForceOrder ORDER>
__device__ __forceinline__ VertexFold fold_vertex(float im, float h, float damp, float accel, float ddN, float ddP,
                                                  float3 y, float3 e, float3 eP) {
    const float a = im != 0.f ? 1.f / (im * h * h) : 0.f;
    const float sk = __fmul_rn(ddN + ddP, 1.f + damp);
    VertexFold b;
    b.as_ = a + sk;
    b.isA = im != 0.f ? accel / sk : 0.f;
    b.isD = im != 0.f ? accel / fmaf(3.f, a, sk) - b.isA : 0.f;
    auto force = [&](float ya, float en, float ep) {
        const float n = __fmul_rn(ddN, en);  // a segment's product enters both its vertices
        if (ORDER == CHAINED) return fmaf(-ddP, ep, fmaf(a, ya, n));
        return __fsub_rn(ORDER == HALF_CHAINED ? fmaf(a, ya, n) : __fadd_rn(__fmul_rn(a, ya), n), __fmul_rn(ddP, ep));
    };
    b.F0 = f3(force(y.x, e.x, eP.x), force(y.y, e.y, eP.y), force(y.z, e.z, eP.z));
    return b;
}

// One position update with folded coefficients (see the file comment).  k2N / k2P are twice kkN / kkP
// for the halved axes hN / hP.  use_n / use_p: whether the next / previous operands may meet arithmetic at
// all (see fused_step_body); mov: whether the vertex moves.
__device__ __forceinline__ void fused_position(V3& dx, V3 F0, float ddN, float k2N, V3 hN, V3 dxN, float ddP, float k2P,
                                               V3 hP, V3 dxP, float as_, float isA, float isD, bool mov, bool use_n,
                                               bool use_p) {
    V3 f = F0;
    auto add = [&](float c, V3 a) {
        f.x = fmaf(c, a.x, f.x);
        f.yz = fma2(both(c), a.yz, f.yz);
    };
    if (use_n) add(ddN, dxN);
    if (use_p) add(ddP, dxP);
    add(-as_, dx);
    add(-k2N, hN);
    if (use_p) add(k2P, hP);
    const float m = ((f.x + f.yz.x) + f.yz.y) * (1.f / 3.f);
    if (mov) {
        dx.x = fmaf(m, isD, fmaf(f.x, isA, dx.x));
        dx.yz = fma2(both(m), both(isD), fma2(f.yz, both(isA), dx.yz));
    }
}

// One orientation update (quaternionLambdaItr).  qrP and qr are zero where the previous / next segment
// is missing, so its product vanishes.  With the signs s1, s2 of the two products (cosserat.cu:316-335),
// b = s1 P1 + s2 P2 = s1 (P1 + s1 s2 P2), and s1 is applied to the normalised result, which is linear
// in b.  R = V b e_x + lambda b with V = (V, 0), written out.  A dot product of zero (an exact half turn between
// two segments) counts as not positive.  Each sign is a predicate or the sign bit of 0 - dot, whichever leaves
// the shorter step; both bits, s1 s2 as bits and s1 as a predicate, both predicates: 10,000 x 64 (2 slots a
// lane) 94.8, 93.0 and 93.1 us, 2,000 uneven strands in 3 substeps 47.0, 45.4 and 46.7; 3,000 x 96 (4 slots)
// 81.7, 82.4 and 80.3; Jacobi, groups, 5,000 x 200 274 with bits and 308 with predicates.
// FROM_E: the components of Ve (all 3, or x and y) that hold the segment vector e instead of m2k e.
template <bool SHORT, int FROM_E, bool Y_FIRST, bool WZ_FIRST, bool S12_BITS>
__device__ __forceinline__ void fused_orientation(Q4& q, V3& h, bool upd, V3 Ve, float m2k, V3 dx, V3 dxN, Q4 qPrev,
                                                  Q4 qrP, Q4 qNext, Q4 qr, bool use_n, bool use_p) {
    constexpr bool S1_BITS = WZ_FIRST;  // Jacobi
    const V3 d = {dxN.x - dx.x, sub2(dxN.yz, dx.yz)};
    V3 V;
    if (FROM_E == 3)
        V = {fmaf(m2k, Ve.x, __fmul_rn(m2k, d.x)), fma2(both(m2k), Ve.yz, mul2(both(m2k), d.yz))};
    else if (FROM_E == 2)
        V = {fmaf(m2k, Ve.x, __fmul_rn(m2k, d.x)),
             make_float2(fmaf(m2k, Ve.yz.x, __fmul_rn(m2k, d.yz.x)), fmaf(m2k, d.yz.y, Ve.yz.y))};
    else
        V = {fmaf(m2k, d.x, Ve.x), fma2(both(m2k), d.yz, Ve.yz)};
    Q4 P1 = qmul(qPrev, qrP), P2 = qmul_conj(qNext, qr);
    const Q4 zero = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    if (!use_p) P1 = zero;
    if (!use_n) P2 = zero;
    const float2 t1 = fma2(q.yz, P1.yz, mul2(q.xw, P1.xw)), t2 = fma2(q.yz, P2.yz, mul2(q.xw, P2.xw));
    const float dot1 = t1.x + t1.y, dot2 = t2.x + t2.y;
    const bool pos1 = dot1 > 0.f, pos2 = dot2 > 0.f;
    const uint32_t g1 = __float_as_uint(0.f - dot1), g2 = __float_as_uint(0.f - dot2);  // sign bit: positive
    const float s12 = S12_BITS ? __uint_as_float(((g1 ^ g2) & 0x80000000u) | 0x3f800000u) : pos1 == pos2 ? 1.f : -1.f;
    const Q4 b = {fma2(both(s12), P2.yz, P1.yz), fma2(both(s12), P2.xw, P1.xw)};
    const float vv = norm2<Y_FIRST>(V), bb = SHORT ? short_norm2(b) : norm2(b);
    const float lambda = SHORT ? sqrt_ftz(vv) + sqrt_ftz(bb)
                               : fmaf(vv, rsqrt_nonneg(vv), __fmul_rn(bb, rsqrt_nonneg(bb)));
    const float Vx = V.x, Vy = V.yz.x, Vz = V.yz.y, bx = b.xw.x, by = b.yz.x, bz = b.yz.y, bw = b.xw.y;
    Q4 R;
    if (SHORT) {
        R = {fma2(both(Vx), b.yz, mul2(both(-bx), V.yz)), fma2(both(-Vx), b.xw, mul2(both(-Vy), b.yz))};
        R.yz.x = fmaf(bw, Vz, R.yz.x);
        R.yz.y = fmaf(-bw, Vy, R.yz.y);
        R.xw.x = fmaf(-Vz, bz, R.xw.x);
        R.xw.y = fmaf(Vz, by, R.xw.y);
        R = {fma2(both(lambda), b.yz, R.yz), fma2(both(lambda), b.xw, R.xw)};
    } else {
        const float2 Pzy = make_float2(fmaf(bw, Vz, fmaf(Vx, by, __fmul_rn(-bx, Vy))),
                                       fmaf(-bw, Vy, fmaf(-Vz, bx, __fmul_rn(bz, Vx))));
        const float2 Pwx = make_float2(fmaf(-Vz, bz, fmaf(-Vx, bx, __fmul_rn(-Vy, by))),
                                       fmaf(-bw, Vx, fmaf(-Vy, bz, __fmul_rn(by, Vz))));
        R = {fma2(both(lambda), b.yz, Pzy), fma2(both(lambda), b.xw, Pwx)};
    }
    const float inv = rsqrt_ftz(SHORT ? short_norm2(R) : norm2(R));
    const float2 si = both(S1_BITS ? __uint_as_float(__float_as_uint(inv) ^ (~g1 & 0x80000000u)) : pos1 ? inv : -inv);
    if (upd) {
        q.yz = mul2(si, R.yz);
        q.xw = mul2(si, R.xw);
    }
    h = half_axis<false, WZ_FIRST, SHORT>(q);
}

// Values a group's warps hand across their tile boundaries (GROUPED: one CTA of K <= 8 warps per
// group of K tiles, warp w on tile group * K + w): `up` from lane 31 of warp w to lane 0 of warp
// w + 1 (its previous lane), `down` from lane 0 of warp w to lane 31 of warp w - 1 (its next lane).
// Each slot is written once per substep or iteration and read after the __syncthreads that follows;
// the next write to it comes after at least one more __syncthreads, which every reader has passed.
enum : int { XU_QR, XU_DK, XU_E, XU_DX, XU_Q, XU_D3, XU_N };
enum : int { XD_X, XD_DX, XD_Q, XD_DX2, XD_N };
struct GroupExchange {
    float4 up[8][XU_N];
    float4 down[8][XD_N];
};

// A host frame's strands of tile t between the host buffers and the warp's staging area: positions, then
// velocities, 3 floats per tile position p = lane * C + k (coalesced 4-byte accesses over PCIe).
template <int C>
__device__ __forceinline__ void frame_in(const HostIO& hio, int64_t t, float* stage) {
    const int lane = threadIdx.x & 31;
    const int r_end = hio.x_in ? hio.run_begin[t + 1] : 0;
    for (int r = hio.run_begin[t]; r < r_end; r++) {
        const int4 run = hio.runs[r];
        const float* gx = hio.x_in + 3LL * run.y;
        const float* gv = hio.v_in + 3LL * run.y;
        for (int j = lane; j < 3 * run.z; j += 32) {
            stage[3 * run.x + j] = gx[j];
            stage[96 * C + 3 * run.x + j] = gv[j];
        }
    }
    __syncwarp();
}
template <int C>
__device__ __forceinline__ void frame_out(const HostIO& hio, int64_t t, const float* stage) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    const int r_end = hio.run_begin[t + 1];
    for (int r = hio.run_begin[t]; r < r_end; r++) {
        const int4 run = hio.runs[r];
        float* gx = hio.x_out + 3LL * run.y;
        float* gv = hio.v_out + 3LL * run.y;
        for (int j = lane; j < 3 * run.z; j += 32) {
            gx[j] = stage[3 * run.x + j];
            gv[j] = stage[96 * C + 3 * run.x + j];
        }
    }
}

// Floats of shared memory a slot takes in a fused kernel: position, velocity, last velocity, inverse
// mass.  A host frame stages the tile's positions and velocities in the same cells before and after.
enum : int { PARK_X = 0, PARK_V = 3, PARK_VL = 6, PARK_IM = 9, PARK_FLOATS = 10 };
constexpr size_t park_bytes(int C, int warps) { return sizeof(float) * PARK_FLOATS * 32 * (size_t)C * warps; }
enum : uint32_t { F_MOVES = 1u << 31 };  // in the kernels' flags: the vertex has mass

// One launch runs `nsteps` consecutive steps, step j with clock and body transform steps[j] (or
// `sp` when steps is null), keeping the tile's state on chip between them.  HOSTIO steps tile `frame_tile` of
// a host frame (fused_frame_kernel): the warp's shared memory holds the tile's positions then velocities from
// the host buffers of `hio`, 3 floats per tile position p = lane * C + k, and the step writes its results back to the host buffers
// through the same area, as well as to the device state.  Every fused kernel is launched with
// park_bytes(C, warps) of dynamic shared memory.
// EXPLICIT_TILE steps tile `frame_tile` (the persistent kernels' tile loop) instead of the launch's own.
template <int C, bool JACOBI, bool HOSTIO = false, bool GROUPED = false, bool EXPLICIT_TILE = false>
__device__ __forceinline__ void fused_step_body(DeviceState st, PhysParams pp, StepParams sp, SdfParams sdf,
                                                const StepParams* __restrict__ steps, int nsteps,
                                                HostIO hio = HostIO{}, int64_t frame_tile = 0) {
    static_assert(C == 2 || C == 4, "2 or 4 slots per lane");
    constexpr bool SHORT = GROUPED;
    constexpr int FROM_E = SHORT ? 0 : HOSTIO ? 2 : 3;  // see fused_orientation
    const int lane = threadIdx.x & 31;
    const int64_t tile = (HOSTIO || EXPLICIT_TILE) ? frame_tile
                                                   : (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (tile >= st.num_tiles) return;  // uniform per warp (per CTA for groups: num_tiles is a multiple of K)
    const int64_t base = tile * (32LL * C) + lane;

    V3 dx[C], hd[C], F0[C], Ve[C];
    Q4 q[C];
    Q4 qr[C];
    float ddN[C], k2N[C], as_[C], isA[C], isD[C];
    uint32_t fl[C];

    // The step's position, velocities and inverse mass are only needed between the iterations: they stay
    // in this lane's cells of shared memory (PARK_FLOATS a slot), not in registers, during them.
    extern __shared__ float kami_park[];
    float* const warp_park = kami_park + (threadIdx.x >> 5) * (PARK_FLOATS * 32 * C);
    auto cell = [&](int j, int k) -> float& { return warp_park[(j * C + k) * 32 + lane]; };
    auto park3 = [&](int j, int k, float3 a) {
        cell(j, k) = a.x;
        cell(j + 1, k) = a.y;
        cell(j + 2, k) = a.z;
    };
    auto parked3 = [&](int j, int k) { return f3(cell(j, k), cell(j + 1, k), cell(j + 2, k)); };

    {
    float3 x[C], v[C];
    float im[C];
#pragma unroll
    for (int k = 0; k < C; k++) {
        const int64_t g = base + 32LL * k;
        const float4 a = st.xm[g];
        x[k] = xyz(a);
        im[k] = a.w;
        v[k] = xyz(st.vel[g]);
        q[k] = q4(st.q[g]);
        const float4 p = st.prm[g];
        const float invl = 1.f / p.x;
        const float kk = p.y * invl;
        fl[k] = __float_as_uint(p.w) | (im[k] != 0.f ? F_MOVES : 0u);
        ddN[k] = (fl[k] & F_HAS_NEXT) ? kk * invl : 0.f;
        k2N[k] = (fl[k] & F_HAS_NEXT) ? 2.f * kk : 0.f;
        // zero where segment k + 1 has no orientation update to take part in: the segment then adds
        // nothing to its own update, and no other segment's update reads it
        const float4 r = st.qr[g];
        qr[k] = q4((fl[k] & F_HAS_NEXT_ORIENTATION) ? r : make_float4(0.f, 0.f, 0.f, 0.f));
    }
    if (HOSTIO && hio.x_in) {  // (no input buffers: the frame starts from the device state)
#pragma unroll
        for (int k = 0; k < C; k++) {
            if (fl[k] & F_VALID) {  // padding slots keep their device values
                const int o = 3 * (lane * C + k);
                x[k] = f3(warp_park[o], warp_park[o + 1], warp_park[o + 2]);
                v[k] = f3(warp_park[96 * C + o], warp_park[96 * C + o + 1], warp_park[96 * C + o + 2]);
            }
        }
        __syncwarp();  // the staged input is read before its cells are reused
    }
#pragma unroll
    for (int k = 0; k < C; k++) {
        const float3 vl = xyz(st.vlast[base + 32LL * k]);
        park3(PARK_X, k, x[k]);
        park3(PARK_V, k, v[k]);
        park3(PARK_VL, k, vl);
        cell(PARK_IM, k) = im[k];
    }
    }
    // Neighbours across lanes: slot 0's previous slot is the previous lane's last one, slot C - 1's
    // next slot the next lane's first one.  A lane whose neighbour is missing reads its own opposite slot
    // instead, by the shuffle's source lane, so that another strand's values (which may not be finite) never
    // meet arithmetic: with C = 2 that slot is in the same strand (or, in padding, finite), and its
    // coefficients are zero.  With C = 4 it may belong to another strand too, as may the neighbours between
    // slots 1 and 2 of a lane, so there the operands' use is predicated (use_next, use_prev).
    const bool hp0 = fl[0] & F_HAS_PREV, hnL = fl[C - 1] & F_HAS_NEXT, nxL = fl[C - 1] & F_HAS_NEXT_ORIENTATION;
    const int from_prev = hp0 ? (lane - 1) & 31 : lane, from_next = hnL ? (lane + 1) & 31 : lane,
              from_next_q = nxL ? (lane + 1) & 31 : lane;
    auto use_prev = [&](int k) { return C == 2 || (k & 1) || (fl[k] & F_HAS_PREV); };
    auto use_next = [&](int k) { return C == 2 || !(k & 1) || (fl[k] & F_HAS_NEXT); };
    auto use_next_q = [&](int k) { return C == 2 || !(k & 1) || (fl[k] & F_HAS_NEXT_ORIENTATION); };
    // tile groups: neighbours across the warps of the CTA (see GroupExchange)
    const int gw = threadIdx.x >> 5, gK = blockDim.x >> 5;
    GroupExchange* gx = nullptr;
    if constexpr (GROUPED) {
        __shared__ GroupExchange group_exchange;
        gx = &group_exchange;
    }
    const bool take_up = GROUPED && lane == 0 && gw > 0 && hp0, take_down = GROUPED && lane == 31 && gw < gK - 1 && hnL,
               take_down_q = GROUPED && lane == 31 && gw < gK - 1 && nxL;
    auto up_put = [&](int slot, float4 a) {
        if (GROUPED && lane == 31) gx->up[gw][slot] = a;
    };
    auto down_put = [&](int slot, float4 a) {
        if (GROUPED && lane == 0) gx->down[gw][slot] = a;
    };
    auto up_v = [&](int slot, V3 a) { return take_up ? v3(xyz(gx->up[gw - 1][slot])) : a; };
    auto up_q = [&](int slot, Q4 a) { return take_up ? q4(gx->up[gw - 1][slot]) : a; };
    auto down_v = [&](int slot, V3 a) { return take_down ? v3(xyz(gx->down[gw + 1][slot])) : a; };
    auto down_q = [&](int slot, Q4 a) { return take_down_q ? q4(gx->down[gw + 1][slot]) : a; };
    auto group_sync = [&]() {
        if (GROUPED) __syncthreads();
    };
    auto upd = [&](int k) { return (fl[k] & F_HAS_NEXT) && !(fl[k] & F_FIX_ORIENTATION); };
    auto mov = [&](int k) { return (fl[k] & F_MOVES) != 0; };

    // constants of the previous lane's last segment (segment i-1 of slot 0), zero where there is none
    Q4 qrH;
    float ddH, k2H;
    {
        Q4 r = shfl(qr[C - 1], from_prev);
        ddH = __shfl_sync(0xffffffffu, ddN[C - 1], from_prev);
        k2H = __shfl_sync(0xffffffffu, k2N[C - 1], from_prev);
        if (GROUPED) {
            up_put(XU_QR, f4(qr[C - 1]));
            up_put(XU_DK, make_float4(ddN[C - 1], k2N[C - 1], 0.f, 0.f));
            group_sync();
            r = up_q(XU_QR, r);
            const V3 dk = up_v(XU_DK, V3{ddH, make_float2(k2H, 0.f)});
            ddH = dk.x;
            k2H = dk.yz.x;
        }
        qrH = q4(hp0 ? f4(r) : make_float4(0.f, 0.f, 0.f, 0.f));
        ddH = hp0 ? ddH : 0.f;
        k2H = hp0 ? k2H : 0.f;
    }

    const float accel = pp.accel_ratio;
    bool bad = false;
    for (int step = 0; step < nsteps; step++) {
    if (steps) sp = steps[step];
    const float h = sp.h;
    const float damp = pp.damping / h;

    for (int s = 0; s < sp.substeps; s++) {
        {
            float3 x[C], e[C];
#pragma unroll
            for (int k = 0; k < C; k++) x[k] = parked3(PARK_X, k);
#pragma unroll
            for (int k = 0; k < C - 1; k++) e[k] = x[k + 1] - x[k];
            V3 xN0 = shfl(v3(x[0]), from_next);
            if (GROUPED) {
                down_put(XD_X, f4(v3(x[0])));
                group_sync();
                xN0 = down_v(XD_X, xN0);
            }
            e[C - 1] = f3(xN0) - x[C - 1];
#pragma unroll
            for (int k = 0; k < C; k++) e[k] = (fl[k] & F_HAS_NEXT) ? e[k] : f3(0.f, 0.f, 0.f);
            V3 eH = shfl(v3(e[C - 1]), from_prev);
            if (GROUPED) {
                up_put(XU_E, f4(v3(e[C - 1])));
                group_sync();
                eH = up_v(XU_E, eH);
            }
            const float3 e0 = hp0 ? f3(eH) : f3(0.f, 0.f, 0.f);
#pragma unroll
            for (int k = 0; k < C; k++) {
                float3 dx0, y;
                const float3 v = parked3(PARK_V, k);
                const float im = cell(PARK_IM, k);
                vbd_predict<C == 4>(x[k], v, parked3(PARK_VL, k), im, pp, h, sp.last_h, sp.time, dx0, y);
                park3(PARK_VL, k, v);
                dx[k] = v3(dx0);
                const float ddP = k > 0 ? ddN[k > 0 ? k - 1 : 0] : ddH;
                const float3 eP = k > 0 ? e[k > 0 ? k - 1 : 0] : e0;
                const VertexFold b = SHORT || k == 0 || (C == 2 && !HOSTIO)
                                         ? fold_vertex<CHAINED>(im, h, damp, accel, ddN[k], ddP, y, e[k], eP)
                                         : fold_vertex<SEPARATE>(im, h, damp, accel, ddN[k], ddP, y, e[k], eP);
                as_[k] = b.as_;
                isA[k] = b.isA;
                isD[k] = b.isD;
                F0[k] = v3(b.F0);
                const float3 ve = -k2N[k] * e[k];
                Ve[k] = v3(C == 2 && k == 0 && FROM_E ? f3(e[k].x, e[k].y, FROM_E == 3 ? e[k].z : ve.z) : ve);
                hd[k] = half_axis<true, false>(q[k]);
            }
        }
        auto position = [&](V3& d, int k, V3 dN, V3 dP, V3 hP) {
            const int kp = k > 0 ? k - 1 : 0;
            fused_position(d, F0[k], ddN[k], k2N[k], hd[k], dN, k ? ddN[kp] : ddH, k ? k2N[kp] : k2H, hP, dP, as_[k],
                           isA[k], isD[k], mov(k), use_next(k), use_prev(k));
        };
        auto orientation = [&](Q4& n, V3& hn, int k, V3 dN, Q4 qP, Q4 qN) {
            const int kp = k > 0 ? k - 1 : 0;
            constexpr bool Y_FIRST = !JACOBI;  // of the odd slots of 4
            constexpr bool BITS = (C == 2 && !SHORT) || JACOBI;
            if (C == 2 && k == 0)
                fused_orientation<SHORT, FROM_E, false, JACOBI, BITS>(n, hn, upd(k), Ve[k], -k2N[k], dx[k], dN, qP, qrH,
                                                                      qN, qr[k], use_next_q(k), use_prev(k));
            else if (C == 4 && (k & 1))
                fused_orientation<SHORT, 0, Y_FIRST, JACOBI, BITS>(n, hn, upd(k), Ve[k], -k2N[k], dx[k], dN, qP, qr[kp],
                                                                   qN, qr[k], use_next_q(k), use_prev(k));
            else
                fused_orientation<SHORT, 0, false, JACOBI, BITS>(n, hn, upd(k), Ve[k], -k2N[k], dx[k], dN, qP,
                                                                 k ? qr[kp] : qrH, qN, qr[k], use_next_q(k),
                                                                 use_prev(k));
        };
        Q4 qP = shfl(q[C - 1], from_prev);
        V3 hP = shfl(hd[C - 1], from_prev);  // the previous lane's half axis
        for (int it = 0; it < pp.num_itr; it++) {
            V3 dxP = shfl(dx[C - 1], from_prev);
            if (GROUPED) {  // the previous lane's last slot, unchanged until the odd sweeps
                up_put(XU_DX, f4(dx[C - 1]));
                up_put(XU_Q, f4(q[C - 1]));
                up_put(XU_D3, f4(hd[C - 1]));
                if (JACOBI) down_put(XD_DX, f4(dx[0]));
                group_sync();
                dxP = up_v(XU_DX, dxP);
                qP = up_q(XU_Q, qP);
                hP = up_v(XU_D3, hP);
            }
            if (!JACOBI) {
                // positions, even slots (neighbours are odd: own registers or the previous lane)
#pragma unroll
                for (int k = 0; k < C; k += 2) {
                    const int kp = k > 0 ? k - 1 : 0;
                    position(dx[k], k, dx[k + 1], k ? dx[kp] : dxP, k ? hd[kp] : hP);
                }
                // positions, odd slots
                V3 dxN = shfl(dx[0], from_next);
                if (GROUPED) {
                    down_put(XD_DX, f4(dx[0]));
                    group_sync();
                    dxN = down_v(XD_DX, dxN);
                }
#pragma unroll
                for (int k = 1; k < C; k += 2)
                    position(dx[k], k, k == C - 1 ? dxN : dx[k + 1 < C ? k + 1 : k], dx[k - 1], hd[k - 1]);
                // orientations, even segments
#pragma unroll
                for (int k = 0; k < C; k += 2)
                    orientation(q[k], hd[k], k, dx[k + 1], k ? q[k > 0 ? k - 1 : 0] : qP, q[k + 1]);
                // orientations, odd segments
                Q4 qN = shfl(q[0], from_next_q);
                if (GROUPED) {
                    down_put(XD_Q, f4(q[0]));
                    group_sync();
                    qN = down_q(XD_Q, qN);
                }
#pragma unroll
                for (int k = 1; k < C; k += 2) {
                    const int kn = k + 1 < C ? k + 1 : k;
                    orientation(q[k], hd[k], k, k == C - 1 ? dxN : dx[kn], q[k - 1], k == C - 1 ? qN : q[kn]);
                }
            } else {
                // positions, every slot from the previous sweep
                V3 dxN = shfl(dx[0], from_next);
                if (GROUPED) dxN = down_v(XD_DX, dxN);
                V3 nd[C];
#pragma unroll
                for (int k = 0; k < C; k++) {
                    const int kp = k > 0 ? k - 1 : 0, kn = k + 1 < C ? k + 1 : k;
                    nd[k] = dx[k];
                    position(nd[k], k, k == C - 1 ? dxN : dx[kn], k ? dx[kp] : dxP, k ? hd[kp] : hP);
                }
#pragma unroll
                for (int k = 0; k < C; k++) dx[k] = nd[k];
                // orientations, every segment from the previous sweep
                dxN = shfl(dx[0], from_next);
                Q4 qN = shfl(q[0], from_next_q);
                if (GROUPED) {
                    down_put(XD_DX2, f4(dx[0]));
                    down_put(XD_Q, f4(q[0]));
                    group_sync();
                    dxN = down_v(XD_DX2, dxN);
                    qN = down_q(XD_Q, qN);
                }
                Q4 nq[C];
#pragma unroll
                for (int k = 0; k < C; k++) {
                    const int kp = k > 0 ? k - 1 : 0, kn = k + 1 < C ? k + 1 : k;
                    nq[k] = q[k];
                    orientation(nq[k], hd[k], k, k == C - 1 ? dxN : dx[kn], k ? q[kp] : qP, k == C - 1 ? qN : q[kn]);
                }
#pragma unroll
                for (int k = 0; k < C; k++) q[k] = nq[k];
            }
            qP = shfl(q[C - 1], from_prev);
            hP = shfl(hd[C - 1], from_prev);
        }
        asm volatile("" ::: "memory");  // the parked values are read back, not kept in registers meanwhile
#pragma unroll
        for (int k = 0; k < C; k++) {
            float3 x = parked3(PARK_X, k), v = parked3(PARK_V, k);
            vbd_finish(x, v, f3(dx[k]), cell(PARK_IM, k), h, pp.velocity_decay);
            park3(PARK_X, k, x);
            park3(PARK_V, k, v);
        }
    }
#pragma unroll
    for (int k = 0; k < C; k++) {
        float3 x = parked3(PARK_X, k), v = parked3(PARK_V, k);
        if (sdf.grid && (fl[k] & F_VALID) && !(fl[k] & F_ROOT)) {
            vbd_sdf(x, v, sdf, sp);
            park3(PARK_X, k, x);
            park3(PARK_V, k, v);
        }
        bad |= !finite3(x) || !finite3(v) || !finite4(f4(q[k]));
    }
    }  // steps

    float3 x[C], v[C];
#pragma unroll
    for (int k = 0; k < C; k++) {
        const int64_t g = base + 32LL * k;
        x[k] = parked3(PARK_X, k);
        v[k] = parked3(PARK_V, k);
        const float3 vl = parked3(PARK_VL, k);
        st.xm[g] = make_float4(x[k].x, x[k].y, x[k].z, cell(PARK_IM, k));
        st.vel[g] = make_float4(v[k].x, v[k].y, v[k].z, 0.f);
        st.vlast[g] = make_float4(vl.x, vl.y, vl.z, 0.f);
        st.q[g] = f4(q[k]);
    }
    if (HOSTIO && hio.x_out) {  // (no output buffers: the results stay on the device)
        float* const sx = warp_park;
        float* const sv = warp_park + 96 * C;
        __syncwarp();  // every lane has read its cells
#pragma unroll
        for (int k = 0; k < C; k++) {
            const int o = 3 * (lane * C + k);
            sx[o] = x[k].x;
            sx[o + 1] = x[k].y;
            sx[o + 2] = x[k].z;
            sv[o] = v[k].x;
            sv[o + 1] = v[k].y;
            sv[o + 2] = v[k].z;
        }
        frame_out<C>(hio, tile, sx);
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(st.status, STATUS_NONFINITE);
}

template <int C, bool JACOBI>
__global__ void __launch_bounds__(256) fused_step_kernel(DeviceState st, PhysParams pp, StepParams sp, SdfParams sdf,
                                                         const StepParams* __restrict__ steps, int nsteps) {
    fused_step_body<C, JACOBI>(st, pp, sp, sdf, steps, nsteps);
}

// ---- host frames: one launch uploads, steps and downloads ---------------------------------------------

// One upload-step-download frame in one launch: each warp copies its tile's strands from the host
// buffers into its staging area (6 * 32C floats of dynamic shared memory; coalesced 4-byte loads
// over PCIe), steps the tile and writes it back (fused_step_body, HOSTIO).  The waves of tiles keep
// the host reads of one wave apart from the host writes of the wave before, which is faster here
// than interleaving them: SM-issued reads and writes over PCIe slow each other down.
template <int C, bool JACOBI, bool GROUPED = false>
__device__ __forceinline__ void fused_frame(DeviceState st, PhysParams pp, StepParams sp, SdfParams sdf, HostIO hio) {
    extern __shared__ float kami_park[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + w;
    if (t >= st.num_tiles) return;  // uniform per warp (per CTA for groups)
    float* const stage = kami_park + w * (PARK_FLOATS * 32 * C);
    frame_in<C>(hio, t, stage);
    fused_step_body<C, JACOBI, true, GROUPED>(st, pp, sp, sdf, nullptr, 1, hio, t);
}
template <int C, bool JACOBI>
__global__ void __launch_bounds__(256) fused_frame_kernel(DeviceState st, PhysParams pp, StepParams sp, SdfParams sdf,
                                                          HostIO hio) {
    fused_frame<C, JACOBI>(st, pp, sp, sdf, hio);
}
template <int C, bool JACOBI>
__global__ void __maxnreg__(120) fused_frame_kernel_r120(DeviceState st, PhysParams pp, StepParams sp, SdfParams sdf,
                                                        HostIO hio) {
    fused_frame<C, JACOBI>(st, pp, sp, sdf, hio);
}
// The same over groups of tiles (4 slots a lane: scalar_frame_group_kernel): one CTA of K warps per group.
template <int C, bool JACOBI>
__global__ void __launch_bounds__(256) fused_frame_group_kernel(DeviceState st, PhysParams pp, StepParams sp,
                                                                SdfParams sdf, HostIO hio) {
    fused_frame<C, JACOBI, true>(st, pp, sp, sdf, hio);
}

// The step with 4 slots per lane at most 168 registers per thread (a few bytes of spills): 12 instead
// of 8 warps share an SM, which hides more of the colour sweeps' dependency latency.
template <int C, bool JACOBI>
__global__ void __maxnreg__(168) fused_step_kernel_r168(DeviceState st, PhysParams pp, StepParams sp, SdfParams sdf,
                                                       const StepParams* __restrict__ steps, int nsteps) {
    fused_step_body<C, JACOBI>(st, pp, sp, sdf, steps, nsteps);
}

// The step over groups of K tiles (strands longer than a tile): one CTA of K warps per group, plain
// and with the register caps of the single-tile variants.
template <int C, bool JACOBI>
__global__ void __launch_bounds__(256) fused_group_kernel(DeviceState st, PhysParams pp, StepParams sp, SdfParams sdf,
                                                          const StepParams* __restrict__ steps, int nsteps) {
    fused_step_body<C, JACOBI, false, true>(st, pp, sp, sdf, steps, nsteps);
}
template <int C, bool JACOBI>
__global__ void __maxnreg__(120) fused_group_kernel_r120(DeviceState st, PhysParams pp, StepParams sp, SdfParams sdf,
                                                        const StepParams* __restrict__ steps, int nsteps) {
    fused_step_body<C, JACOBI, false, true>(st, pp, sp, sdf, steps, nsteps);
}
template <int C, bool JACOBI>
__global__ void __maxnreg__(168) fused_group_kernel_r168(DeviceState st, PhysParams pp, StepParams sp, SdfParams sdf,
                                                        const StepParams* __restrict__ steps, int nsteps) {
    fused_step_body<C, JACOBI, false, true>(st, pp, sp, sdf, steps, nsteps);
}

// The same step with at most 120 registers per thread, so 17 warps (instead of 16) share an SM: a
// launch whose tile count is just above a multiple of 16 warps per SM then needs one wave less.
template <int C, bool JACOBI>
__global__ void __maxnreg__(120) fused_step_kernel_r120(DeviceState st, PhysParams pp, StepParams sp, SdfParams sdf,
                                                       const StepParams* __restrict__ steps, int nsteps) {
    fused_step_body<C, JACOBI>(st, pp, sp, sdf, steps, nsteps);
}

// ---- persistent form ----------------------------------------------------------------------------
// A grid of at most as many CTAs as stay resident: CTA b's warp w steps tiles u * W + w for
// u = b, b + gridDim.x, ... (W warps per CTA), or, for groups of K tiles (GROUPED, W = K), the groups
// b, b + gridDim.x, ...  With the grid at the resident count, the SMs' shares differ by one unit.
template <int C, bool JACOBI, bool GROUPED>
__device__ __forceinline__ void fused_persistent(DeviceState st, PhysParams pp, StepParams sp, SdfParams sdf,
                                                 const StepParams* __restrict__ steps, int nsteps) {
    // only the 32-bit unit index stays live across the step body (register pressure)
    for (int u = blockIdx.x; (int64_t)u * (blockDim.x >> 5) < st.num_tiles; u += gridDim.x) {
        fused_step_body<C, JACOBI, false, GROUPED, true>(
            st, pp, sp, sdf, steps, nsteps, HostIO{}, (int64_t)u * (blockDim.x >> 5) + (threadIdx.x >> 5));
        if (GROUPED) __syncthreads();  // the group exchange area is reused by the next group
    }
}
template <int C, bool JACOBI>
__global__ void __launch_bounds__(256) fused_persistent_kernel(DeviceState st, PhysParams pp, StepParams sp,
                                                               SdfParams sdf, const StepParams* __restrict__ steps,
                                                               int nsteps) {
    fused_persistent<C, JACOBI, false>(st, pp, sp, sdf, steps, nsteps);
}
template <int C, bool JACOBI>
__global__ void __maxnreg__(120) fused_persistent_kernel_r120(DeviceState st, PhysParams pp, StepParams sp,
                                                              SdfParams sdf, const StepParams* __restrict__ steps,
                                                              int nsteps) {
    fused_persistent<C, JACOBI, false>(st, pp, sp, sdf, steps, nsteps);
}
template <int C, bool JACOBI>
__global__ void __maxnreg__(168) fused_persistent_kernel_r168(DeviceState st, PhysParams pp, StepParams sp,
                                                              SdfParams sdf, const StepParams* __restrict__ steps,
                                                              int nsteps) {
    fused_persistent<C, JACOBI, false>(st, pp, sp, sdf, steps, nsteps);
}
template <int C, bool JACOBI>
__global__ void __launch_bounds__(256) fused_persistent_group_kernel(DeviceState st, PhysParams pp, StepParams sp,
                                                                     SdfParams sdf, const StepParams* __restrict__ steps,
                                                                     int nsteps) {
    fused_persistent<C, JACOBI, true>(st, pp, sp, sdf, steps, nsteps);
}
template <int C, bool JACOBI>
__global__ void __maxnreg__(120) fused_persistent_group_kernel_r120(DeviceState st, PhysParams pp, StepParams sp,
                                                                    SdfParams sdf,
                                                                    const StepParams* __restrict__ steps, int nsteps) {
    fused_persistent<C, JACOBI, true>(st, pp, sp, sdf, steps, nsteps);
}
template <int C, bool JACOBI>
__global__ void __maxnreg__(168) fused_persistent_group_kernel_r168(DeviceState st, PhysParams pp, StepParams sp,
                                                                    SdfParams sdf,
                                                                    const StepParams* __restrict__ steps, int nsteps) {
    fused_persistent<C, JACOBI, true>(st, pp, sp, sdf, steps, nsteps);
}

}  // namespace kami
