// vbd_scalar.cuh -- the fused colour2 step (vbd_fused.cuh) in scalar FP32 instructions, state in registers: for
// the recorded steps of the adjoint, and for groups of tiles.
//
// Every result equals the paired step's to the bit: each sum below is written with the operands, the order and
// the contractions that the paired form takes for the same slot, so that a checkpoint, a recomputed segment, a
// step, a host frame or several steps of one launch can follow one another in any mix.  One case is left out: the
// recorded step of single tiles with 4 slots a lane sums the force of slots 1 to 3 in an order of its own, which
// its gradients have always had: another rounding of a step moves a stiffness gradient that sits on the kinks of
// the predict's clamp or of the body pass by 1e-5 to 1e-4 of itself.  It is an ulp of the force away.
//
// What it is for.  A group's barriers make the chain of dependent instructions the bound, which the paired form's
// moves between layouts lengthen (launch_scalar_groups has the times of both); and a recorded step is bound by the
// tape it writes.
#pragma once
#include "vbd_fused.cuh"

namespace kami {

__device__ __forceinline__ float3 fma3(float c, float3 a, float3 f) {
    return f3(fmaf(c, a.x, f.x), fmaf(c, a.y, f.y), fmaf(c, a.z, f.z));
}
template <bool Y_FIRST>
__device__ __forceinline__ float scalar_norm2(float3 a) {
    return fmaf(a.z, a.z, Y_FIRST ? fmaf(a.y, a.y, __fmul_rn(a.x, a.x)) : fmaf(a.x, a.x, __fmul_rn(a.y, a.y)));
}
__device__ __forceinline__ float scalar_norm2(float4 a) {
    return fmaf(a.w, a.w, fmaf(a.z, a.z, fmaf(a.x, a.x, __fmul_rn(a.y, a.y))));
}
__device__ __forceinline__ float scalar_short_norm2(float4 a) {
    return fmaf(a.y, a.y, __fmul_rn(a.x, a.x)) + fmaf(a.z, a.z, __fmul_rn(a.w, a.w));
}
// half_axis
template <bool X_FIRST, bool SHORT = false>
__device__ __forceinline__ float3 scalar_axis(float4 q) {
    if (SHORT)
        return f3(fmaf(-q.z, q.z, fmaf(-q.y, q.y, 0.5f)), fmaf(q.w, q.z, __fmul_rn(q.x, q.y)),
                  fmaf(-q.w, q.y, __fmul_rn(q.x, q.z)));
    const float xw = X_FIRST ? fmaf(q.x, q.x, __fmul_rn(q.w, q.w)) : fmaf(q.w, q.w, __fmul_rn(q.x, q.x));
    return f3(0.5f * fmaf(-q.z, q.z, fmaf(-q.y, q.y, xw)), fmaf(q.x, q.y, __fmul_rn(q.w, q.z)),
              fmaf(q.x, q.z, __fmul_rn(-q.w, q.y)));
}

// fused_position.  Neighbour operands from another strand (no segment in between: hn / hp false) are replaced
// by the vertex's own values before they meet their zero coefficient, and vertices that do not move (mov
// false) keep dx, so a non-finite strand cannot leak into the strands or padding that share its tile.
// Strands start at even tile positions, so only the previous neighbour of an even slot and the next
// neighbour of an odd slot can belong to another strand; the others are the same strand or padding (always
// finite), and guard_next / guard_prev say which operands need the replacement.
__device__ __forceinline__ float3 scalar_position(float3 dx, float3 F0, float ddN, float k2N, float3 hN, float3 dxN,
                                                  float ddP, float k2P, float3 hP, float3 dxP, float as_, float isA,
                                                  float isD, bool hn, bool hp, bool mov, bool guard_next,
                                                  bool guard_prev) {
    if (guard_next) dxN = hn ? dxN : dx;
    if (guard_prev) {
        dxP = hp ? dxP : dx;
        hP = hp ? hP : hN;
    }
    const float3 f = fma3(k2P, hP, fma3(-k2N, hN, fma3(-as_, dx, fma3(ddP, dxP, fma3(ddN, dxN, F0)))));
    const float m = ((f.x + f.y) + f.z) * (1.f / 3.f);
    const float3 n = f3(fmaf(m, isD, fmaf(f.x, isA, dx.x)), fmaf(m, isD, fmaf(f.y, isA, dx.y)),
                        fmaf(m, isD, fmaf(f.z, isA, dx.z)));
    return mov ? n : dx;
}

// fused_orientation: pre / nxt say whether the previous / next segment exists, upd whether this segment is
// updated at all; guards as above.  FROM_E: Ve holds the segment vector e instead of m2k e.
template <bool SHORT, bool FROM_E, bool Y_FIRST>
__device__ __forceinline__ void scalar_orientation(float4& q, float3& h, bool upd, bool pre, bool nxt,
                                                   float3 Ve, float m2k, float3 dx, float3 dxN, float4 qPrev,
                                                   float4 qrPrev, float4 qNext, float4 qr, bool guard_prev,
                                                   bool guard_next) {
    const float3 d = dxN - dx;
    const float3 V = FROM_E ? f3(fmaf(m2k, Ve.x, __fmul_rn(m2k, d.x)), fmaf(m2k, Ve.y, __fmul_rn(m2k, d.y)),
                                 fmaf(m2k, Ve.z, __fmul_rn(m2k, d.z)))
                            : fma3(m2k, d, Ve);
    if (guard_prev) qPrev = pre ? qPrev : q;  // operands from another strand never meet arithmetic
    if (guard_next) qNext = nxt ? qNext : q;
    const float4 P1 = qmul_fma(qPrev, qrPrev);
    const float4 P2 = qmul_conj_fma(qNext, qr);
    auto dot = [&](float4 P) {
        return fmaf(q.y, P.y, __fmul_rn(q.x, P.x)) + fmaf(q.z, P.z, __fmul_rn(q.w, P.w));
    };
    float s1 = dot(P1) > 0.f ? 1.f : -1.f;
    float s2 = dot(P2) > 0.f ? 1.f : -1.f;
    s1 = pre ? s1 : 0.f;
    s2 = nxt ? s2 : 0.f;
    const float4 b = make_float4(fmaf(s2, P2.x, __fmul_rn(s1, P1.x)), fmaf(s2, P2.y, __fmul_rn(s1, P1.y)),
                                 fmaf(s2, P2.z, __fmul_rn(s1, P1.z)), fmaf(s2, P2.w, __fmul_rn(s1, P1.w)));
    const float vv = scalar_norm2<Y_FIRST>(V), bb = SHORT ? scalar_short_norm2(b) : scalar_norm2(b);
    const float lambda = SHORT ? sqrt_ftz(vv) + sqrt_ftz(bb)
                               : fmaf(vv, rsqrt_nonneg(vv), __fmul_rn(bb, rsqrt_nonneg(bb)));
    float4 R;  // V (x) b (x) e_x + lambda b
    if (SHORT)
        R = make_float4(fmaf(-V.z, b.z, fmaf(-V.x, b.x, __fmul_rn(-V.y, b.y))),
                        fmaf(b.w, V.z, fmaf(V.x, b.y, __fmul_rn(-b.x, V.y))),
                        fmaf(-b.w, V.y, fmaf(V.x, b.z, __fmul_rn(-b.x, V.z))),
                        fmaf(V.z, b.y, fmaf(-V.x, b.w, __fmul_rn(-V.y, b.z))));
    else
        R = make_float4(fmaf(-V.z, b.z, fmaf(-V.x, b.x, __fmul_rn(-V.y, b.y))),
                        fmaf(b.w, V.z, fmaf(V.x, b.y, __fmul_rn(-b.x, V.y))),
                        fmaf(-b.w, V.y, fmaf(-V.z, b.x, __fmul_rn(b.z, V.x))),
                        fmaf(-b.w, V.x, fmaf(-V.y, b.z, __fmul_rn(b.y, V.z))));
    R = make_float4(fmaf(lambda, b.x, R.x), fmaf(lambda, b.y, R.y), fmaf(lambda, b.z, R.z), fmaf(lambda, b.w, R.w));
    const float inv = rsqrt_ftz(SHORT ? scalar_short_norm2(R) : scalar_norm2(R));
    const float4 n = scale4(inv, R);
    q = upd ? n : q;
    h = scalar_axis<false, SHORT>(q);
}

// RECORD: one step of one substep whose start state and iterates go into the tape too (steps / nsteps are null
// and 1).  HOSTIO: `stage` holds the tile's positions and velocities from the host buffers of `hio`, and the
// step writes its results back through the same area, as fused_step_body does.
template <int C, bool JACOBI, bool GROUPED, bool RECORD, bool HOSTIO>
__device__ __forceinline__ void scalar_step_body(DeviceState st, PhysParams pp, StepParams sp, SdfParams sdf,
                                                 TapeView tp, const StepParams* __restrict__ steps, int nsteps,
                                                 HostIO hio, float* stage, int64_t tile) {
    constexpr bool SHORT = GROUPED;  // the sums of a group's step (vbd_fused.cuh)
    static_assert(!JACOBI || SHORT, "Jacobi on groups only");
    const int lane = threadIdx.x & 31;
    const int64_t base = tile * (32LL * C) + lane;
    // tile groups: neighbours across the warps of the CTA (see GroupExchange)
    const int gw = threadIdx.x >> 5, gK = blockDim.x >> 5;
    GroupExchange* gx = nullptr;
    if constexpr (GROUPED) {
        __shared__ GroupExchange group_exchange;
        gx = &group_exchange;
    }
    auto up_put = [&](int slot, float4 v) {
        if (GROUPED && lane == 31) gx->up[gw][slot] = v;
    };
    auto up_get = [&](int slot, float4 v) { return (GROUPED && lane == 0 && gw > 0) ? gx->up[gw - 1][slot] : v; };
    auto down_put = [&](int slot, float4 v) {
        if (GROUPED && lane == 0) gx->down[gw][slot] = v;
    };
    auto down_get = [&](int slot, float4 v) {
        return (GROUPED && lane == 31 && gw < gK - 1) ? gx->down[gw + 1][slot] : v;
    };
    auto group_sync = [&]() {
        if (GROUPED) __syncthreads();
    };
    auto f4 = [](float3 a) { return make_float4(a.x, a.y, a.z, 0.f); };

    float3 x[C], v[C], vl[C], dx[C], hd[C], F0[C], Ve[C];
    float4 q[C], qr[C];
    float im[C], ddN[C], k2N[C], as_[C], isA[C], isD[C];
    uint32_t fl[C];
    bool mov[C];  // the vertex's position is updated (not pinned, not padding)

#pragma unroll
    for (int k = 0; k < C; k++) {
        const int64_t g = base + 32LL * k;
        const float4 a = st.xm[g];
        x[k] = xyz(a);
        im[k] = a.w;
        v[k] = xyz(st.vel[g]);
        vl[k] = xyz(st.vlast[g]);
        q[k] = st.q[g];
        qr[k] = st.qr[g];
        const float4 p = st.prm[g];
        const float invl = 1.f / p.x;
        const float kk = p.y * invl;
        fl[k] = __float_as_uint(p.w);
        mov[k] = im[k] != 0.f;
        ddN[k] = (fl[k] & F_HAS_NEXT) ? kk * invl : 0.f;
        k2N[k] = (fl[k] & F_HAS_NEXT) ? 2.f * kk : 0.f;
        if (HOSTIO && hio.x_in && (fl[k] & F_VALID)) {  // padding slots keep their device values
            const int o = 3 * (lane * C + k);
            x[k] = f3(stage[o], stage[o + 1], stage[o + 2]);
            v[k] = f3(stage[96 * C + o], stage[96 * C + o + 1], stage[96 * C + o + 2]);
        }
    }
    const int64_t tS = tp.slots;
    const int64_t tslot = base - (RECORD ? tp.tile_begin * 32LL * C : 0);  // this lane's slot in the tape window
    const int64_t tbase = ((int64_t)tp.step * (tp.num_itr + 1)) * tS + tslot;  // tape row of iteration 0
    if (RECORD) {
#pragma unroll
        for (int k = 0; k < C; k++) {
            const int64_t o = (int64_t)tp.step * tS + tslot + 32LL * k;
            tp.x[o] = make_float4(x[k].x, x[k].y, x[k].z, im[k]);
            tp.v[o] = make_float4(v[k].x, v[k].y, v[k].z, 0.f);
            tp.vl[o] = make_float4(vl[k].x, vl[k].y, vl[k].z, 0.f);
        }
    }
    // constants of the previous lane's last segment (segment i-1 of slot 0)
    float4 qrH = shfl_up4(qr[C - 1], 1);
    float ddH = __shfl_up_sync(0xffffffffu, ddN[C - 1], 1);
    float k2H = __shfl_up_sync(0xffffffffu, k2N[C - 1], 1);
    if (GROUPED) {
        up_put(XU_QR, qr[C - 1]);
        up_put(XU_DK, make_float4(ddN[C - 1], k2N[C - 1], 0.f, 0.f));
        group_sync();
        qrH = up_get(XU_QR, qrH);
        const float4 dk = up_get(XU_DK, make_float4(ddH, k2H, 0.f, 0.f));
        ddH = dk.x;
        k2H = dk.y;
    }
    const bool hp0 = fl[0] & F_HAS_PREV;  // (a shuffle gives lane 0 its own values)
    ddH = hp0 ? ddH : 0.f;
    k2H = hp0 ? k2H : 0.f;

    const float accel = pp.accel_ratio;
    bool bad = false;
    for (int step = 0; step < nsteps; step++) {
    if (steps) sp = steps[step];
    const float h = sp.h;
    const float damp = pp.damping / h;

    for (int s = 0; s < sp.substeps; s++) {
        {
            float3 e[C];
#pragma unroll
            for (int k = 0; k < C - 1; k++) e[k] = x[k + 1] - x[k];
            float3 xN0 = shfl_down3(x[0], 1);
            if (GROUPED) {
                down_put(XD_X, f4(x[0]));
                group_sync();
                xN0 = xyz(down_get(XD_X, f4(xN0)));
            }
            e[C - 1] = xN0 - x[C - 1];
#pragma unroll
            for (int k = 0; k < C; k++) e[k] = (fl[k] & F_HAS_NEXT) ? e[k] : f3(0.f, 0.f, 0.f);
            float3 eH = shfl_up3(e[C - 1], 1);
            if (GROUPED) {
                up_put(XU_E, f4(e[C - 1]));
                group_sync();
                eH = xyz(up_get(XU_E, f4(eH)));
            }
            eH = hp0 ? eH : f3(0.f, 0.f, 0.f);
#pragma unroll
            for (int k = 0; k < C; k++) {
                float3 y;
                vbd_predict<C == 4>(x[k], v[k], vl[k], im[k], pp, h, sp.last_h, sp.time, dx[k], y);
                vl[k] = v[k];
                const float ddP = k > 0 ? ddN[k > 0 ? k - 1 : 0] : ddH;
                const float3 eP = k > 0 ? e[k > 0 ? k - 1 : 0] : eH;
                constexpr ForceOrder INNER = RECORD ? HALF_CHAINED : SEPARATE;  // of the slots 1 to 3 of 4
                const bool chained = SHORT || k == 0 || C == 2 || (RECORD && k == C - 1);
                const VertexFold b = chained
                                         ? fold_vertex<CHAINED>(im[k], h, damp, accel, ddN[k], ddP, y, e[k], eP)
                                         : fold_vertex<INNER>(im[k], h, damp, accel, ddN[k], ddP, y, e[k], eP);
                as_[k] = b.as_;
                isA[k] = b.isA;
                isD[k] = b.isD;
                F0[k] = b.F0;
                Ve[k] = C == 2 && k == 0 && !SHORT ? e[k] : -k2N[k] * e[k];
                hd[k] = scalar_axis<true>(q[k]);
            }
        }
        float4 qP = shfl_up4(q[C - 1], 1);
        float3 hP = shfl_up3(hd[C - 1], 1);  // the previous lane's axis
        if (RECORD) {
#pragma unroll
            for (int k = 0; k < C; k++) {
                tp.dx[tbase + 32LL * k] = make_float4(dx[k].x, dx[k].y, dx[k].z, 0.f);
                tp.q[tbase + 32LL * k] = q[k];
            }
        }

        for (int it = 0; it < pp.num_itr; it++) {
            float3 dxP = shfl_up3(dx[C - 1], 1);
            if (GROUPED) {  // the previous lane's last slot, unchanged until the odd sweeps
                up_put(XU_DX, f4(dx[C - 1]));
                up_put(XU_Q, q[C - 1]);
                up_put(XU_D3, f4(hd[C - 1]));
                if (JACOBI) down_put(XD_DX, f4(dx[0]));
                group_sync();
                dxP = xyz(up_get(XU_DX, f4(dxP)));
                qP = up_get(XU_Q, qP);
                hP = xyz(up_get(XU_D3, f4(hP)));
            }
            // slot k's updates from its neighbours' values
            auto position = [&](int k, float3 dN, float3 dP) {
                const int kp = k > 0 ? k - 1 : 0;
                return scalar_position(dx[k], F0[k], ddN[k], k2N[k], hd[k], dN, k ? ddN[kp] : ddH, k ? k2N[kp] : k2H,
                                       k ? hd[kp] : hP, dP, as_[k], isA[k], isD[k], fl[k] & F_HAS_NEXT,
                                       fl[k] & F_HAS_PREV, mov[k], k & 1, !(k & 1));
            };
            auto orientation = [&](float4& n, int k, float3 dN, float4 qp, float4 qn) {
                const int kp = k > 0 ? k - 1 : 0;
                const bool upd = (fl[k] & F_HAS_NEXT) && !(fl[k] & F_FIX_ORIENTATION);
                const bool pre = fl[k] & F_HAS_PREV, nxt = fl[k] & F_HAS_NEXT_ORIENTATION;
                if (k & 1)
                    scalar_orientation<SHORT, false, C == 4 && !JACOBI>(n, hd[k], upd, pre, nxt, Ve[k], -k2N[k],
                                                                        dx[k], dN, qp, qr[kp], qn, qr[k], false, true);
                else
                    scalar_orientation<SHORT, C == 2 && !SHORT, false>(n, hd[k], upd, pre, nxt, Ve[k], -k2N[k],
                                                                       dx[k], dN, qp, k ? qr[kp] : qrH, qn, qr[k], true,
                                                                       false);
            };
            if (!JACOBI) {
                // positions, even slots (neighbours are odd: own registers or the previous lane)
#pragma unroll
                for (int k = 0; k < C; k += 2) dx[k] = position(k, dx[k + 1], k ? dx[k > 0 ? k - 1 : 0] : dxP);
                // positions, odd slots
                float3 dxN0 = shfl_down3(dx[0], 1);
                if (GROUPED) {
                    down_put(XD_DX, f4(dx[0]));
                    group_sync();
                    dxN0 = xyz(down_get(XD_DX, f4(dxN0)));
                }
#pragma unroll
                for (int k = 1; k < C; k += 2)
                    dx[k] = position(k, k == C - 1 ? dxN0 : dx[k + 1 < C ? k + 1 : k], dx[k - 1]);
                // orientations, even segments
#pragma unroll
                for (int k = 0; k < C; k += 2) orientation(q[k], k, dx[k + 1], k ? q[k > 0 ? k - 1 : 0] : qP, q[k + 1]);
                // orientations, odd segments
                float4 qN0 = shfl_down4(q[0], 1);
                if (GROUPED) {
                    down_put(XD_Q, q[0]);
                    group_sync();
                    qN0 = down_get(XD_Q, qN0);
                }
#pragma unroll
                for (int k = 1; k < C; k += 2) {
                    const int kn = k + 1 < C ? k + 1 : k;
                    orientation(q[k], k, k == C - 1 ? dxN0 : dx[kn], q[k - 1], k == C - 1 ? qN0 : q[kn]);
                }
            } else {
                // positions, every slot from the previous sweep
                float3 dxN0 = shfl_down3(dx[0], 1);
                if (GROUPED) dxN0 = xyz(down_get(XD_DX, f4(dxN0)));
                float3 nd[C];
#pragma unroll
                for (int k = 0; k < C; k++)
                    nd[k] = position(k, k == C - 1 ? dxN0 : dx[k + 1 < C ? k + 1 : k], k ? dx[k > 0 ? k - 1 : 0] : dxP);
#pragma unroll
                for (int k = 0; k < C; k++) dx[k] = nd[k];
                // orientations, every segment from the previous sweep
                dxN0 = shfl_down3(dx[0], 1);
                float4 qN0 = shfl_down4(q[0], 1);
                if (GROUPED) {
                    down_put(XD_DX2, f4(dx[0]));
                    down_put(XD_Q, q[0]);
                    group_sync();
                    dxN0 = xyz(down_get(XD_DX2, f4(dxN0)));
                    qN0 = down_get(XD_Q, qN0);
                }
                float4 nq[C];
#pragma unroll
                for (int k = 0; k < C; k++) {
                    const int kn = k + 1 < C ? k + 1 : k;
                    nq[k] = q[k];
                    orientation(nq[k], k, k == C - 1 ? dxN0 : dx[kn], k ? q[k > 0 ? k - 1 : 0] : qP,
                                k == C - 1 ? qN0 : q[kn]);
                }
#pragma unroll
                for (int k = 0; k < C; k++) q[k] = nq[k];
            }
            qP = shfl_up4(q[C - 1], 1);
            hP = shfl_up3(hd[C - 1], 1);
            if (RECORD) {
                const int64_t row = tbase + (int64_t)(it + 1) * tS;
#pragma unroll
                for (int k = 0; k < C; k++) {
                    tp.dx[row + 32LL * k] = make_float4(dx[k].x, dx[k].y, dx[k].z, 0.f);
                    tp.q[row + 32LL * k] = q[k];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < C; k++) vbd_finish(x[k], v[k], dx[k], im[k], h, pp.velocity_decay);
    }
#pragma unroll
    for (int k = 0; k < C; k++) {
        if (sdf.grid && (fl[k] & F_VALID) && !(fl[k] & F_ROOT)) vbd_sdf(x[k], v[k], sdf, sp);
        bad |= !finite3(x[k]) || !finite3(v[k]) || !finite4(q[k]);
    }
    }  // steps

#pragma unroll
    for (int k = 0; k < C; k++) {
        const int64_t g = base + 32LL * k;
        st.xm[g] = make_float4(x[k].x, x[k].y, x[k].z, im[k]);
        st.vel[g] = make_float4(v[k].x, v[k].y, v[k].z, 0.f);
        st.vlast[g] = make_float4(vl[k].x, vl[k].y, vl[k].z, 0.f);
        st.q[g] = q[k];
    }
    if (HOSTIO && hio.x_out) {  // (no output buffers: the results stay on the device)
        __syncwarp();  // every lane has read its staged input
#pragma unroll
        for (int k = 0; k < C; k++) {
            const int o = 3 * (lane * C + k);
            stage[o] = x[k].x;
            stage[o + 1] = x[k].y;
            stage[o + 2] = x[k].z;
            stage[96 * C + o] = v[k].x;
            stage[96 * C + o + 1] = v[k].y;
            stage[96 * C + o + 2] = v[k].z;
        }
        frame_out<C>(hio, tile, stage);
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(st.status, STATUS_NONFINITE);
}

// A recorded step: one warp per tile, or (GROUPED) one CTA of K warps per group of tiles.
template <int C, bool GROUPED>
__global__ void __launch_bounds__(256) recorded_step_kernel(DeviceState st, PhysParams pp, StepParams sp, SdfParams sdf,
                                                            TapeView tp) {
    const int64_t tile = tp.tile_begin + (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (tile >= st.num_tiles) return;  // uniform per warp (per CTA for groups: num_tiles is a multiple of K)
    scalar_step_body<C, false, GROUPED, true, false>(st, pp, sp, sdf, tp, nullptr, 1, HostIO{}, nullptr, tile);
}
// The plain step of groups of tiles, one CTA of K warps per group, from group `first` on.
template <int C>
__global__ void __launch_bounds__(256) scalar_group_kernel(DeviceState st, PhysParams pp, StepParams sp, SdfParams sdf,
                                                           const StepParams* __restrict__ steps, int nsteps, int first) {
    const int64_t tile = (int64_t)(first + blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
    scalar_step_body<C, false, true, false, false>(st, pp, sp, sdf, TapeView{}, steps, nsteps, HostIO{}, nullptr, tile);
}
// The same with resident CTAs that loop over the groups (LAUNCH_PERSISTENT).
template <int C>
__global__ void __launch_bounds__(256) scalar_persistent_group_kernel(DeviceState st, PhysParams pp, StepParams sp,
                                                                      SdfParams sdf,
                                                                      const StepParams* __restrict__ steps, int nsteps) {
    const int K = blockDim.x >> 5;
    for (int u = blockIdx.x; (int64_t)u * K < st.num_tiles; u += gridDim.x) {
        scalar_step_body<C, false, true, false, false>(st, pp, sp, sdf, TapeView{}, steps, nsteps, HostIO{}, nullptr,
                                                       (int64_t)u * K + (threadIdx.x >> 5));
        __syncthreads();  // the group exchange area is reused by the next group
    }
}
// A host frame of the groups [first, last): resident CTAs loop over them, which keeps the SMs evenly filled.  Frames
// of 42 substeps from and to host arrays, colour2 and Jacobi: 900 strands (365 groups) 2.61 and 2.67 ms with a CTA
// for each group, 2.12 and 2.17 looping (2.25 and 2.32 paired); 60 strands 0.78 and 0.78 (0.94 and 0.96 paired).
template <int C, bool JACOBI>
__global__ void __launch_bounds__(256) scalar_frame_group_kernel(DeviceState st, PhysParams pp, StepParams sp,
                                                                 SdfParams sdf, HostIO hio, int first, int last) {
    extern __shared__ float scalar_stage[];
    float* const stage = scalar_stage + (threadIdx.x >> 5) * (6 * 32 * C);
    const int K = blockDim.x >> 5;
    for (int u = first + blockIdx.x; u < last; u += gridDim.x) {
        const int64_t t = (int64_t)u * K + (threadIdx.x >> 5);
        frame_in<C>(hio, t, stage);
        scalar_step_body<C, JACOBI, true, false, true>(st, pp, sp, sdf, TapeView{}, nullptr, 1, hio, stage, t);
        __syncthreads();  // the group exchange and staging areas are reused by the next group
    }
}

}  // namespace kami
