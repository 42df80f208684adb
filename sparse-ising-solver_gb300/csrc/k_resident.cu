// k_resident.cu -- resident MaxCut SB kernels: one CTA owns KA agents of every
// row and keeps their x, y and sign words on chip for all the steps of a
// launch.  Agents never interact (the product J.X couples rows of one agent
// only), so a CTA needs no other CTA between steps: one __syncthreads() per
// step separates the writes of the sign words of step k from their reads in
// step k+1 (double-buffered), which is the Jacobi order of the reference
// kernel (src/kernels.cu:211-269).
//
// k_res8 (8 agents, the kernel's own choice).  Thread t owns the slots t,
// t + T, ... of the degree-sorted rows.  The matrix is read in sliced form (engine.h, DevSell),
// so a warp's four entries per row are one coalesced 256-byte load; read row
// by row from the CSR, every entry was 32 cache lines per warp and the loads
// bounded the kernel (er800: 8.6 us a step).  A row's signs are one word of
// eight nibbles, agent j in nibble 2 j (j < 4) or 2 (j - 4) + 1, one bit
// each.  +-1 weights: the words (XORed with the weight's sign) add up as
// nibble counters, widened to bytes every 12 entries -- one shared load and
// about four instructions per neighbour for 8 agents.  Other weights: the
// sign bits go into the weight's top byte (one XOR for four agents, one PRMT
// per agent), summed in FP32 in the row's order.
// Bound: issue, and the bank conflicts of the gather.
//
// k_resident (16 or 32 agents, when asked for).  Force for +-1 weights: the
// neighbour's sign word (KA bits) XOR the weight's sign gives the negative
// products; their per-agent counts are kept 8 agents at a time in byte lanes
// of two 32-bit registers (a 4-bit nibble times 0x00204081 spreads its bits
// to bit 0 of four bytes).  Rows are visited in degree order (perm).
#include "k_step.cuh"

#include <algorithm>

namespace sbx {

namespace {

struct ResP {
    const int32_t *__restrict__ rowptr;
    const uint32_t *__restrict__ colw;
    const float *__restrict__ valf;
    const int32_t *__restrict__ perm;
    const float4 *__restrict__ coef;    // per step: k1, k2 (clamped), k1, k2 (raw)
    void *x, *y;                        // global [n][Ap]
    uint32_t *Wp, *fin;                 // global planes [n][W]
    int32_t *stab;
    uint8_t *bif, *prev;
    int32_t *ctl;
    int32_t *wincount;                  // bifurcated agents after each window
    int64_t n;
    int32_t A, Ap, W, period, threshold, uw, fused;
    int32_t step0, nsteps, first, unit;
    float c0;
};

__device__ __forceinline__ uint32_t spread4(uint32_t nib) { return (nib * 0x00204081u) & 0x01010101u; }

// Merge `bits` (KA wide, at bit offset sh) into a shared global plane word.
template <int KA>
__device__ __forceinline__ void plane_put(uint32_t *p, uint32_t bits, int sh)
{
    if constexpr (KA == 32) {
        *p = bits;
    } else {
        const uint32_t m = ((1u << KA) - 1u) << sh;
        atomicAnd(p, ~m);
        atomicOr(p, (bits << sh) & m);
    }
}

template <class T, int KA>
__global__ void __launch_bounds__(1024) k_resident(const ResP P)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int64_t n = P.n;
    T *xs = (T *)smem;
    T *ys = xs + n * KA;
    uint32_t *S0 = (uint32_t *)(ys + n * KA);
    uint32_t *S1 = S0 + n;
    uint32_t *Wps = S1 + n;
    __shared__ uint32_t s_chg, s_new, s_stop;
    __shared__ int32_t s_stab[KA];
    __shared__ uint8_t s_bif[KA], s_prev[KA];

    pdl_wait();
    const int tid = threadIdx.x, T_ = blockDim.x;
    const int a0 = blockIdx.x * KA;          // first agent of this CTA
    const int wg = a0 >> 5, sh = a0 & 31;    // its word and bit offset in planes
    T *xg = (T *)P.x, *yg = (T *)P.y;

    // Early exit of the update-window mode (src/ising.cu:200-211): the
    // previous window left every agent bifurcated.
    if (tid == 0) {
        s_stop = P.ctl[CTL_STOP];
        if (!s_stop && P.uw && P.step0 > 0) {
            const int widx = P.step0 / P.period - 1;
            if (P.wincount[widx] == P.A) s_stop = 1;
        }
        s_chg = 0;
    }
    if (tid < KA) {
        const int a = a0 + tid;
        s_stab[tid] = P.stab[a];
        s_bif[tid] = P.bif[a];
        s_prev[tid] = P.prev[a];
    }
    __syncthreads();
    if (s_stop) {
        if (blockIdx.x == 0 && tid == 0) P.ctl[CTL_STOP] = 1;
        return;
    }

    // Load the state; build the sign words of the step about to run.
    const int32_t k0 = P.step0;
    uint32_t *Scur = (k0 & 1) ? S1 : S0;
    for (int64_t r = tid; r < n; r += T_) {
        uint32_t bits = 0;
        const float4 cu = P.coef[k0];
#pragma unroll
        for (int q = 0; q < KA; q++) {
            float x = St<T>::ld(xg[r * P.Ap + a0 + q]);
            float y = St<T>::ld(yg[r * P.Ap + a0 + q]);
            if (P.first) {   // the pre-step Update_XY at step 0 (src/ising.cu:188)
                y = y + cu.w * x;
                x = x + cu.z * y;
            }
            if (!P.fused) {  // the unfused step begins with Update_XY(k0)
                y = y + cu.w * x;
                x = x + cu.z * y;
            }
            T xt = St<T>::st(x), yt = St<T>::st(y);
            xs[r * KA + q] = xt;
            ys[r * KA + q] = yt;
            bits |= sbit(St<T>::ld(xt)) << q;
        }
        Scur[r] = bits;
        Wps[r] = (P.Wp[r * P.W + wg] >> sh) & (KA == 32 ? 0xffffffffu : ((1u << KA) - 1u));
    }
    __syncthreads();

    for (int32_t it = 0; it < P.nsteps; it++) {
        const int32_t k = k0 + it;
        const uint32_t *Sin = (k & 1) ? S1 : S0;
        uint32_t *Snx = (k & 1) ? S0 : S1;
        const bool win = ((k + 1) % P.period) == 0;
        const bool last = it == P.nsteps - 1;
        const float4 ck = P.coef[k];
        const float4 cn = P.coef[k + 1];
        uint32_t chg = 0;
        for (int64_t i = tid; i < n; i += T_) {
            const int32_t r = P.perm[i];
            const int32_t e0 = P.rowptr[r], e1 = P.rowptr[r + 1];
            const int deg = e1 - e0;
            uint32_t nbits = 0, wbits = 0;
#pragma unroll
            for (int g = 0; g < KA / 8; g++) {
                int cnt[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                float ftot[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                if (P.unit) {
                    for (int32_t base = e0; base < e1; base += 255) {
                        const int32_t end = min(e1, base + 255);
                        uint32_t lo = 0, hi = 0;
#pragma unroll 4
                        for (int32_t e = base; e < end; e++) {
                            const uint32_t cw = __ldg(&P.colw[e]);
                            uint32_t wd = Sin[cw & 0x7fffffffu] >> (8 * g);
                            wd ^= 0u - (cw >> 31);
                            lo += spread4(wd & 0xfu);
                            hi += spread4((wd >> 4) & 0xfu);
                        }
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            cnt[q] += (lo >> (8 * q)) & 0xffu;
                            cnt[4 + q] += (hi >> (8 * q)) & 0xffu;
                        }
                    }
                } else {
                    for (int32_t e = e0; e < e1; e++) {
                        const uint32_t cw = __ldg(&P.colw[e]);
                        const float v = __ldg(&P.valf[e]);
                        const uint32_t wd = Sin[cw & 0x7fffffffu] >> (8 * g);
#pragma unroll
                        for (int q = 0; q < 8; q++) ftot[q] -= ((wd >> q) & 1u) ? -v : v;
                    }
                }
#pragma unroll
                for (int q8 = 0; q8 < 8; q8++) {
                    const int q = g * 8 + q8;
                    const float total = P.unit ? (float)(2 * cnt[q8] - deg) : ftot[q8];
                    float x = St<T>::ld(xs[(int64_t)r * KA + q]);
                    float y = St<T>::ld(ys[(int64_t)r * KA + q]);
                    if (P.fused) {
                        // src/kernels.cu:236-262
                        if (fabsf(x) > 1.f) {
                            x = spin_of(x);
                            y = 0.f;
                        } else {
                            y = y + P.c0 * total;
                        }
                        x = x + ck.x * y;
                        y = y + ck.y * x;
                        wbits |= sbit(x) << q;
                    } else {
                        // mat_mult + confine of step k (src/kernels.cu:150-209);
                        // the window sees x here; then Update_XY of step k+1
                        // unless the launch ends with this step.
                        y = y + P.c0 * total;
                        if (fabsf(x) > 1.f) {
                            x = spin_of(x);
                            y = 0.f;
                        }
                        wbits |= sbit(x) << q;
                        if (!last) {
                            y = y + cn.w * x;
                            x = x + cn.z * y;
                        }
                    }
                    nbits |= sbit(x) << q;
                    xs[(int64_t)r * KA + q] = St<T>::st(x);
                    ys[(int64_t)r * KA + q] = St<T>::st(y);
                }
            }
            if (win) {
                chg |= wbits ^ Wps[r];
                Wps[r] = wbits;
            }
            Snx[r] = nbits;
        }
        if (win) {
            // Per-agent window bookkeeping inside the CTA, src/kernels.cu:46-79.
            chg = __reduce_or_sync(FULL, chg);
            if ((tid & 31) == 0 && chg) atomicOr(&s_chg, chg);
            __syncthreads();
            if (tid < KA) {
                const int a = a0 + tid;
                const bool equal = !((s_chg >> tid) & 1u);
                const bool nb = !s_bif[tid];
                int s = s_stab[tid];
                s += (equal && nb);
                s = (!equal && nb) ? 0 : s;
                const bool b = (s == P.threshold - 1);
                const bool newb = b ^ (s_prev[tid] != 0);
                s_prev[tid] = b;
                s_bif[tid] = b;
                s_stab[tid] = s;
                const uint32_t nm = __ballot_sync((KA == 32) ? FULL : ((1u << KA) - 1u), newb && a < P.A);
                const uint32_t bm = __ballot_sync((KA == 32) ? FULL : ((1u << KA) - 1u), b && a < P.A);
                if (tid == 0) {
                    s_new = nm;
                    if (P.uw) atomicAdd(&P.wincount[(k + 1) / P.period - 1], __popc(bm));
                }
            }
            __syncthreads();
            if (s_new) {
                for (int64_t r = tid; r < n; r += T_) {
                    uint32_t *p = &P.fin[r * P.W + wg];
                    const uint32_t m = s_new << sh;
                    if (KA == 32) *p = (*p & ~m) | (Wps[r] & s_new);
                    else {
                        atomicAnd(p, ~m);
                        atomicOr(p, (Wps[r] & s_new) << sh);
                    }
                }
            }
            if (tid == 0) s_chg = 0;
        }
        __syncthreads();
    }

    // Write the state back (chunked runs continue from it; get_state reads it).
    for (int64_t r = tid; r < n; r += T_) {
#pragma unroll
        for (int q = 0; q < KA; q++) {
            xg[r * P.Ap + a0 + q] = xs[r * KA + q];
            yg[r * P.Ap + a0 + q] = ys[r * KA + q];
        }
        plane_put<KA>(&P.Wp[r * P.W + wg], Wps[r], sh);
    }
    if (tid < KA) {
        const int a = a0 + tid;
        P.stab[a] = s_stab[tid];
        P.bif[a] = s_bif[tid];
        P.prev[a] = s_prev[tid];
    }
    if (blockIdx.x == 0 && tid == 0) {
        P.ctl[CTL_STEP] = P.step0 + P.nsteps;
        P.ctl[CTL_WINDOWS] = (P.step0 + P.nsteps) / P.period;
    }
}

// ---- 8 agents per CTA

struct Res8P {
    ResP r;
    const int2 *__restrict__ off;      // sliced matrix (engine.h, DevSell)
    const float *__restrict__ deg;
    const uint2 *__restrict__ col;
    const float4 *__restrict__ val;
    int32_t allpos;
};

// A row's x, y of 8 agents: FP32 values, or packed 16-bit pairs.
template <class T> struct Row8 {
    uint32_t x[4], y[4];
};
template <> struct Row8<float> {
    float x[8], y[8];
};

__device__ __forceinline__ void update8(Row8<float> &v, const float (&tv)[8], float c0, const float4 &ck,
                                        const float4 &cn, int fused, bool last, uint32_t &w0, uint32_t &w1)
{
    if (fused) {
        sb_update<K_FUSED, false, 8>(v.x, v.y, tv, c0, ck, ck);
        sign_masks(v.x, w0, w1);
        return;
    }
    // mat_mult + confine (src/kernels.cu:150-209); the window sees x here;
    // then Update_XY of the next step unless the launch ends
    sb_update<K_FC, true, 8>(v.x, v.y, tv, c0, ck, cn);
    sign_masks(v.x, w0, w1);
    if (last) return;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        v.y[q] = fmaf(cn.w, v.x[q], v.y[q]);
        v.x[q] = fmaf(cn.z, v.y[q], v.x[q]);
    }
}
template <class T>
__device__ __forceinline__ void update8(Row8<T> &v, const float (&tv)[8], float c0, const float4 &ck,
                                        const float4 &cn, int fused, bool last, uint32_t &w0, uint32_t &w1)
{
    if (fused) {
        sb_update16<T, K_FUSED, false, 8>(v.x, v.y, tv, c0, ck, ck);
        sign_masks(v.x, w0, w1);
        return;
    }
    // one rounding per step, after the next step's Update_XY; the clamp keeps
    // the sign, so the window's signs are those of the x the step began with
    sign_masks(v.x, w0, w1);
    if (last) sb_update16<T, K_FC, true, 8>(v.x, v.y, tv, c0, ck, cn);
    else sb_update16<T, K_FC, false, 8>(v.x, v.y, tv, c0, ck, cn);
}
template <class T> __device__ __forceinline__ uint32_t sign_word(const Row8<T> &v)
{
    uint32_t m0, m1;
    sign_masks(v.x, m0, m1);
    return (m0 & 0x01010101u) | (m1 & 0x10101010u);
}

__device__ __forceinline__ uint32_t lds32(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}

// Byte counters of nb blocks (at most 63) of a row's entries, the first at
// cp: agents 0..3 in lo, 4..7 in hi.
template <bool NEG>
__device__ __forceinline__ void count8_blocks(const uint2 *cp, int32_t nb, uint32_t S, uint32_t &lo, uint32_t &hi)
{
    for (int32_t b = 0; b < nb; b += 3) {
        uint2 c[3];
#pragma unroll
        for (int j = 0; j < 3; j++)
            if (b + j < nb) c[j] = __ldg(cp + (b + j) * 32);
        uint32_t acc = 0;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            if (b + j >= nb) break;   // warp-uniform
            const uint32_t v[2] = {c[j].x, c[j].y};
#pragma unroll
            for (int h = 0; h < 2; h++) {
                uint32_t w0, w1;
                if (NEG) {
                    w0 = lds32(S + (v[h] & 0x7fffu)) ^ (prmt<0x9999>(v[h], 0u) & 0x11111111u);
                    w1 = lds32(S + ((v[h] >> 16) & 0x7fffu)) ^ (prmt<0xbbbb>(v[h], 0u) & 0x11111111u);
                } else {
                    w0 = lds32(S + (v[h] & 0xffffu));
                    w1 = lds32(S + (v[h] >> 16));
                }
                acc += w0 + w1;
            }
        }
        lo += acc & 0x0f0f0f0fu;
        hi += (acc >> 4) & 0x0f0f0f0fu;
    }
}

// Totals from byte counters of `m` entries (at most 120): PRMT builds the
// float 2^23 + 2 * count; minus 2^23 + m it is 2 * count - m, exactly.
__device__ __forceinline__ void totals8(uint32_t lo, uint32_t hi, float m, float (&tv)[8])
{
    lo += lo;
    hi += hi;
    const float b = -8388608.0f - m;
    const float2 bias = make_float2(b, b);
#pragma unroll
    for (int q = 0; q < 8; q += 2) {
        const uint32_t w = q < 4 ? lo : hi;
        const float2 t = __fadd2_rn(make_float2(__uint_as_float(__byte_perm(w, 0x4b000000u, 0x7440u + (q & 3))),
                                                __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7441u + (q & 3)))),
                                    bias);
        tv[q] = t.x;
        tv[q + 1] = t.y;
    }
}

// Force totals of slot s's 8 agents from the sign words at shared address S.
template <bool NEG>
__device__ __forceinline__ void count8(const Res8P &P, int s, uint32_t S, float (&tv)[8])
{
    const int sl = s >> 5, lane = s & 31;
    const int2 o = __ldg(&P.off[sl]);   // warp-uniform
    const int32_t b0 = o.x, nb = o.y;
    const float deg = __ldg(&P.deg[s]);
    const uint2 *cp = P.col + (int64_t)b0 * 32 + lane;
#pragma unroll
    for (int q = 0; q < 8; q++) tv[q] = 0.f;
#pragma unroll 1
    for (int32_t c0 = 0; c0 < nb; c0 += 30) {   // 120 entries at a time
        float t[8];
        uint32_t lo = 0, hi = 0;
        count8_blocks<NEG>(cp + c0 * 32, min(nb - c0, 30), S, lo, hi);
        totals8(lo, hi, fmaxf(0.f, fminf(deg - (float)(4 * c0), 120.f)), t);
#pragma unroll
        for (int q = 0; q < 8; q++) tv[q] += t[q];
    }
}

// The same for real weights: the sum of -w s over the row in its order.
__device__ __forceinline__ void sum8(const Res8P &P, int s, uint32_t S, float (&tv)[8])
{
    const int sl = s >> 5, lane = s & 31;
    const int2 o2 = __ldg(&P.off[sl]);   // warp-uniform
    const int32_t b0 = o2.x, nb = o2.y;
    const uint2 *cp = P.col + (int64_t)b0 * 32 + lane;
    const float4 *vp = P.val + (int64_t)b0 * 32 + lane;
    float2 t[4];
#pragma unroll
    for (int q = 0; q < 4; q++) t[q] = make_float2(0.f, 0.f);
    for (int32_t b = 0; b < nb; b++) {
        const uint2 c = __ldg(cp + b * 32);
        const float4 v4 = __ldg(vp + b * 32);
        const uint32_t o[4] = {c.x & 0xffffu, c.x >> 16, c.y & 0xffffu, c.y >> 16};
        const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t w = lds32(S + o[j]);
            const uint32_t u = __float_as_uint(v[j]), top = __byte_perm(u, 0u, 0x3333);
            // four top bytes of -w s each
            const uint32_t e = ((w << 7) & 0x80808080u) ^ top, f = ((w << 3) & 0x80808080u) ^ top;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint32_t src = q < 2 ? e : f;
                const int k = 2 * (q & 1);
                t[q] = __fadd2_rn(t[q], make_float2(__uint_as_float(__byte_perm(u, src, 0x4210 + (k << 12))),
                                                    __uint_as_float(__byte_perm(u, src, 0x5210 + (k << 12)))));
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        tv[2 * q] = t[q].x;
        tv[2 * q + 1] = t[q].y;
    }
}

// Global state of 8 agents (16 or 32 contiguous bytes) <-> a row.
template <class T> __device__ __forceinline__ void get8(const T *p, const T *q, Row8<T> &v)
{
    const uint4 a = *(const uint4 *)p, b = *(const uint4 *)q;
    v.x[0] = a.x, v.x[1] = a.y, v.x[2] = a.z, v.x[3] = a.w;
    v.y[0] = b.x, v.y[1] = b.y, v.y[2] = b.z, v.y[3] = b.w;
}
__device__ __forceinline__ void get8(const float *p, const float *q, Row8<float> &v)
{
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const float4 a = ((const float4 *)p)[h], b = ((const float4 *)q)[h];
        v.x[4 * h] = a.x, v.x[4 * h + 1] = a.y, v.x[4 * h + 2] = a.z, v.x[4 * h + 3] = a.w;
        v.y[4 * h] = b.x, v.y[4 * h + 1] = b.y, v.y[4 * h + 2] = b.z, v.y[4 * h + 3] = b.w;
    }
}
template <class T> __device__ __forceinline__ void put8(T *p, T *q, const Row8<T> &v)
{
    *(uint4 *)p = make_uint4(v.x[0], v.x[1], v.x[2], v.x[3]);
    *(uint4 *)q = make_uint4(v.y[0], v.y[1], v.y[2], v.y[3]);
}
__device__ __forceinline__ void put8(float *p, float *q, const Row8<float> &v)
{
#pragma unroll
    for (int h = 0; h < 2; h++) {
        ((float4 *)p)[h] = make_float4(v.x[4 * h], v.x[4 * h + 1], v.x[4 * h + 2], v.x[4 * h + 3]);
        ((float4 *)q)[h] = make_float4(v.y[4 * h], v.y[4 * h + 1], v.y[4 * h + 2], v.y[4 * h + 3]);
    }
}
// Rows kept in shared memory: 16-byte pieces, piece p of row i at [p][i], so
// that a warp's rows are consecutive.
template <class T> constexpr int kPieces = sizeof(T) == 4 ? 4 : 2;
template <class T> __device__ __forceinline__ void ld_row(const uint4 *st, int ns, int i, Row8<T> &v)
{
#pragma unroll
    for (int p = 0; p < kPieces<T>; p++) {
        const uint4 u = st[p * ns + i];
        memcpy((unsigned char *)&v + 16 * p, &u, 16);
    }
}
template <class T> __device__ __forceinline__ void st_row(uint4 *st, int ns, int i, const Row8<T> &v)
{
#pragma unroll
    for (int p = 0; p < kPieces<T>; p++) {
        uint4 u;
        memcpy(&u, (const unsigned char *)&v + 16 * p, 16);
        st[p * ns + i] = u;
    }
}

// Update_XY (src/kernels.cu:8-22), rounded to the storage type if ROUND.
__device__ __forceinline__ void xy8(Row8<float> &v, const float4 &c, int times)
{
    for (int t = 0; t < times; t++)
#pragma unroll
        for (int q = 0; q < 8; q++) {
            v.y[q] = fmaf(c.w, v.x[q], v.y[q]);
            v.x[q] = fmaf(c.z, v.y[q], v.x[q]);
        }
}
template <class T> __device__ __forceinline__ void xy8(Row8<T> &v, const float4 &c, int times)
{
    if (times == 0) return;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        Raw<4> r;
        float x[2], y[2];
        r.u = v.x[i];
        to_vals<T, 2>(r, x);
        r.u = v.y[i];
        to_vals<T, 2>(r, y);
        for (int t = 0; t < times; t++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                y[h] = fmaf(c.w, x[h], y[h]);
                x[h] = fmaf(c.z, y[h], x[h]);
            }
        v.x[i] = from_vals<T, 2>(x).u;
        v.y[i] = from_vals<T, 2>(y).u;
    }
}

// MODE: real weights, all +1, or +-1.
enum { R8_REAL = 0, R8_POS = 1, R8_PM1 = 2 };

template <class T, int MODE>
__global__ void __launch_bounds__(1024, 1) k_res8(const Res8P Q)
{
    const ResP &P = Q.r;
    extern __shared__ __align__(16) unsigned char smem[];
    const int n = (int)P.n, NT = blockDim.x, tid = threadIdx.x;
    uint4 *st = (uint4 *)smem;
    uint32_t *S0 = (uint32_t *)(st + kPieces<T> * n), *S1 = S0 + n + 1;   // sign words, and the zero row
    uint8_t *Wb = (uint8_t *)(S1 + n + 1);                                 // window spins, one byte a row
    __shared__ uint32_t s_chg, s_new, s_stop;
    __shared__ int32_t s_stab[8];
    __shared__ uint8_t s_bif[8], s_prev[8];

    pdl_wait();
    const int a0 = blockIdx.x * 8;           // first agent of this CTA
    const int wg = a0 >> 5, sh = a0 & 31;    // its word and bit offset in planes
    T *xg = (T *)P.x, *yg = (T *)P.y;

    // Early exit of the update-window mode (src/ising.cu:200-211): the
    // previous window left every agent bifurcated.
    if (tid == 0) {
        s_stop = P.ctl[CTL_STOP];
        if (!s_stop && P.uw && P.step0 > 0) {
            const int widx = P.step0 / P.period - 1;
            if (P.wincount[widx] == P.A) s_stop = 1;
        }
        s_chg = 0;
        S0[n] = 0;
        S1[n] = 0;
    }
    if (tid < 8) {
        const int a = a0 + tid;
        s_stab[tid] = P.stab[a];
        s_bif[tid] = P.bif[a];
        s_prev[tid] = P.prev[a];
    }
    __syncthreads();
    if (s_stop) {
        if (blockIdx.x == 0 && tid == 0) P.ctl[CTL_STOP] = 1;
        return;
    }

    // Load the state: at step 0 the pre-step Update_XY (src/ising.cu:188); the
    // unfused step begins with Update_XY of its own step.
    const int32_t k0 = P.step0;
    uint32_t *Scur = (k0 & 1) ? S1 : S0;
    const float4 cu = P.coef[k0];
    const int nxy = (P.first ? 1 : 0) + (P.fused ? 0 : 1);
    for (int s = tid; s < n; s += NT) {
        const int64_t r = __ldg(&P.perm[s]);
        Row8<T> v;
        get8(xg + r * P.Ap + a0, yg + r * P.Ap + a0, v);
        xy8(v, cu, nxy);
        Scur[s] = sign_word(v);
        Wb[s] = (uint8_t)((P.Wp[r * P.W + wg] >> sh) & 0xffu);
        st_row(st, n, s, v);
    }
    __syncthreads();

    const uint32_t sa0 = smem_u32(S0), sa1 = smem_u32(S1);
    for (int32_t it = 0; it < P.nsteps; it++) {
        const int32_t k = k0 + it;
        const uint32_t Sin = (k & 1) ? sa1 : sa0;
        uint32_t *Snx = (k & 1) ? S0 : S1;
        const bool win = ((k + 1) % P.period) == 0;
        const bool last = it == P.nsteps - 1;
        const float4 ck = P.coef[k];
        const float4 cn = P.coef[k + 1];
        uint32_t chg = 0;
        for (int s = tid; s < n; s += NT) {
            float tv[8];
            if (MODE == R8_REAL) sum8(Q, s, Sin, tv);
            else count8<MODE == R8_PM1>(Q, s, Sin, tv);
            Row8<T> v;
            ld_row(st, n, s, v);
            uint32_t m0, m1;   // the signs the window sees
            update8(v, tv, P.c0, ck, cn, P.fused, last, m0, m1);
            st_row(st, n, s, v);
            Snx[s] = P.fused ? (m0 & 0x01010101u) | (m1 & 0x10101010u) : sign_word(v);
            if (win) {
                const uint32_t b = sign_byte(m0, m1);
                chg |= b ^ Wb[s];
                Wb[s] = (uint8_t)b;
            }
        }
        if (win) {
            // Per-agent window bookkeeping inside the CTA, src/kernels.cu:46-79.
            chg = __reduce_or_sync(FULL, chg);
            if ((tid & 31) == 0 && chg) atomicOr(&s_chg, chg);
            __syncthreads();
            if (tid < 8) {
                const int a = a0 + tid;
                const bool equal = !((s_chg >> tid) & 1u);
                const bool nb = !s_bif[tid];
                int sb = s_stab[tid];
                sb += (equal && nb);
                sb = (!equal && nb) ? 0 : sb;
                const bool b = (sb == P.threshold - 1);
                const bool newb = b ^ (s_prev[tid] != 0);
                s_prev[tid] = b;
                s_bif[tid] = b;
                s_stab[tid] = sb;
                const uint32_t nm = __ballot_sync(0xffu, newb && a < P.A);
                const uint32_t bm = __ballot_sync(0xffu, b && a < P.A);
                if (tid == 0) {
                    s_new = nm;
                    if (P.uw) atomicAdd(&P.wincount[(k + 1) / P.period - 1], __popc(bm));
                }
            }
            __syncthreads();
            if (s_new) {
                for (int s = tid; s < n; s += NT) {
                    uint32_t *p = &P.fin[(int64_t)__ldg(&P.perm[s]) * P.W + wg];
                    atomicAnd(p, ~(s_new << sh));
                    atomicOr(p, ((uint32_t)Wb[s] & s_new) << sh);
                }
            }
            if (tid == 0) s_chg = 0;
        }
        __syncthreads();
    }

    // Write the state back (chunked runs continue from it; get_state reads it).
    for (int s = tid; s < n; s += NT) {
        const int64_t r = __ldg(&P.perm[s]);
        Row8<T> v;
        ld_row(st, n, s, v);
        put8(xg + r * P.Ap + a0, yg + r * P.Ap + a0, v);
        plane_put<8>(&P.Wp[r * P.W + wg], Wb[s], sh);
    }
    if (tid < 8) {
        const int a = a0 + tid;
        P.stab[a] = s_stab[tid];
        P.bif[a] = s_bif[tid];
        P.prev[a] = s_prev[tid];
    }
    if (blockIdx.x == 0 && tid == 0) {
        P.ctl[CTL_STEP] = P.step0 + P.nsteps;
        P.ctl[CTL_WINDOWS] = (P.step0 + P.nsteps) / P.period;
    }
}

template <class K, class PT>
cudaError_t launch_res(K kern, const PT &P, size_t smem, int threads, int grid, cudaStream_t s, bool pdl)
{
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return launch(kern, dim3(grid), dim3(threads), smem, s, pdl, P);
}

template <class T>
cudaError_t launch_res8(const Res8P &P, int threads, int grid, cudaStream_t s, bool pdl)
{
    const size_t smem = (size_t)P.r.n * (16 * kPieces<T> + 9) + 8;
    if (P.val) return launch_res(k_res8<T, R8_REAL>, P, smem, threads, grid, s, pdl);
    if (P.allpos) return launch_res(k_res8<T, R8_POS>, P, smem, threads, grid, s, pdl);
    return launch_res(k_res8<T, R8_PM1>, P, smem, threads, grid, s, pdl);
}

}  // namespace

size_t resident_smem_bytes(const SolveDims &d, int ka)
{
    return (size_t)d.n * ka * 2 * prec_bytes(d.prec) + (size_t)d.n * 3 * sizeof(uint32_t);
}

int resident_pick_ka(const SolveDims &d, const DevCsr &J, int requested)
{
    (void)J;
    if (d.prec == P_F64) return 0;
    int dev = 0, smax = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&smax, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const size_t budget = (size_t)smax - 1024;
    auto fits = [&](int ka) { return resident_smem_bytes(d, ka) <= budget; };
    if (requested) return (requested == 8 || requested == 16 || requested == 32) && fits(requested) ? requested : 0;
    return fits(8) ? 8 : 0;
}

namespace {

template <class T>
cudaError_t launch_ka(int ka, const Res8P &Q, size_t smem, int threads, int grid, cudaStream_t s, bool pdl)
{
    if (ka == 8) return launch_res8<T>(Q, threads, grid, s, pdl);
    if (ka == 16) return launch_res(k_resident<T, 16>, Q.r, smem, threads, grid, s, pdl);
    return launch_res(k_resident<T, 32>, Q.r, smem, threads, grid, s, pdl);
}

}  // namespace

cudaError_t launch_resident(const SolveDims &d, const DevCsr &J, Work &w, int ka,
                            int32_t step0, int32_t nsteps, bool first, cudaStream_t s)
{
    Res8P Q;
    ResP &P = Q.r;
    if (ka == 8 && !J.sell[0].base) return cudaErrorInvalidValue;
    Q.off = J.sell[0].off;
    Q.deg = J.sell[0].deg;
    Q.col = J.sell[0].col;
    Q.val = J.sell[0].val;
    Q.allpos = J.allpos ? 1 : 0;
    P.rowptr = J.rowptr;
    P.colw = J.colw;
    P.valf = J.valf;
    P.perm = J.perm;
    P.coef = (const float4 *)w.coef32;
    P.x = w.x;
    P.y = w.y;
    P.Wp = w.Wp;
    P.fin = w.fin;
    P.stab = w.stab;
    P.bif = w.bif;
    P.prev = w.prev;
    P.ctl = w.ctl;
    P.wincount = w.wincount;
    P.n = d.n;
    P.A = d.A;
    P.Ap = d.Ap;
    P.W = d.W;
    P.period = d.period;
    P.threshold = d.threshold;
    P.uw = d.uw;
    P.fused = d.fused;
    P.step0 = step0;
    P.nsteps = nsteps;
    P.first = first ? 1 : 0;
    P.unit = J.unit ? 1 : 0;
    P.c0 = (float)d.c0;
    const size_t smem = resident_smem_bytes(d, ka);
    int threads = (int)((d.n + 31) / 32 * 32);
    if (threads > 1024) threads = 1024;
    if (threads < 64) threads = 64;
    const int grid = (d.A + ka - 1) / ka;
    switch (d.prec) {
    case P_F32: return launch_ka<float>(ka, Q, smem, threads, grid, s, d.pdl);
    case P_BF16: return launch_ka<__nv_bfloat16>(ka, Q, smem, threads, grid, s, d.pdl);
    case P_F16: return launch_ka<__half>(ka, Q, smem, threads, grid, s, d.pdl);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace sbx
