// k_resident_rs.cu -- resident MaxCut SB kernel for state too large for one
// SM's shared memory: a CTA owns KA agents of every row (8 of 16-bit state, 4
// of FP32: 32 bytes of x, y a row) and keeps 8,192 rows of them in tensor
// memory -- all of its 256 KB, used as plain storage: a thread's rows are
// eight columns each of its own lane -- and the rest in shared memory, with
// the rows' sign bytes double-buffered in shared memory.  (Register rows
// instead, 4 a thread, left 32 registers to count with: 48 spilled words a
// warp and step, all L1 misses beside 219 KB of shared memory.)  The whole solve (or one window, in the update-window mode) is one
// launch; agents never interact, so a CTA needs no other CTA and one
// __syncthreads() per step gives the Jacobi order of the reference kernel
// (src/kernels.cu:211-269).  The arithmetic is the streaming kernel's (exact
// force, sb_update's roundings), so the two give identical states.
//
// Thread t owns the slots s = i*NT + t of the degree-sorted row list (row
// perm[s]): slots i < 8 in tensor memory, the others in shared memory.  The
// kernel reads the matrix in sliced form (engine.h, DevSell), so a warp's
// entries are coalesced; perm maps slots back to rows only where the global
// state is read or written.
//
// Force for +-1 weights: a block's four neighbour bytes (8 agents each) are
// put together in a word and XORed with the four weights' signs (one PRMT
// makes the mask); the words add up in bit planes, full adders over four
// byte lanes at once, as many planes as the row's blocks can fill; the lanes
// are then summed plane by plane and the planes turned into forces by byte dot
// products.  Bound: issue and the ALU pipe.
#include "k_step.cuh"

#include <algorithm>

namespace sbx {

namespace {

struct RsP {
    const int2 *__restrict__ off;       // sliced matrix (engine.h, DevSell)
    const float *__restrict__ deg;
    const uint2 *__restrict__ col;
    const float4 *__restrict__ val;
    const int32_t *__restrict__ perm;   // slot -> row
    const float4 *__restrict__ coef;    // per step: k1, k2 (clamped), k1, k2 (raw)
    void *x, *y;                        // global [n][Ap]
    uint32_t *Wp, *fin;                 // global planes [n][W]
    int32_t *stab;
    uint8_t *bif, *prev;
    int32_t *ctl;
    int32_t *wincount;                  // bifurcated agents after each window
    int32_t *gbar;                      // co-resident launch: CTAs past each window
    int32_t coop;                       // 1: all windows in one co-resident launch
    int32_t n, A, Ap, W, period, threshold, uw;
    int32_t step0, nsteps, first;
    float c0;
    int32_t giveup;                     // test only: the window barrier gives up at once
};

// agents per CTA: their x and y take 32 bytes a row, their signs a byte
template <class T> constexpr int kAgents = sizeof(T) == 4 ? 4 : 8;
constexpr int kTmRows = 8;     // rows of a thread in tensor memory: 512 columns / 8 warps a lane quarter / 8 words
constexpr int kNT = 1024;
// weights: real, all +1, or +-1
enum { RS_REAL = 0, RS_POS = 1, RS_PM1 = 2 };

// A row's eight state words (x then y) in tensor memory, one column each.
// The load waits for its own data; stores are waited for once a step.
__device__ __forceinline__ void tm_ld(uint32_t ta, uint4 &a, uint4 &b)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
                 : "r"(ta)
                 : "memory");
}
__device__ __forceinline__ void tm_st(uint32_t ta, const uint4 &a, const uint4 &b)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(ta), "r"(a.x),
                 "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}
__device__ __forceinline__ void tm_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Merge the CTA's KA bits (at bit offset sh) into a global plane word.
template <int KA> __device__ __forceinline__ void plane_put(uint32_t *p, uint32_t bits, int sh)
{
    const uint32_t m = ((1u << KA) - 1u) << sh;
    atomicAnd(p, ~m);
    atomicOr(p, (bits << sh) & m);
}

// The four neighbour bytes of block b of a row (8 agents each, at shared
// address S) as one word, signs of the weights applied.
__device__ __forceinline__ uint32_t lds8(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t block_word(const uint2 &c, uint32_t S, bool neg)
{
    const uint32_t b0 = lds8(S + (c.x & 0x7fffu)), b1 = lds8(S + ((c.x >> 16) & 0x7fffu));
    const uint32_t b2 = lds8(S + (c.y & 0x7fffu)), b3 = lds8(S + ((c.y >> 16) & 0x7fffu));
    const uint32_t w = __byte_perm(__byte_perm(b0, b1, 0x0040), __byte_perm(b2, b3, 0x0040), 0x5410);
    return neg ? w ^ prmt<0xfdb9>(c.x, c.y) : w;
}

// p[0..N) += the same planes shifted down by SH bits; one plane more.
template <int N, int SH> __device__ __forceinline__ void fold(uint32_t (&p)[8])
{
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < N; k++) {
        const uint32_t b = p[k] >> SH;
        if (k == 0) {
            c = p[0] & b;
            p[0] ^= b;
        } else {
            c = fadd(p[k], b, c);
        }
    }
    p[N] = c;
}

// The force 2 count - degree of KA agents over nb blocks (fewer than 2^PL).
// The byte lanes' planes are summed; then a byte of each of planes 0 to 3 in
// one word, of 4 to 6 in another, and agent q's bits (2^q each) times twice
// their planes' weights, added to the bits of 2^23 by byte dot products (FMA
// pipe), are the float 2^23 + 2^q 2 count; one FMA scales that by 2^-q and
// takes 2^(23 - q) + degree off, exactly.
template <int PL, int KA, bool NEG>
__device__ __forceinline__ void count_force(const uint2 *cp, int32_t nb, uint32_t S, float negdeg, float (&tv)[8])
{
    uint32_t p[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (PL == 1) {
        p[0] = nb ? block_word(__ldg(cp), S, NEG) : 0u;
    } else {
        for (int32_t b = 0; b < nb; b += 2) {
            const uint2 c0 = __ldg(cp + b * 32);
            uint2 c1;
            const bool two = b + 1 < nb;   // warp-uniform
            if (two) c1 = __ldg(cp + (b + 1) * 32);
            const uint32_t w0 = block_word(c0, S, NEG), w1 = two ? block_word(c1, S, NEG) : 0u;
            uint32_t c = fadd(p[0], w0, w1);
#pragma unroll
            for (int k = 1; k < PL; k++) {
                const uint32_t t = p[k] & c;
                p[k] ^= c;
                c = t;
            }
        }
    }
    fold<PL, 16>(p);
    fold<PL + 1, 8>(p);   // the low byte of each plane: PL + 2 planes, counts of at most 127
    const uint32_t lo = __byte_perm(__byte_perm(p[0], p[1], 0x0040), __byte_perm(p[2], p[3], 0x0040), 0x5410);
    const uint32_t hi = __byte_perm(__byte_perm(p[4], p[5], 0x0040), p[6], 0x5410);
#pragma unroll
    for (int q = 0; q < KA; q++) {
        const uint32_t m = 0x01010101u << q;
        uint32_t v = __dp4a(lo & m, 0x10080402u, 0x4b000000u);
        if (PL > 2) v = __dp4a(hi & m, 0x00804020u, v);
        tv[q] = fmaf(__uint_as_float(v), 1.0f / (1 << q), negdeg - 8388608.0f / (1 << q));
    }
}

// The update of a row's agents; the new signs as a byte.
template <class T>
__device__ __forceinline__ uint32_t update_row(uint4 &xv, uint4 &yv, const float (&tv)[8], float c0, const float4 &c)
{
    uint32_t x[4] = {xv.x, xv.y, xv.z, xv.w}, y[4] = {yv.x, yv.y, yv.z, yv.w}, m0, m1;
    sb_update16<T, K_FUSED, false, 8>(x, y, tv, c0, c, c);
    xv = make_uint4(x[0], x[1], x[2], x[3]);
    yv = make_uint4(y[0], y[1], y[2], y[3]);
    sign_masks(x, m0, m1);
    return sign_byte(m0, m1);
}
template <>
__device__ __forceinline__ uint32_t update_row<float>(uint4 &xv, uint4 &yv, const float (&tv)[8], float c0,
                                                      const float4 &c)
{
    float x[4], y[4];
    const float t[4] = {tv[0], tv[1], tv[2], tv[3]};
    memcpy(x, &xv, 16);
    memcpy(y, &yv, 16);
    sb_update<K_FUSED, false, 4>(x, y, t, c0, c, c);
    memcpy(&xv, x, 16);
    memcpy(&yv, y, 16);
    const uint32_t m0 = __byte_perm(prmt<0x00fb>(xv.x, xv.y), prmt<0x00fb>(xv.z, xv.w), 0x5410);
    return (uint32_t)__dp4a((int)m0, (int)0xf8fcfeffu, 0);
}

// Force totals of slot s's agents (s < n; a lane past the rows repeats the
// last one's degree: its result is not kept).
template <class T, int MODE>
__device__ __forceinline__ void row_force(const RsP &P, int s, uint32_t S, float (&tv)[8])
{
    constexpr int KA = kAgents<T>;
    const int sl = s >> 5, lane = s & 31;
    const int2 o2 = __ldg(&P.off[sl]);   // warp-uniform
    const int32_t b0 = o2.x, nb = o2.y;
    const uint2 *cp = P.col + (int64_t)b0 * 32 + lane;
    if (MODE != RS_REAL) {
        constexpr bool neg = MODE == RS_PM1;
        const float nd = -__ldg(&P.deg[min(s, P.n - 1)]);
        if (nb < 2) count_force<1, KA, neg>(cp, nb, S, nd, tv);
        else if (nb < 8) count_force<3, KA, neg>(cp, nb, S, nd, tv);
        else count_force<6, KA, neg>(cp, nb, S, nd, tv);   // degree <= 127: at most 32 blocks
    } else {
#pragma unroll
        for (int v = 0; v < KA; v++) tv[v] = 0.0f;
        for (int32_t b = 0; b < nb; b++) {
            const uint2 c4 = __ldg(cp + b * 32);
            const float4 v4 = __ldg(P.val + ((int64_t)b0 + b) * 32 + lane);
            const uint32_t o[4] = {c4.x & 0xffffu, c4.x >> 16, c4.y & 0xffffu, c4.y >> 16};
            const float wv[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t w = lds8(S + o[j]);
                // wv is the negated weight; a set bit is spin -1
#pragma unroll
                for (int v = 0; v < KA; v++) tv[v] += ((w >> v) & 1u) ? -wv[j] : wv[j];
            }
        }
    }
}

template <class T, int MODE>
__global__ void __launch_bounds__(kNT, 1) k_resident_rs(const RsP P)
{
    constexpr int KA = kAgents<T>, NT = kNT;
    constexpr uint32_t KM = (1u << KA) - 1u;
    extern __shared__ __align__(16) unsigned char smem[];
    const int n = P.n;
    const int ns = n > kTmRows * NT ? n - kTmRows * NT : 0;   // rows kept in shared memory
    uint4 *xs = (uint4 *)smem;
    uint4 *ys = xs + ns;
    uint8_t *Sb0 = (uint8_t *)(ys + ns);
    uint8_t *Sb1 = Sb0 + n + 1;   // one byte more each: the zero row
    uint8_t *Wb = Sb1 + n + 1;
    __shared__ uint32_t s_chg, s_new, s_stop, s_tmem;
    __shared__ int32_t s_stab[KA];
    __shared__ uint8_t s_bif[KA], s_prev[KA];

    pdl_wait();
    const int tid = threadIdx.x;
    const int a0 = blockIdx.x * KA;          // first agent of this CTA
    const int wg = a0 >> 5, sh = a0 & 31;    // its word and bit offset in the planes
    T *xg = (T *)P.x, *yg = (T *)P.y;

    // early exit of the update-window mode (src/ising.cu:200-211)
    if (tid == 0) {
        s_stop = P.ctl[CTL_STOP];
        if (!s_stop && P.uw && P.step0 > 0) {
            const int widx = P.step0 / P.period - 1;
            if (P.wincount[widx] == P.A) s_stop = 1;
        }
        s_chg = 0;
        Sb0[n] = 0;
        Sb1[n] = 0;
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

    // All of the SM's tensor memory: 1,024 threads of 55 registers and more
    // leave room for no second CTA that would wait for it.
    const int warp = tid >> 5;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    // this warp's lane quarter and columns
    const uint32_t tw = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(8 * kTmRows * (warp >> 2));
    // a row's state: tensor memory (whole warps), then shared memory
    auto get_row = [&](int i, int s, uint4 &xv, uint4 &yv) {
        if (i < kTmRows) {
            tm_ld(tw + 8u * (uint32_t)i, xv, yv);
        } else if (s < n) {
            xv = xs[s - kTmRows * NT];
            yv = ys[s - kTmRows * NT];
        }
    };
    auto put_row = [&](int i, int s, const uint4 &xv, const uint4 &yv) {
        if (i < kTmRows) {
            tm_st(tw + 8u * (uint32_t)i, xv, yv);
        } else if (s < n) {
            xs[s - kTmRows * NT] = xv;
            ys[s - kTmRows * NT] = yv;
        }
    };
    // this warp's slots: i * NT + 32 * warp + lane while any is a row
    const int w0 = 32 * warp;

    // Load the state (the pre-step Update_XY at step 0, src/ising.cu:188, as
    // the streaming pre-step computes it) and the sign words of step k0.
    const int32_t k0 = P.step0;
    uint8_t *Scur = (k0 & 1) ? Sb1 : Sb0;
    const float4 c00 = P.coef[0];
    for (int i = 0; i * NT + w0 < n; i++) {
        const int s = i * NT + tid;
        uint4 xv = make_uint4(0, 0, 0, 0), yv = xv;
        if (s < n) {
            const int r = __ldg(&P.perm[s]);
            xv = *(const uint4 *)(xg + (int64_t)r * P.Ap + a0);
            yv = *(const uint4 *)(yg + (int64_t)r * P.Ap + a0);
            Raw<16> xw, yw;
            xw.u = xv;
            yw.u = yv;
            float x[KA], y[KA];
            to_vals<T, KA>(xw, x);
            to_vals<T, KA>(yw, y);
            if (P.first) {
#pragma unroll
                for (int v = 0; v < KA; v++) {
                    y[v] = fmaf(c00.w, x[v], y[v]);
                    x[v] = fmaf(c00.z, y[v], x[v]);
                }
                xv = from_vals<T, KA>(x).u;
                yv = from_vals<T, KA>(y).u;
            }
            uint32_t bits = 0;
#pragma unroll
            for (int v = 0; v < KA; v++) bits |= sbit(x[v]) << v;
            Scur[s] = (uint8_t)bits;
            Wb[s] = (uint8_t)((P.Wp[(int64_t)r * P.W + wg] >> sh) & KM);
        }
        put_row(i, s, xv, yv);
    }
    tm_wait_st();
    __syncthreads();

    const uint32_t sa0 = smem_u32(Sb0), sa1 = smem_u32(Sb1);
    int32_t nrun = P.nsteps;   // steps run (fewer at an update-window exit)
    for (int32_t it = 0; it < P.nsteps; it++) {
        const int32_t k = k0 + it;
        const uint32_t Sin = (k & 1) ? sa1 : sa0;
        uint8_t *Snx = (k & 1) ? Sb0 : Sb1;
        const bool win = ((k + 1) % P.period) == 0;
        const float4 ck = P.coef[k];
        uint32_t chg = 0;
        // the signs of row s, new and in window steps against the last window's
        auto put_sign = [&](int s, uint32_t nb) {
            Snx[s] = (uint8_t)nb;
            if (win) {
                chg |= nb ^ Wb[s];
                Wb[s] = (uint8_t)nb;
            }
        };
        // rows in tensor memory (whole warps: a lane past the rows steps what
        // lies there and keeps nothing), then the others
        const int nt = min(kTmRows, (n - w0 + NT - 1) / NT);
        for (int i = 0; i < nt; i++) {
            const int s = i * NT + tid;
            float tv[8];
            row_force<T, MODE>(P, s, Sin, tv);
            uint4 xv, yv;
            tm_ld(tw + 8u * (uint32_t)i, xv, yv);
            const uint32_t nb = update_row<T>(xv, yv, tv, P.c0, ck);
            tm_st(tw + 8u * (uint32_t)i, xv, yv);
            if (s < n) put_sign(s, nb);
        }
        for (int s = kTmRows * NT + tid; s < n; s += NT) {
            float tv[8];
            row_force<T, MODE>(P, s, Sin, tv);
            uint4 xv = xs[s - kTmRows * NT], yv = ys[s - kTmRows * NT];
            const uint32_t nb = update_row<T>(xv, yv, tv, P.c0, ck);
            xs[s - kTmRows * NT] = xv;
            ys[s - kTmRows * NT] = yv;
            put_sign(s, nb);
        }
        tm_wait_st();
        if (win) {
            // per-agent window bookkeeping inside the CTA, src/kernels.cu:46-79
            chg = __reduce_or_sync(FULL, chg);
            if ((tid & 31) == 0 && chg) atomicOr(&s_chg, chg);
            __syncthreads();
            if (tid < KA) {
                const int a = a0 + tid;
                const bool equal = !((s_chg >> tid) & 1u);
                const bool nbf = !s_bif[tid];
                int st = s_stab[tid];
                st += (equal && nbf);
                st = (!equal && nbf) ? 0 : st;
                const bool b = (st == P.threshold - 1);
                const bool newb = b ^ (s_prev[tid] != 0);
                s_prev[tid] = b;
                s_bif[tid] = b;
                s_stab[tid] = st;
                const uint32_t nm = __ballot_sync(KM, newb && a < P.A);
                const uint32_t bm = __ballot_sync(KM, b && a < P.A);
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
            if (P.uw && P.coop) {
                // The update-window exit inside one co-resident launch: after
                // every CTA has counted its bifurcated agents for this window,
                // all of them read the total (src/ising.cu:200-211).  The
                // barrier's wait is bounded; giving up flags an error.
                const int widx = (k + 1) / P.period - 1;
                __syncthreads();
                if (tid == 0) {
                    __threadfence();
                    atomicAdd(P.gbar, 1);
                    // test only (giveup): a target no window reaches and a
                    // short limit, the path of a CTA that never arrives
                    const int target = (int)gridDim.x * (widx + 1 + P.giveup);
                    const uint32_t limit = P.giveup ? (1u << 12) : (1u << 26);
                    uint32_t spins = 0;
                    while (atomicAdd(P.gbar, 0) < target) {
                        if (++spins > limit) {
                            atomicExch(&P.ctl[CTL_ERR], 1);
                            s_stop = 1;
                            break;
                        }
                        __nanosleep(64);
                    }
                    __threadfence();
                    if (!s_stop && atomicAdd(&P.wincount[widx], 0) == P.A) s_stop = 2;
                }
                __syncthreads();
                if (s_stop) {
                    nrun = it + 1;
                    break;
                }
            }
        }
        __syncthreads();
    }

    // write the state back (chunked runs continue from it; get_state reads it)
    for (int i = 0; i * NT + w0 < n; i++) {
        const int s = i * NT + tid;
        uint4 xv = make_uint4(0, 0, 0, 0), yv = xv;
        get_row(i, s, xv, yv);
        if (s < n) {
            const int r = __ldg(&P.perm[s]);
            *(uint4 *)(xg + (int64_t)r * P.Ap + a0) = xv;
            *(uint4 *)(yg + (int64_t)r * P.Ap + a0) = yv;
        }
    }
    for (int s = tid; s < n; s += NT) plane_put<KA>(&P.Wp[(int64_t)__ldg(&P.perm[s]) * P.W + wg], Wb[s], sh);
    if (tid < KA) {
        const int a = a0 + tid;
        P.stab[a] = s_stab[tid];
        P.bif[a] = s_bif[tid];
        P.prev[a] = s_prev[tid];
    }
    if (blockIdx.x == 0 && tid == 0) {
        P.ctl[CTL_STEP] = P.step0 + nrun;
        P.ctl[CTL_WINDOWS] = (P.step0 + nrun) / P.period;
        if (s_stop == 2) P.ctl[CTL_STOP] = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

// shared memory of n rows: those past tensor memory's, and three bytes each
size_t rs_smem(int64_t n)
{
    const int64_t ns = n > (int64_t)kTmRows * kNT ? n - (int64_t)kTmRows * kNT : 0;
    return (size_t)ns * 32 + (size_t)n * 3 + 2;
}

template <class T, int MODE>
cudaError_t launch_rs_m(const RsP &P, size_t smem, int grid, cudaStream_t s, bool pdl)
{
    auto kern = k_resident_rs<T, MODE>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    if (P.coop) {
        // every CTA must be resident at once for the window barrier
        int per_sm = 0;
        const int nsm = dev_attr(cudaDevAttrMultiProcessorCount);
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kNT, smem);
        if (e != cudaSuccess) return e;
        // one CTA an SM: it holds all of the SM's tensor memory
        if ((int64_t)std::min(per_sm, 1) * nsm < grid) return cudaErrorCooperativeLaunchTooLarge;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kNT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    if (P.coop) {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    } else {
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = (pdl || P.coop) ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, P);
}

template <class T>
cudaError_t launch_rs_t(const DevCsr &J, const RsP &P, size_t smem, cudaStream_t s, bool pdl)
{
    const int grid = (P.A + kAgents<T> - 1) / kAgents<T>;
    if (!J.unit) return launch_rs_m<T, RS_REAL>(P, smem, grid, s, pdl);
    if (J.allpos) return launch_rs_m<T, RS_POS>(P, smem, grid, s, pdl);
    return launch_rs_m<T, RS_PM1>(P, smem, grid, s, pdl);
}

}  // namespace

int resident_rs_pick(const SolveDims &d, const DevCsr &J, bool forced, bool tile)
{
    const bool half = d.prec == P_BF16 || d.prec == P_F16;
    if (!half && (forced || d.prec != P_F32)) return 0;
    if (!d.fused || d.n > (1 << 24)) return 0;
    if (J.unit && J.max_deg > kHeavy) return 0;   // the planes hold 127 neighbours
    const int nsm = dev_attr(cudaDevAttrMultiProcessorCount);
    const int64_t budget = (int64_t)dev_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin) - 1024;
    // asked for: the rows that four a thread in registers and shared memory
    // hold (what the entry point has always taken)
    const int held = std::max<int64_t>(0, d.n - 4096) * 32 + d.n * 3 <= budget ? 8 : 0;
    if (forced) return held;
    // a streaming tile asked for without a kernel: 16-bit state whose agents
    // fill half the SMs has always stayed on chip, the rest streamed with it
    if (tile) return half && (d.A + 7) / 8 >= nsm / 2 ? held : 0;
    const int ka = half ? 8 : 4;
    if ((int64_t)rs_smem(d.n) > budget) return 0;
    // Chosen by itself where its step is clearly the shorter one (by 5%, the
    // fits' error).  Both sides fitted on GB300 (mean error 3 to 10%) on 13
    // graphs each of 3,136 to 14,000 rows (16 bits: 5,400 to 14,000) and mean
    // degrees 2 to 85, +-1 and real weights apart, at 32 to 2,000 agents.  A
    // wave of one CTA an SM has a fixed time and one per row and neighbour, and
    // rows past tensor memory's cost more; the streaming step has a fixed time
    // and one per row and agent, the agents as its tile holds them.  E.g. FP32
    // (us a step, resident against streaming): 5,929 rows of degree 4 at 32
    // agents 4.5 against 2.7, at 1,024 9.2 against 16.8; 3,136 of degree 8 at 32
    // agents 4.1 against 2.9; 12,500 of degree 16, real weights, at 480 agents
    // 25 against 43; at degree 85, 256 agents 105 against 83.
    struct Fit {
        double wave, row4, row, nbr, past;     // us; ns per row (up to degree 4), per row, per neighbour, past 8,192
        double step, cell4, cell, cell_nbr;    // us; ps per row and agent (up to degree 4), ..., per neighbour
    };
    static const Fit kFit[2][2] = {
        {{1.0, 0.61, 0.65, 0.043, 0.32, 2.65, 2.2, 2.65, 0.025}, {1.2, 0, 0.35, 0.094, 0.30, 3.9, 0, 1.75, 0.27}},
        {{1.25, 0.77, 0.86, 0.041, 0.28, 2.9, 1.23, 1.5, 0.02}, {2.2, 0, 0.52, 0.122, 0.36, 4.7, 0, 0.73, 0.19}},
    };
    const Fit &f = kFit[half][!J.unit];
    const double n = (double)d.n, deg = (double)J.nnz / n;
    const bool low = J.unit && deg <= 4;   // one block of four neighbours a row
    const double waves = (double)(((d.A + ka - 1) / ka + nsm - 1) / nsm);
    const double res = waves * (f.wave + 1e-3 * (n * (low ? f.row4 : f.row + f.nbr * deg) +
                                                 std::max(0.0, n - kTmRows * kNT) * f.past));
    const double str = f.step + 1e-6 * n * tile_agents(d) * (low ? f.cell4 : f.cell + f.cell_nbr * deg);
    return 1.05 * res < str ? ka : 0;
}

cudaError_t launch_resident_rs(const SolveDims &d, const DevCsr &J, Work &w, int ka, int32_t step0,
                               int32_t nsteps, bool first, bool coop, cudaStream_t s)
{
    RsP P;
    if (ka < 1 || !J.sell[1].base) return cudaErrorInvalidValue;
    P.off = J.sell[1].off;
    P.deg = J.sell[1].deg;
    P.col = J.sell[1].col;
    P.val = J.sell[1].val;
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
    P.gbar = w.gbar;
    P.coop = (coop && d.uw && w.gbar) ? 1 : 0;
    P.n = (int32_t)d.n;
    P.A = d.A;
    P.Ap = d.Ap;
    P.W = d.W;
    P.period = d.period;
    P.threshold = d.threshold;
    P.uw = d.uw;
    P.step0 = step0;
    P.nsteps = nsteps;
    P.first = first ? 1 : 0;
    P.c0 = (float)d.c0;
    P.giveup = d.giveup;
    const size_t smem = rs_smem(d.n);
    if (d.prec == P_BF16) return launch_rs_t<__nv_bfloat16>(J, P, smem, s, d.pdl);
    if (d.prec == P_F16) return launch_rs_t<__half>(J, P, smem, s, d.pdl);
    if (d.prec == P_F32) return launch_rs_t<float>(J, P, smem, s, d.pdl);
    return cudaErrorInvalidValue;
}

}  // namespace sbx
