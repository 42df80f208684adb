// k_batch_res.cu -- batched MaxCut with the state on chip for the whole solve:
// the instances are packed into bins (whole instances; a large one is a bin of
// its own), and a cluster of C = 1, 2 or 4 CTAs owns 16 agents of every row of
// one bin from the first step to the last.  Instances never interact and
// neither do agents, so a cluster needs no other.  +-1 weights, degree <= 127,
// fused steps, 16-bit or FP32 state (FP32: 8 agents for 16 in all of this, a
// row's signs in a byte, four neighbours to a word); the arithmetic is the streaming kernel's (exact
// force, sb_update's roundings), so the results are identical.
//
// A step launched per kernel (k_bsm) reads and writes the whole state each
// time and waits for it: at 20 warps an SM it took 234 us a step on 512
// instances (1.9 M rows x 64 agents) with the issue slots 38% busy, and no
// less per row when the state fitted in L2.  Here the loop touches only the
// columns (L2) and shared and tensor memory.
//
// Rows.  A bin's rows are in decreasing degree ("slots"), in slices of 32;
// CTA r of the cluster takes slices r, r + C, ..., its warps a round of 32 of
// them at a time, forwards and backwards in turn (equal work to the barrier); x and y of 16 agents are 64 bytes: the first 4 rows of a thread
// in tensor memory (16 columns each of its own lane), the rest in shared
// memory.  Every CTA holds the signs of all the bin's rows, a 16-bit word a
// row, double-buffered; a new word is stored to all CTAs of the cluster
// (distributed shared memory), and one cluster barrier a step orders the
// stores against the next step's gathers (Jacobi, src/kernels.cu:211-269).
//
// Force.  Columns are blocks of four 16-bit entries (2 slot + sign) per row,
// one coalesced 8-byte load a lane.  Two neighbours' 16-bit words make one
// 32-bit word (XORed with their weights' signs); the words add up in bit
// planes with full adders, the halves are summed, and the planes transposed
// into byte counters.  Sixteen agents a row because a gather and its adders
// then serve twice the agents of eight; thirty-two would not leave a
// 20,000-row instance on eight SMs.  Bound: issue and the ALU pipe.
#include "k_step.cuh"

#include <algorithm>

namespace sbx {

namespace {

constexpr int kNT = 1024;
constexpr int kTmRows = 4;   // rows of a thread in tensor memory: 512 columns / 8 warps a lane quarter / 16 words

struct BresP {
    const int32_t *__restrict__ bins;    // bins of this launch, largest first
    const int32_t *__restrict__ slot0;   // per bin: first slot (of perm and cb), slots + 1 entries in all
    const int32_t *__restrict__ slice0;  // per bin: first slice (of off)
    const int32_t *__restrict__ rows;    // per bin: rows
    const int32_t *__restrict__ off;     // per slice: first block, and the end after a bin's last slice
    const uint2 *__restrict__ col;       // [blocks][32]
    const float2 *__restrict__ cb;       // per slot: dt * xi0 of its instance, -degree
    const int32_t *__restrict__ perm;    // slot -> state row
    const float4 *__restrict__ coef;
    void *x, *y;                         // global [rows][Ap]
    uint32_t *Wp;                        // global plane [rows][W]: signs of the last step
    int32_t *ctl;
    int32_t Ap, W, groups, nsteps;
    uint32_t smem;                       // bytes of dynamic shared memory
    int32_t misfit;                      // test only: the layout is taken not to fit
};

// agents of a cluster: 64 bytes of x and y a row
template <class T> constexpr int kAgents = sizeof(T) == 4 ? 8 : 16;

// Shared memory: the sign planes at kPlane and 2 kPlane of the CTA's shared
// window, the rows past tensor memory's in chunks of 32 (a warp's, [4 pieces of
// 16 bytes][32]) before (from kFirst), between and after them.
constexpr uint32_t kPlane = 0x10000, kChunk = 2048, kFirst = 0x800;
// Sign planes of all +1 or +-1 weights as words (the sign in bit 0 of an
// entry), or words with their complement (the only ones of FP32 state).
enum { BR_POS = 0, BR_BIT = 1, BR_DUAL = 2 };
// bytes of a row's signs
template <class T, int MODE> constexpr uint32_t kRowB = kAgents<T> / 8 * (MODE == BR_DUAL ? 2 : 1);

struct Row16 {
    uint32_t x[8], y[8];   // packed pairs of 16 agents, or FP32 of 8
};

__device__ __forceinline__ uint32_t lds8(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void tm_ld16(uint32_t ta, Row16 &v)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(v.x[0]), "=r"(v.x[1]), "=r"(v.x[2]), "=r"(v.x[3]), "=r"(v.x[4]), "=r"(v.x[5]),
                   "=r"(v.x[6]), "=r"(v.x[7]), "=r"(v.y[0]), "=r"(v.y[1]), "=r"(v.y[2]), "=r"(v.y[3]),
                   "=r"(v.y[4]), "=r"(v.y[5]), "=r"(v.y[6]), "=r"(v.y[7])
                 : "r"(ta)
                 : "memory");
}
__device__ __forceinline__ void tm_st16(uint32_t ta, const Row16 &v)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
                 "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(ta),
                 "r"(v.x[0]), "r"(v.x[1]), "r"(v.x[2]), "r"(v.x[3]), "r"(v.x[4]), "r"(v.x[5]), "r"(v.x[6]),
                 "r"(v.x[7]), "r"(v.y[0]), "r"(v.y[1]), "r"(v.y[2]), "r"(v.y[3]), "r"(v.y[4]), "r"(v.y[5]),
                 "r"(v.y[6]), "r"(v.y[7])
                 : "memory");
}
// Address of the same shared location in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t peer(uint32_t a, uint32_t rank)
{
    uint32_t d;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(rank));
    return d;
}
// A row's signs, 2 or 4 bytes, into this CTA's shared memory or a peer's.
template <int BYTES, bool PEER> __device__ __forceinline__ void st_sign(uint32_t a, uint32_t v)
{
    if (BYTES == 4 && PEER) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
    else if (BYTES == 4) asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
    else if (PEER) asm volatile("st.shared::cluster.u16 [%0], %1;" ::"r"(a), "h"((unsigned short)v) : "memory");
    else asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((unsigned short)v) : "memory");
}
// All threads of the cluster's CTAs; orders their shared stores.
template <int C> __device__ __forceinline__ void step_barrier()
{
    if (C == 1) {
        __syncthreads();
    } else {
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

// A block's four neighbour words as two 32-bit words of two.  S: the plane's
// shared address, a multiple of 64 KB.
template <int MODE> __device__ __forceinline__ void block_words(const uint2 &c, uint32_t S, uint32_t &w0, uint32_t &w1)
{
    const uint32_t u0 = MODE == BR_BIT ? c.x & 0xfffefffeu : c.x, u1 = MODE == BR_BIT ? c.y & 0xfffefffeu : c.y;
    w0 = __byte_perm(lds16(__byte_perm(u0, S, 0x7610)), lds16(__byte_perm(u0, S, 0x7632)), 0x5410);
    w1 = __byte_perm(lds16(__byte_perm(u1, S, 0x7610)), lds16(__byte_perm(u1, S, 0x7632)), 0x5410);
    if (MODE == BR_BIT) {   // 0 or 0xffff per half
        w0 ^= (c.x & 0x00010001u) * 0xffffu;
        w1 ^= (c.y & 0x00010001u) * 0xffffu;
    }
}

// FP32 state: a block's four neighbour bytes as one word.
__device__ __forceinline__ uint32_t block_word8(const uint2 &c, uint32_t S)
{
    const uint32_t b0 = lds8(__byte_perm(c.x, S, 0x7610)), b1 = lds8(__byte_perm(c.x, S, 0x7632));
    const uint32_t b2 = lds8(__byte_perm(c.y, S, 0x7610)), b3 = lds8(__byte_perm(c.y, S, 0x7632));
    return __byte_perm(__byte_perm(b0, b1, 0x0040), __byte_perm(b2, b3, 0x0040), 0x5410);
}

// The same counts for it: the nb entries of a byte lane in PL planes (nb <
// 2^PL), the lanes summed; the low byte of each plane counts.
template <int PL>
__device__ __forceinline__ void count_blocks8(const uint2 *cp, int32_t nb, uint32_t S, uint32_t (&p)[7])
{
    uint32_t q[9];
#pragma unroll
    for (int k = 0; k < 9; k++) q[k] = 0;
    uint2 n0 = make_uint2(0, 0), n1 = n0;
    if (nb > 0) n0 = __ldg(cp);
    if (nb > 1) n1 = __ldg(cp + 32);
    for (int32_t b = 0; b < nb; b += 2) {
        const uint2 c0 = n0, c1 = n1;
        const bool two = b + 1 < nb;   // warp-uniform
        if (b + 2 < nb) n0 = __ldg(cp + (b + 2) * 32);
        if (b + 3 < nb) n1 = __ldg(cp + (b + 3) * 32);
        const uint32_t w0 = block_word8(c0, S), w1 = two ? block_word8(c1, S) : 0u;
        uint32_t c = fadd(q[0], w0, w1);
#pragma unroll
        for (int k = 1; k < PL; k++) {
            const uint32_t t = q[k] & c;
            q[k] ^= c;
            c = t;
        }
    }
#pragma unroll
    for (int f = 0; f < 2; f++) {   // 32 -> 16 -> 8 bits, a plane more each
        uint32_t c = 0;
#pragma unroll
        for (int k = 0; k < PL + f; k++) {
            const uint32_t b = q[k] >> (16 >> f);
            if (k == 0) {
                c = q[0] & b;
                q[0] ^= b;
            } else {
                c = fadd(q[k], b, c);
            }
        }
        q[PL + f] = c;
    }
#pragma unroll
    for (int k = 0; k < 7; k++) p[k] = q[k];   // degree <= 127: seven planes
}

// Counts of the neighbours whose term is -1 over nb blocks as bit planes: bit
// j of p[k] is bit k of agent j's count.  PL planes hold the 2 nb entries of
// a half word (2 nb < 2^PL); one plane more comes out, seven at most (degree
// <= 127).
template <int PL, int MODE>
__device__ __forceinline__ void count_blocks(const uint2 *cp, int32_t nb, uint32_t S, uint32_t (&p)[7])
{
#pragma unroll
    for (int k = 0; k < 7; k++) p[k] = 0;
    // the next two blocks' columns (L2) in flight while two are counted
    uint2 n0 = make_uint2(0, 0), n1 = n0;
    if (nb > 0) n0 = __ldg(cp);
    if (nb > 1) n1 = __ldg(cp + 32);
    for (int32_t b = 0; b < nb; b += 2) {
        const uint2 c0 = n0, c1 = n1;
        const bool two = b + 1 < nb;   // warp-uniform
        if (b + 2 < nb) n0 = __ldg(cp + (b + 2) * 32);
        if (b + 3 < nb) n1 = __ldg(cp + (b + 3) * 32);
        uint32_t w0, w1, w2 = 0u, w3 = 0u;
        block_words<MODE>(c0, S, w0, w1);
        if (two) block_words<MODE>(c1, S, w2, w3);
        const uint32_t a = fadd(p[0], w0, w1), d = fadd(p[0], w2, w3);
        uint32_t c = fadd(p[1], a, d);
#pragma unroll
        for (int k = 2; k < PL; k++) {
            const uint32_t t = p[k] & c;
            p[k] ^= c;
            c = t;
        }
    }
    // the halves together
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < PL; k++) {
        const uint32_t b = p[k] >> 16;
        if (k == 0) {
            c = p[0] & b;
            p[0] ^= b;
        } else {
            c = fadd(p[k], b, c);
        }
    }
    if (PL < 7) p[PL] = c;
}

// The force 2 count - degree of agents 8 h .. 8 h + 7 from the planes.  Byte h
// of planes 0 to 3 in one word, of 4 to 6 in another; agent q's bits of both
// (2^q each) times twice their planes' weights, added to the bits of 2^23 by
// byte dot products, are the float 2^23 + 2^q 2 count, and one FMA scales that
// by 2^-q and takes 2^(23 - q) + degree off: every step is exact.  (An 8x8 bit
// transpose and a PRMT per agent took 70 ALU instructions for 16 agents, this
// takes 42; dot products run on the FMA pipe.)
__device__ __forceinline__ void force8(const uint32_t (&p)[7], int h, float negdeg, float (&tv)[8])
{
    const uint32_t s01 = (uint32_t)h | (((uint32_t)h + 4) << 4);
    const uint32_t lo = __byte_perm(__byte_perm(p[0], p[1], s01), __byte_perm(p[2], p[3], s01), 0x5410);
    const uint32_t hi = __byte_perm(__byte_perm(p[4], p[5], s01), p[6] >> (8 * h), 0x5410);
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const uint32_t m = 0x01010101u << q;
        const uint32_t v = __dp4a(hi & m, 0x00804020u, __dp4a(lo & m, 0x10080402u, 0x4b000000u));
        tv[q] = fmaf(__uint_as_float(v), 1.0f / (1 << q), negdeg - 8388608.0f / (1 << q));
    }
}

template <class T, int C, int MODE>
__global__ void __launch_bounds__(kNT, 1) k_batch_res(const BresP P)
{
    constexpr int KA = kAgents<T>;
    constexpr uint32_t RB = kRowB<T, MODE>;
    static_assert(sizeof(T) == 2 || MODE == BR_DUAL, "FP32 state: words with their complement");
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = C == 1 ? 0 : (int)(blockIdx.x % C);
    const int unit = blockIdx.x / C;
    const int bin = __ldg(&P.bins[unit / P.groups]);
    const int a0 = (unit % P.groups) * KA;
    const int R = __ldg(&P.rows[bin]), sl0 = __ldg(&P.slice0[bin]), s0 = __ldg(&P.slot0[bin]);
    const int nsl = (R + 31) / 32, mine = (nsl - rank + C - 1) / C;   // the bin's slices, this CTA's
    // A CTA's window of the shared address space starts at a multiple of 16 MB
    // (its rank in the cluster); below, offsets in the window.
    const uint32_t sb = smem_u32(smem), win = sb & 0xff000000u, so = sb - win;
    const uint32_t pb = ((uint32_t)(R + 1) * RB + 15) & ~15u;   // bytes of a sign plane
    // chunks before, between and after the planes
    const uint32_t q0 = (kPlane - kFirst) / kChunk, q1 = (kPlane - pb) / kChunk, q2 = (P.smem - 2 * kPlane - pb) / kChunk;
    // Never expected: the layout does not fit.  It assumes that a CTA's shared
    // window starts at a multiple of 16 MB and dynamic shared memory below
    // kFirst in it, which no document promises.  The CTAs of a cluster agree
    // before any of them leaves; the host then takes another kernel.
    __shared__ uint32_t s_bad;
    if (tid == 0)
        s_bad = P.misfit || so > kFirst || pb > kPlane || 2 * kPlane + pb > P.smem ||
                mine - kTmRows * (kNT / 32) > (int)(q0 + q1 + q2);
    step_barrier<C>();
    uint32_t bad = 0;
    if (C == 1) bad = s_bad;
#pragma unroll
    for (int c = 0; c < C; c++)
        if (C > 1) {
            uint32_t v;
            asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(peer(smem_u32(&s_bad), (uint32_t)c)) : "memory");
            bad |= v;
        }
    if (bad) {
        if (tid == 0) atomicExch(&P.ctl[CTL_ERR], kErrMisfit);
        step_barrier<C>();
        return;
    }
    T *xg = (T *)P.x, *yg = (T *)P.y;

    // All of the SM's tensor memory: 1,024 threads of 55 registers and more
    // leave room for no second CTA that would wait for it.
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {   // the zero row that padded entries read
        const uint32_t z = MODE == BR_DUAL ? ~0u << KA : 0u;
        st_sign<RB, false>(win + kPlane + RB * (uint32_t)R, z);
        st_sign<RB, false>(win + 2 * kPlane + RB * (uint32_t)R, z);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    step_barrier<C>();   // the cluster's CTAs are running: their shared memory may be written
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    const uint32_t tw = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(16 * kTmRows * (warp >> 2));

    // the CTA's slice that this warp takes in round i
    auto slice = [&](int i) { return 32 * i + ((i & 1) ? 31 - warp : warp); };
    // this lane's piece 0 of the chunk of round i (past tensor memory's)
    auto chunk = [&](int i) {
        const uint32_t q = (uint32_t)(slice(i) - kTmRows * (kNT / 32));
        const uint32_t a = q < q0 ? kFirst + q * kChunk
                                  : q < q0 + q1 ? kPlane + pb + (q - q0) * kChunk
                                                : 2 * kPlane + pb + (q - q0 - q1) * kChunk;
        return (uint4 *)(smem + (a - so)) + lane;
    };
    auto get_row = [&](int i, Row16 &v) {
        if (i < kTmRows) {
            tm_ld16(tw + 16u * (uint32_t)i, v);
        } else {
            const uint4 *c = chunk(i);
#pragma unroll
            for (int p = 0; p < 4; p++) {
                const uint4 u = c[32 * p];
                memcpy((unsigned char *)&v + 16 * p, &u, 16);
            }
        }
    };
    auto put_row = [&](int i, const Row16 &v) {
        if (i < kTmRows) {
            tm_st16(tw + 16u * (uint32_t)i, v);
        } else {
            uint4 *c = chunk(i);
#pragma unroll
            for (int p = 0; p < 4; p++) {
                uint4 u;
                memcpy(&u, (const unsigned char *)&v + 16 * p, 16);
                c[32 * p] = u;
            }
        }
    };
    uint32_t pk[C];   // the window of every CTA of the cluster
#pragma unroll
    for (int c = 0; c < C; c++) pk[c] = C == 1 ? win : peer(sb, (uint32_t)c) - so;
    auto put_sign = [&](uint32_t plane, int s, uint32_t w) {
        const uint32_t v = MODE == BR_DUAL ? w | (~w << KA) : w, a = plane + RB * (uint32_t)s;
#pragma unroll
        for (int c = 0; c < C; c++) st_sign<RB, (C > 1)>(pk[c] + a, v);
    };
    // signs of a row's agents, agent j in bit j
    auto sign_word = [&](const Row16 &v) {
        if constexpr (sizeof(T) == 4) {
            float x[8];
            memcpy(x, v.x, 32);
            uint32_t m0, m1;
            sign_masks(x, m0, m1);
            return sign_byte(m0, m1);
        } else {
        const uint32_t h0[4] = {v.x[0], v.x[1], v.x[2], v.x[3]}, h1[4] = {v.x[4], v.x[5], v.x[6], v.x[7]};
        uint32_t m0, m1, m2, m3;
        sign_masks(h0, m0, m1);
        sign_masks(h1, m2, m3);
        return sign_byte(m0, m1) | (sign_byte(m2, m3) << 8);
        }
    };

    // The state after the pre-step Update_XY of step 0 (src/ising.cu:188),
    // computed and rounded as the streaming pre-step does.
    const float4 c00 = P.coef[0];
    for (int i = 0; slice(i) < mine; i++) {
        const int s = 32 * (slice(i) * C + rank) + lane;   // slot of the bin
        Row16 v = {};
        if (s < R) {
            const int64_t g = (int64_t)__ldg(&P.perm[s0 + s]) * P.Ap + a0;
            const uint4 xl = ((const uint4 *)(xg + g))[0], xh = ((const uint4 *)(xg + g))[1];
            const uint4 yl = ((const uint4 *)(yg + g))[0], yh = ((const uint4 *)(yg + g))[1];
            memcpy(v.x, &xl, 16);
            memcpy(v.x + 4, &xh, 16);
            memcpy(v.y, &yl, 16);
            memcpy(v.y + 4, &yh, 16);
            T x[KA], y[KA];
            memcpy(x, v.x, 32);
            memcpy(y, v.y, 32);
#pragma unroll
            for (int q = 0; q < KA; q++) {
                float a = St<T>::ld(x[q]), b = St<T>::ld(y[q]);
                b = fmaf(c00.w, a, b);
                a = fmaf(c00.z, b, a);
                x[q] = St<T>::st(a);
                y[q] = St<T>::st(b);
            }
            memcpy(v.x, x, 32);
            memcpy(v.y, y, 32);
            put_sign(kPlane, s, sign_word(v));   // step 0 reads the first plane
        }
        put_row(i, v);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    step_barrier<C>();

    for (int32_t k = 0; k < P.nsteps; k++) {
        const float4 ck = __ldg(&P.coef[k]);
        const uint32_t Sin = win + ((k & 1) ? 2 * kPlane : kPlane), Snx = (k & 1) ? kPlane : 2 * kPlane;
        for (int i = 0; slice(i) < mine; i++) {
            const int sl = slice(i) * C + rank, s = 32 * sl + lane;
            const bool live = s < R;
            const int32_t b0 = __ldg(&P.off[sl0 + sl]), nb = __ldg(&P.off[sl0 + sl + 1]) - b0;   // warp-uniform
            const uint2 *cp = P.col + (int64_t)b0 * 32 + lane;
            const float2 cb = __ldg(&P.cb[s0 + min(s, R - 1)]);
            uint32_t p[7];
            Row16 v;
            if constexpr (sizeof(T) == 4) {
                if (nb < 8) count_blocks8<3>(cp, nb, Sin, p);
                else count_blocks8<6>(cp, nb, Sin, p);   // degree <= 127: at most 32 blocks
                get_row(i, v);
                float tv[8], x[8], y[8];
                force8(p, 0, cb.y, tv);
                memcpy(x, v.x, 32);
                memcpy(y, v.y, 32);
                sb_update<K_FUSED, false, 8>(x, y, tv, cb.x, ck, ck);
                memcpy(v.x, x, 32);
                memcpy(v.y, y, 32);
            } else {
            if (nb < 8) count_blocks<4, MODE>(cp, nb, Sin, p);
            else count_blocks<7, MODE>(cp, nb, Sin, p);
            get_row(i, v);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                float tv[8];
                force8(p, h, cb.y, tv);
                uint32_t x[4], y[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    x[q] = v.x[4 * h + q];
                    y[q] = v.y[4 * h + q];
                }
                sb_update16<T, K_FUSED, false, 8>(x, y, tv, cb.x, ck, ck);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    v.x[4 * h + q] = x[q];
                    v.y[4 * h + q] = y[q];
                }
            }
            }
            put_row(i, v);
            if (live) put_sign(Snx, s, sign_word(v));
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        step_barrier<C>();
    }

    // the state and the signs of the last step back to global memory
    for (int i = 0; slice(i) < mine; i++) {
        const int s = 32 * (slice(i) * C + rank) + lane;
        Row16 v;
        get_row(i, v);
        if (s < R) {
            const int64_t r = __ldg(&P.perm[s0 + s]), g = r * P.Ap + a0;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                ((uint4 *)(xg + g))[h] = make_uint4(v.x[4 * h], v.x[4 * h + 1], v.x[4 * h + 2], v.x[4 * h + 3]);
                ((uint4 *)(yg + g))[h] = make_uint4(v.y[4 * h], v.y[4 * h + 1], v.y[4 * h + 2], v.y[4 * h + 3]);
            }
            if (KA == 16) ((uint16_t *)P.Wp)[r * P.W * 2 + a0 / 16] = (uint16_t)sign_word(v);
            else ((uint8_t *)P.Wp)[r * P.W * 4 + a0 / 8] = (uint8_t)sign_word(v);
        }
    }
    if (blockIdx.x == 0 && tid == 0) {
        P.ctl[CTL_STEP] = P.nsteps;
        P.ctl[CTL_WINDOWS] = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

// Dynamic shared memory of a launch, and whether a bin of R rows fits C CTAs
// with it (the kernel's layout).
uint32_t smem_bytes() { return (uint32_t)std::max(0, dev_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin) - 1024); }
bool fits(int64_t R, int C, uint32_t row_bytes, uint32_t smem)
{
    const int64_t pb = ((R + 1) * row_bytes + 15) / 16 * 16;
    if (pb > kPlane || 2 * (int64_t)kPlane + pb > (int64_t)smem) return false;
    const int64_t chunks = (kPlane - kFirst) / kChunk + (kPlane - pb) / kChunk + (smem - 2 * (int64_t)kPlane - pb) / kChunk;
    const int64_t mine = ((R + 31) / 32 + C - 1) / C;
    return mine - kTmRows * (kNT / 32) <= chunks;
}

template <class T, int C, int MODE>
cudaError_t launch_m(const BresP &P, int units, cudaStream_t s)
{
    auto kern = k_batch_res<T, C, MODE>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P.smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(units * C));
    cfg.blockDim = dim3(kNT);
    cfg.dynamicSmemBytes = P.smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = C > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, P);
}

template <class T>
cudaError_t launch_t(const BresP &P, int c, bool allpos, int units, cudaStream_t s)
{
    if constexpr (sizeof(T) == 4) {
        switch (c) {
        case 0: return launch_m<T, 1, BR_DUAL>(P, units, s);
        case 1: return launch_m<T, 2, BR_DUAL>(P, units, s);
        default: return launch_m<T, 4, BR_DUAL>(P, units, s);
        }
    } else
    switch (c) {
    case 0: return allpos ? launch_m<T, 1, BR_POS>(P, units, s) : launch_m<T, 1, BR_DUAL>(P, units, s);
    case 1: return allpos ? launch_m<T, 2, BR_POS>(P, units, s) : launch_m<T, 2, BR_DUAL>(P, units, s);
    case 2: return allpos ? launch_m<T, 4, BR_POS>(P, units, s) : launch_m<T, 4, BR_DUAL>(P, units, s);
    default: return allpos ? launch_m<T, 4, BR_POS>(P, units, s) : launch_m<T, 4, BR_BIT>(P, units, s);
    }
}

}  // namespace

int batch_res_ctas(int c) { return c == 3 ? 4 : 1 << c; }

int64_t batch_res_rows(int c, bool f32)
{
    const uint32_t smem = smem_bytes();
    const int C = batch_res_ctas(c);
    const bool two = f32 || c == 3;                // bytes of a row's signs: two, or four
    int64_t lo = 0, hi = two ? 32767 : 16383;      // offsets of 16 bits
    while (lo < hi) {
        const int64_t mid = (lo + hi + 1) / 2;
        if (fits(mid, C, two ? 2 : 4, smem)) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

uint32_t batch_res_entry(int c, bool f32, bool allpos, uint32_t slot, bool neg)
{
    return f32 || allpos || c == 3 ? 2 * slot + neg : 4 * slot + 2 * neg;
}

cudaError_t launch_batch_res(const SolveDims &d, const DevBres &B, bool allpos, int32_t agents, Work &w,
                             cudaStream_t s, cudaStream_t *side, cudaEvent_t fork, cudaEvent_t *join, int *launches)
{
    BresP P;
    P.slot0 = B.slot0;
    P.slice0 = B.slice0;
    P.rows = B.rows;
    P.off = B.off;
    P.col = (const uint2 *)B.col;
    P.cb = (const float2 *)B.cb;
    P.perm = B.perm;
    P.coef = (const float4 *)w.coef32;
    P.x = w.x;
    P.y = w.y;
    P.Wp = w.Wp;
    P.ctl = w.ctl;
    P.Ap = d.Ap;
    P.W = d.W;
    const int ka = d.prec == P_F32 ? kAgents<float> : kAgents<__half>;
    P.groups = (agents + ka - 1) / ka;   // groups of padded agents alone stay as they began
    P.nsteps = d.steps_run;
    P.smem = smem_bytes();
    P.misfit = d.giveup;
    // the cluster sizes on streams of their own, largest first: the smaller
    // ones' CTAs fill the SMs that whole clusters leave
    cudaError_t e = cudaEventRecord(fork, s);
    int nside = 0;
    for (int c = 3; c >= 0 && e == cudaSuccess; c--) {
        if (!B.nbins[c]) continue;
        P.bins = B.bins + B.bin0[c];
        cudaStream_t t = side[nside];
        e = cudaStreamWaitEvent(t, fork, 0);
        if (e != cudaSuccess) break;
        const int units = B.nbins[c] * P.groups;
        e = d.prec == P_F32    ? launch_t<float>(P, c, allpos, units, t)
            : d.prec == P_BF16 ? launch_t<__nv_bfloat16>(P, c, allpos, units, t)
                               : launch_t<__half>(P, c, allpos, units, t);
        if (e == cudaSuccess) e = cudaEventRecord(join[nside], t);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(s, join[nside], 0);
        nside++;
        (*launches)++;
    }
    return e;
}

}  // namespace sbx
