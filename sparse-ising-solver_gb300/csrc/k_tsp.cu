// k_tsp.cu -- TSP-QUBO ballistic SB (src/kernels.cu:543-599) with the
// validity window (src/kernels.cu:461-541).
//
// Structured kernel.  The QUBO of tsp_gpu.cu:76-112 over spins (position i,
// city k) is C/4 between equal cities at different positions, A d_kl/8 between
// cyclically adjacent positions at different cities, B/4 between different
// cities at one position and (B+C)/4 on the diagonal.  Hence, exactly,
//   (J x)[i][k] = C/4 colsum[k] + B/4 rowsum[i] + A/8 sum_l d_kl (x[i-1][l] + x[i+1][l])
// (the diagonal cancels the self terms of the two penalty sums; for N = 2 the
// two neighbours are one position).  A CTA owns KA agents and keeps their x in
// shared memory for the whole run.  H threads share a (position i, agent a)
// row's cities: each reads the two neighbouring rows and multiplies them with
// its cities' distances, while one part also sums its row and one its
// column; after a barrier each updates its cities.  The distances are
// constant operands of the multiply-adds (a kernel parameter, addressed at
// compile time: warp w takes part w mod H, so a scheduler's warps share one
// part's kilobyte).  No CTA talks to another, so the whole solve is one
// launch.  Bound: issue (5 FP32 operations per 4 products).  29 cities x 1,000
// agents: 6.0 us a step with one thread a row, 4.2 with four and the distances
// in shared memory (a 16-byte shared load takes four cycles even when all
// lanes share its address).
//
// Streaming kernel.  The CSR form of the same QUBO, one launch per step, x
// double-buffered (Jacobi); used in FP64 (which it reproduces operation by
// operation) and when N > 32.
#include "common.cuh"
#include "engine.h"

#include <algorithm>

namespace sbx {

namespace {

struct TspP {
    const float *__restrict__ I2;     // [N] linear field per city
    const float2 *__restrict__ sched; // per step: b_t, dt*-(1-a_t)
    void *x, *y;                      // global [n][Ap], n = N*N, row = i*N + k
    uint32_t *Wp;                     // global plane [n][W] (window spins)
    int32_t *tours, *valid;           // [Ap][N], [Ap]
    int32_t *stab;
    uint8_t *bif, *prev;
    int32_t *ctl;
    int32_t N, A, Ap, W, nwin, period, threshold;
    float qa8, qb4, qc4;              // A/8, B/4, C/4
    float dtxi0, dt, k1u, k2u;        // pre-step Update_XY coefficients
};

template <class T> __device__ __forceinline__ float rnd(float v) { return St<T>::ld(St<T>::st(v)); }

template <int NP> struct TspD {
    float d[NP * NP];   // distances, zero past the cities
};

// Cities [K0, K0 + CPT) of the distance product of a row's two neighbours.
template <int NP, int CPT, int K0>
__device__ __forceinline__ void dist_product(const TspD<NP> &D, const float *rm, const float *rp, bool two,
                                             float (&dk)[CPT])
{
#pragma unroll
    for (int j = 0; j < CPT; j++) dk[j] = 0.f;
#pragma unroll
    for (int l = 0; l < NP; l += 4) {
        const float4 m4 = *(const float4 *)&rm[l];
        const float4 p4 = two ? *(const float4 *)&rp[l] : make_float4(0, 0, 0, 0);
        const float nb[4] = {m4.x + p4.x, m4.y + p4.y, m4.z + p4.z, m4.w + p4.w};
#pragma unroll
        for (int j = 0; j < CPT; j++) {
            const float *d = &D.d[(K0 + j) * NP + l];
            dk[j] += d[0] * nb[0] + d[1] * nb[1] + d[2] * nb[2] + d[3] * nb[3];
        }
    }
}

// H parts of a row's NP cities.
template <class T, int NP, int H>
__global__ void __launch_bounds__(H == 1 ? 512 : 1024) k_tsp_resident(const TspP P,
                                                                      const __grid_constant__ TspD<NP> D,
                                                                      const int KA)
{
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int NPS = NP + 4;       // padded row: spreads rows over banks
    constexpr int CPT = NP / H;       // cities of a thread
    const int N = P.N, rows = N * KA;
    float *xs = (float *)smem;                          // [N][KA][NPS]
    float *colsum = xs + (size_t)rows * NPS;            // [KA][NPS]
    float *rsum = colsum + KA * NPS;                    // [N][KA]
    uint32_t *rowbits = (uint32_t *)(rsum + rows);      // [N][KA]
    uint32_t *prevbits = rowbits + rows;                // [N][KA]
    int *aflag = (int *)(prevbits + rows);              // [KA] valid, [KA] changed
    __shared__ float s_I2[NP];

    pdl_wait();
    const int tid = threadIdx.x, warp = tid >> 5;
    const int h = warp % H, m = 32 * (warp / H) + (tid & 31);   // part, row
    const int i = m / KA, a = m - (m / KA) * KA;        // position, local agent
    const int k0 = CPT * h;                             // first city of this thread
    const int ag = blockIdx.x * KA + a;                 // global agent
    const bool active = m < rows;
    const bool real = ag < P.A;                         // padded agents compute on zeros
    T *xg = (T *)P.x, *yg = (T *)P.y;

    for (int t = tid; t < NP; t += blockDim.x) s_I2[t] = t < N ? P.I2[t] : 0.f;
    for (int t = tid; t < KA * NPS; t += blockDim.x) colsum[t] = 0.f;

    // Initial state (x = 0, y from the init stream) and the pre-step
    // Update_XY at step 0 (src/ising_tsp.cu:155).
    float yr[CPT], xo[CPT];
    float *xrow = &xs[(size_t)m * NPS + k0];
#pragma unroll
    for (int j = 0; j < CPT; j++) {
        const int k = k0 + j;
        float x = 0.f, y = 0.f;
        if (active && k < N && real) {
            const int64_t gi = (int64_t)(i * N + k) * P.Ap + ag;
            x = St<T>::ld(xg[gi]);
            y = St<T>::ld(yg[gi]);
            y = rnd<T>(y + P.k2u * x);
            x = rnd<T>(x + P.k1u * y);
        }
        yr[j] = y;
        xo[j] = x;
        if (active) xrow[j] = x;
    }
    if (active && h == 0) {
        prevbits[m] = 0xffffffffu;   // current_spins = -1
        rowbits[m] = 0;
    }
    int stab = 0;
    bool bif = false, prv = false;
    if (active && i == 0 && h == 0 && real) {
        stab = P.stab[ag];
        bif = P.bif[ag];
        prv = P.prev[ag];
    }
    __syncthreads();
    // the linear field of this thread's cities (all 32: from shared memory where
    // it is used, their registers are spent)
    [[maybe_unused]] float i2r[CPT > 8 ? 1 : CPT];
    if constexpr (CPT <= 8) {
#pragma unroll
        for (int j = 0; j < CPT; j++) i2r[j] = s_I2[k0 + j];
    }
    auto field = [&](int j) {
        if constexpr (CPT <= 8) return i2r[j];
        else return s_I2[k0 + j];
    };

    const bool whole = k0 + CPT <= N;   // warp-uniform: no city past N
    // the parts that sum this row and its column: another for the next warp
    // of rows, so that the schedulers (warp mod 4) share the sums
    const int hrow = (warp / H) % H, hcol = (warp / H + H / 2) % H;
    const int im = i == 0 ? N - 1 : i - 1, ip = i + 1 >= N ? 0 : i + 1;
    const float *rm = &xs[(size_t)(im * KA + a) * NPS], *rp = &xs[(size_t)(ip * KA + a) * NPS];
    const int nwin = P.nwin;
    const uint32_t maskN = N == 32 ? 0xffffffffu : ((1u << N) - 1u);
    int k_step = 0;
    for (int wdx = 0; wdx < nwin; wdx++) {
        for (int it = 0; it < P.period; it++, k_step++) {
            const float2 sc = P.sched[k_step];
            // Phase 1: the distance product of this thread's cities; the sum
            // of its row and that of city i's column each by one of its parts.
            float dk[CPT];
            if (active) {
                if (h == 0) dist_product<NP, CPT, 0>(D, rm, rp, N > 2, dk);
                else if (h == 1) dist_product<NP, CPT, CPT % NP>(D, rm, rp, N > 2, dk);
                else if (h == 2) dist_product<NP, CPT, 2 * CPT % NP>(D, rm, rp, N > 2, dk);
                else dist_product<NP, CPT, 3 * CPT % NP>(D, rm, rp, N > 2, dk);
                if (h == hrow) {
                    const float *r = &xs[(size_t)m * NPS];
                    float rs = 0.f;
#pragma unroll
                    for (int l = 0; l < NP; l += 4) {
                        const float4 x4 = *(const float4 *)&r[l];
                        rs += x4.x;
                        rs += x4.y;
                        rs += x4.z;
                        rs += x4.w;
                    }
                    rsum[m] = rs;
                }
                if (h == hcol) {
                    const float *c = &xs[(size_t)a * NPS + i];   // column (city) i over all positions
                    float cs = 0.f;
#pragma unroll 8
                    for (int p = 0; p < N; p++) cs += c[p * KA * NPS];
                    colsum[a * NPS + i] = cs;
                }
            }
            __syncthreads();
            // Phase 2: forces and the bSB update of this thread's spins, two
            // cities at a time in packed FP32 (per component the roundings of
            // the scalar operations), both clamp branches computed and
            // selected; cities past N stay zero.
            if (active) {
                const float rs = rsum[m];
                const float2 qc = make_float2(P.qc4, P.qc4), qb = make_float2(P.qb4, P.qb4);
                const float2 qa = make_float2(P.qa8, P.qa8), rs2 = make_float2(rs, rs);
                const float2 m1005 = make_float2(-1.005f, -1.005f), two = make_float2(2.f, 2.f);
                const float2 bt = make_float2(sc.x, sc.x), cxi = make_float2(P.dtxi0, P.dtxi0);
                const float2 cdt = make_float2(P.dt, P.dt), cy = make_float2(sc.y, sc.y);
#pragma unroll
                for (int j = 0; j < CPT; j += 4) {
                    const float4 c4 = *(const float4 *)&colsum[a * NPS + k0 + j];
#pragma unroll
                    for (int e = 0; e < 4; e += 2) {
                        const int q = j + e;
                        const float2 cs2 = e ? make_float2(c4.z, c4.w) : make_float2(c4.x, c4.y);
                        const float2 jx = __ffma2_rn(qa, make_float2(dk[q], dk[q + 1]),
                                                     __ffma2_rn(qc, cs2, __fmul2_rn(qb, rs2)));
                        const float2 i1 = __fmul2_rn(m1005, jx);
                        const float2 x0 = make_float2(xo[q], xo[q + 1]), y0 = make_float2(yr[q], yr[q + 1]);
                        float2 y = __ffma2_rn(cxi, __ffma2_rn(bt, make_float2(field(q), field(q + 1)),
                                                              __fmul2_rn(two, i1)), y0);
                        y = make_float2(rnd<T>(y.x), rnd<T>(y.y));
                        float2 x = __ffma2_rn(cdt, y, x0);
                        x = make_float2(rnd<T>(x.x), rnd<T>(x.y));
                        y = __ffma2_rn(cy, x, y);
                        y = make_float2(rnd<T>(y.x), rnd<T>(y.y));
                        const bool w0 = fabsf(x0.x) > 1.f, w1 = fabsf(x0.y) > 1.f;
                        if (whole || k0 + q < N) {
                            xo[q] = w0 ? spin_of(x0.x) : x.x;
                            yr[q] = w0 ? 0.f : y.x;
                        }
                        if (whole || k0 + q + 1 < N) {
                            xo[q + 1] = w1 ? spin_of(x0.y) : x.y;
                            yr[q + 1] = w1 ? 0.f : y.y;
                        }
                    }
                }
#pragma unroll
                for (int l = 0; l < CPT; l += 4)
                    *(float4 *)&xrow[l] = make_float4(xo[l], xo[l + 1], xo[l + 2], xo[l + 3]);
            }
            __syncthreads();
        }
        // Window: validity (one +1 per city and per position), stability,
        // tour snapshot of valid agents (src/kernels.cu:473-531); each part
        // adds its cities' sign bits, part 0 of the row decides.
        if (active) {
            uint32_t part = 0;
#pragma unroll
            for (int j = 0; j < CPT; j++)
                if (k0 + j < N) part |= sbit(xo[j]) << (k0 + j);
            if (part) atomicOr(&rowbits[m], part);
        }
        if (tid < 2 * KA) aflag[tid] = tid < KA ? 1 : 0;
        __syncthreads();
        const uint32_t bits = active ? rowbits[m] : 0u;
        if (active && h == 0) {
            const int order_cnt = __popc(~bits & maskN);
            int city_cnt = 0;
            for (int p = 0; p < N; p++) city_cnt += (~rowbits[p * KA + a] >> i) & 1u;
            if (order_cnt != 1 || city_cnt != 1) atomicAnd(&aflag[a], 0);
            if (bits != (prevbits[m] & maskN)) atomicOr(&aflag[KA + a], 1);
        }
        __syncthreads();
        if (active && h == 0) {
            const bool valid = aflag[a] != 0;
            if (valid && real) {
                P.tours[(int64_t)ag * N + i] = __ffs(~bits & maskN) - 1;
                if (i == 0) P.valid[ag] = k_step;
            }
            if (i == 0) {
                const bool equal = aflag[KA + a] == 0;
                const bool nb = !bif;
                stab += (equal && nb);
                stab = (!equal && nb) ? 0 : stab;
                bif = (stab == P.threshold - 1);
                prv = bif;
            }
            prevbits[m] = bits;
            rowbits[m] = 0;
        }
        __syncthreads();
    }

    // State back to global memory (get_state) and the window spins.
    if (active && real) {
#pragma unroll
        for (int j = 0; j < CPT; j++)
            if (k0 + j < N) {
                const int64_t gi = (int64_t)(i * N + k0 + j) * P.Ap + ag;
                xg[gi] = St<T>::st(xo[j]);
                yg[gi] = St<T>::st(yr[j]);
            }
        const uint32_t bits = prevbits[m];
        for (int k = k0; k < k0 + CPT && k < N; k++) {
            const int64_t r = i * N + k;
            const uint32_t bit = (bits >> k) & 1u;
            uint32_t *p = &P.Wp[r * P.W + (ag >> 5)];
            if (bit) atomicOr(p, 1u << (ag & 31));
            else atomicAnd(p, ~(1u << (ag & 31)));
        }
        if (i == 0 && h == 0) {
            P.stab[ag] = stab;
            P.bif[ag] = bif;
            P.prev[ag] = prv;
        }
    }
    if (blockIdx.x == 0 && tid == 0) {
        P.ctl[CTL_STEP] = k_step;
        P.ctl[CTL_WINDOWS] = nwin;
    }
}

// Threads of a part: the rows, whole warps.
int part_threads(int N, int ka) { return (N * ka + 31) / 32 * 32; }

template <class T, int NP, int H>
cudaError_t launch_res(const TspP &P, const DevTsp &t, int ka, cudaStream_t s, bool pdl)
{
    constexpr int NPS = NP + 4;
    const int N = P.N;
    const size_t smem = sizeof(float) * ((size_t)N * ka * NPS + (size_t)ka * NPS + N * ka) +
                        sizeof(uint32_t) * 2 * N * ka + sizeof(int) * 2 * ka;
    cudaError_t e = cudaFuncSetAttribute(k_tsp_resident<T, NP, H>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((P.A + ka - 1) / ka);
    cfg.blockDim = dim3(part_threads(N, ka) * H);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    TspD<NP> D = {};
    size_t pair = 0;   // packed: pairs c1 < c2 in order
    for (int c1 = 0; c1 < N; c1++)
        for (int c2 = c1 + 1; c2 < N; c2++, pair++) D.d[c1 * NP + c2] = D.d[c2 * NP + c1] = (float)t.packed[pair];
    return cudaLaunchKernelEx(&cfg, k_tsp_resident<T, NP, H>, P, D, ka);
}

// Eight cities a thread: two parts of 16, whose rows always fit, and four of 32
// where the CTA's 1,024 threads allow it; more agents a CTA (only when asked
// for) take whole rows (17 cities, 30 agents a CTA: 5.6 us a step, two parts of
// 16 cities 6.3 to 6.9).
template <class T>
cudaError_t launch_np(const TspP &P, const DevTsp &t, int ka, cudaStream_t s, bool pdl)
{
    if (P.N <= 16) return launch_res<T, 16, 2>(P, t, ka, s, pdl);
    if (4 * part_threads(P.N, ka) <= 1024) return launch_res<T, 32, 4>(P, t, ka, s, pdl);
    return launch_res<T, 32, 1>(P, t, ka, s, pdl);
}

}  // namespace

int tsp_pick_ka(const SolveDims &d, const DevTsp &t, int requested)
{
    if (d.prec == P_F64 || t.N > 32 || t.N < 2) return 0;
    const int nsm = dev_attr(cudaDevAttrMultiProcessorCount);
    const int kmax = 512 / t.N;   // registers: <= 512 threads of ~128 registers
    if (kmax < 1) return 0;
    if (requested > 0) return requested <= kmax ? requested : 0;
    // one CTA an SM in as few even waves as leave its rows in eight-city parts
    // (29 cities x 2,500 agents: three waves of six 7.9 us a step, three of the
    // most a CTA so holds, eight, 9.9)
    for (int waves = 1;; waves++) {
        const int ka = std::max(1, (d.A + waves * nsm - 1) / (waves * nsm));
        if (ka == 1 || (t.N <= 16 ? 2 : 4) * part_threads(t.N, ka) <= 1024) return ka;
    }
}

cudaError_t launch_tsp_resident(const SolveDims &d, const DevTsp &t, Work &w, int ka,
                                cudaStream_t s)
{
    TspP P;
    P.I2 = t.I2;
    P.sched = w.sched;
    P.x = w.x;
    P.y = w.y;
    P.Wp = w.Wp;
    P.tours = w.tours;
    P.valid = w.valid;
    P.stab = w.stab;
    P.bif = w.bif;
    P.prev = w.prev;
    P.ctl = w.ctl;
    P.N = t.N;
    P.A = d.A;
    P.Ap = d.Ap;
    P.W = d.W;
    P.nwin = d.nwin;
    P.period = d.period;
    P.threshold = d.threshold;
    P.qa8 = (float)(t.A / 8);
    P.qb4 = (float)(t.B / 4);
    P.qc4 = (float)(t.C / 4);
    P.dtxi0 = (float)(d.dt * 0.002);
    P.dt = (float)d.dt;
    const double p0 = 1.025 * 0.0 / d.steps;   // Update_XY pressure at step 0
    P.k1u = (float)(d.dt * (p0 + 1));
    P.k2u = (float)(d.dt * (p0 - 1));
    switch (d.prec) {
    case P_F32: return launch_np<float>(P, t, ka, s, d.pdl);
    case P_BF16: return launch_np<__nv_bfloat16>(P, t, ka, s, d.pdl);
    case P_F16: return launch_np<__half>(P, t, ka, s, d.pdl);
    default: return cudaErrorInvalidValue;
    }
}

// ---------------------------------------------------------------- streaming

namespace {

struct TspSP {
    const int32_t *__restrict__ rowptr;
    const uint32_t *__restrict__ colw;
    const double *__restrict__ vald;
    const double *__restrict__ I2d;     // [N]
    const double2 *__restrict__ ab;     // per step: a_t, b_t
    const void *xin;
    void *xout, *y;
    int64_t n;
    int32_t N, Ap, W, step;
    double dt, xi0;
};

// One thread of symplectic_kernel_tsp (src/kernels.cu:561-597), Jacobi.
template <class T>
__global__ void __launch_bounds__(256) k_tsp_step(const TspSP P)
{
    using A = typename St<T>::A;
    pdl_wait();
    pdl_trigger();
    const int64_t gw = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (gw >= P.n * P.W) return;
    const int64_t r = gw / P.W;
    const int w = (int)(gw - r * P.W);
    const int64_t idx = r * P.Ap + (int64_t)w * 32 + lane;
    const T *xi = (const T *)P.xin;
    T *xo = (T *)P.xout, *yp = (T *)P.y;
    A x = St<T>::ld(xi[idx]), y = St<T>::ld(yp[idx]);
    if (fabs(x) > A(1)) {
        x = spin_of(x);
        y = A(0);
    } else {
        A i1 = 0;
        for (int32_t e = P.rowptr[r]; e < P.rowptr[r + 1]; e++) {
            const A xv = St<T>::ld(xi[(int64_t)(P.colw[e] & 0x7fffffffu) * P.Ap + (int64_t)w * 32 + lane]);
            const A act = mul(xv, (A)1.005);
            i1 = sub(i1, mul((A)P.vald[e], act));
        }
        const double2 ab = P.ab[P.step];
        const A i2 = (A)P.I2d[r % P.N];
        const A t = mul((A)P.xi0, add(mul((A)2, i1), mul((A)ab.y, i2)));
        y = add(y, mul((A)P.dt, t));
        x = add(x, mul((A)P.dt, y));
        y = add(y, mul((A)mul(P.dt, -sub(1.0, ab.x)), x));
    }
    xo[idx] = St<T>::st(x);
    yp[idx] = St<T>::st(y);
}

// Update_XY at step 0 (the MaxCut kernel the reference reuses, src/ising_tsp.cu:155).
template <class T>
__global__ void k_tsp_prestep(T *x, T *y, int64_t count, double k1, double k2)
{
    using A = typename St<T>::A;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    A xv = St<T>::ld(x[i]), yv = St<T>::ld(y[i]);
    yv = add(yv, mul((A)k2, xv));
    xv = add(xv, mul((A)k1, yv));
    x[i] = St<T>::st(xv);
    y[i] = St<T>::st(yv);
}

struct TspWP {
    const void *x;
    uint32_t *Wp;
    int32_t *visits;   // [2][N][Ap] scratch (city, order)
    int32_t *tours, *valid, *stab;
    uint8_t *bif, *prev;
    int64_t n;
    int32_t N, A, Ap, W, step, threshold;
};

// update_window_tsp, src/kernels.cu:461-541: one thread per agent, serial over
// the N^2 rows, exactly as the reference.
template <class T>
__global__ void k_tsp_window(const TspWP P)
{
    pdl_wait();
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= P.A) return;
    const T *x = (const T *)P.x;
    int32_t *cv = P.visits, *ov = P.visits + (int64_t)P.N * P.Ap;
    bool valid = true, equal = true;
    for (int64_t i = 0; i < P.n; i++) {
        const uint32_t s = sbit(St<T>::ld(x[i * P.Ap + a]));
        const uint32_t cur = (P.Wp[i * P.W + (a >> 5)] >> (a & 31)) & 1u;
        if (s != cur) equal = false;
        if (!s) {
            const int64_t city = i % P.N, order = (i - city) / P.N;
            cv[city * P.Ap + a] += 1;
            ov[order * P.Ap + a] += 1;
        }
    }
    for (int i = 0; i < P.N; i++)
        if (cv[(int64_t)i * P.Ap + a] != 1 || ov[(int64_t)i * P.Ap + a] != 1) {
            valid = false;
            break;
        }
    for (int i = 0; i < P.N; i++) cv[(int64_t)i * P.Ap + a] = ov[(int64_t)i * P.Ap + a] = 0;
    const bool nb = !P.bif[a];
    int st = P.stab[a];
    st += (equal && nb);
    st = (!equal && nb) ? 0 : st;
    const bool b = (st == P.threshold - 1);
    P.stab[a] = st;
    P.bif[a] = b;
    P.prev[a] = b;
    if (valid) {
        P.valid[a] = P.step;
        for (int o = 0; o < P.N; o++)
            for (int c = 0; c < P.N; c++)
                if (!sbit(St<T>::ld(x[((int64_t)o * P.N + c) * P.Ap + a]))) P.tours[(int64_t)a * P.N + o] = c;
    }
    // current_spins = sign(X)
    for (int64_t i = 0; i < P.n; i++) {
        const uint32_t s = sbit(St<T>::ld(x[i * P.Ap + a]));
        uint32_t *p = &P.Wp[i * P.W + (a >> 5)];
        if (s) atomicOr(p, 1u << (a & 31));
        else atomicAnd(p, ~(1u << (a & 31)));
    }
}

template <class T>
cudaError_t stream_t(const SolveDims &d, const DevTsp &t, Work &w, const double2 *ab,
                     const double *I2d, int32_t *visits, cudaStream_t s, int *launches)
{
    const int64_t n = (int64_t)t.N * t.N;
    const double p0 = 1.025 * 0.0 / d.steps;
    k_tsp_prestep<T><<<(unsigned)((n * d.Ap + 255) / 256), 256, 0, s>>>(
        (T *)w.x, (T *)w.y, n * d.Ap, d.dt * (p0 + 1), d.dt * (p0 - 1));
    (*launches)++;
    cudaError_t e = cudaGetLastError();
    TspSP P;
    P.rowptr = t.qubo.rowptr;
    P.colw = t.qubo.colw;
    P.vald = t.qubo.vald;
    P.I2d = I2d;
    P.ab = ab;
    P.y = w.y;
    P.n = n;
    P.N = t.N;
    P.Ap = d.Ap;
    P.W = d.W;
    P.dt = d.dt;
    P.xi0 = 0.002;
    TspWP Q;
    Q.Wp = w.Wp;
    Q.visits = visits;
    Q.tours = w.tours;
    Q.valid = w.valid;
    Q.stab = w.stab;
    Q.bif = w.bif;
    Q.prev = w.prev;
    Q.n = n;
    Q.N = t.N;
    Q.A = d.A;
    Q.Ap = d.Ap;
    Q.W = d.W;
    Q.threshold = d.threshold;
    void *cur = w.x, *nxt = w.x2;
    const int nwin = d.nwin;
    int k = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((n * d.W + 7) / 8));
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = d.pdl ? 1 : 0;
    for (int wdx = 0; wdx < nwin && e == cudaSuccess; wdx++) {
        for (int it = 0; it < d.period && e == cudaSuccess; it++, k++) {
            P.xin = cur;
            P.xout = nxt;
            P.step = k;
            e = cudaLaunchKernelEx(&cfg, k_tsp_step<T>, P);
            void *tmp = cur;
            cur = nxt;
            nxt = tmp;
            (*launches)++;
        }
        Q.x = cur;
        Q.step = k;
        k_tsp_window<T><<<(d.A + 127) / 128, 128, 0, s>>>(Q);
        (*launches)++;
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    if (e == cudaSuccess && cur != w.x)
        e = cudaMemcpyAsync(w.x, cur, (size_t)n * d.Ap * sizeof(T), cudaMemcpyDeviceToDevice, s);
    return e;
}

}  // namespace

cudaError_t launch_tsp_stream(const SolveDims &d, const DevTsp &t, Work &w, cudaStream_t s,
                              int *launches)
{
    switch (d.prec) {
    case P_F32: return stream_t<float>(d, t, w, w.ab, t.I2d, w.visits, s, launches);
    case P_BF16: return stream_t<__nv_bfloat16>(d, t, w, w.ab, t.I2d, w.visits, s, launches);
    case P_F16: return stream_t<__half>(d, t, w, w.ab, t.I2d, w.visits, s, launches);
    default: return stream_t<double>(d, t, w, w.ab, t.I2d, w.visits, s, launches);
    }
}

namespace {

// Length of agent a's tour: the packed distance of every consecutive pair,
// the last city back to the first, summed in tour order in FP64 (src/ising_tsp.cu:272-287).
__global__ void __launch_bounds__(128) k_tsp_lengths(const int32_t *__restrict__ tours,
                                                     const int32_t *__restrict__ valid,
                                                     const double *__restrict__ Dd, int32_t N, int32_t A,
                                                     double *len)
{
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= A) return;
    if (valid[a] <= 0) {
        len[a] = __longlong_as_double(0x7ff8000000000000LL);   // NaN: no valid tour
        return;
    }
    const int32_t *t = tours + (int64_t)a * N;
    double s = 0.0;
    for (int i = 0; i < N; i++) {
        const int c1 = t[i], c2 = t[i + 1 < N ? i + 1 : 0];
        s = __dadd_rn(s, Dd[(int64_t)c1 * N + c2]);
    }
    len[a] = s;
}

}  // namespace

namespace {

// TSP_distances_EUC_2D / TSP_distances_GEO (src/kernels.cu:404-442) on the
// device, one thread per pair c1 < c2, with the reference's expressions and
// its (int) truncation (none for the float kind); the packed upper triangle,
// and the symmetric N x N tables of the TSP kernels (float and FP64).
__global__ void __launch_bounds__(256) k_tsp_dist(const double *__restrict__ xc, const double *__restrict__ yc,
                                                  int32_t N, int32_t kind, double *packed, float *D, double *Dd)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)N * N) return;
    const int c1 = (int)(t / N), c2 = (int)(t - (int64_t)c1 * N);
    if (c2 <= c1) return;
    double d;
    if (kind == 1) {   // GEO, kernels.cu:425-441
        const double R = 6378.388;
        const double q1 = cos(yc[c1] - yc[c2]);
        const double q2 = cos(xc[c1] - xc[c2]);
        const double q3 = cos(xc[c1] + xc[c2]);
        d = (double)(int)(R * acos(0.5 * ((1.0 + q1) * q2 - (1.0 - q1) * q3)) + 1.0);
    } else {           // EUC_2D, kernels.cu:404-423
        const double xd = xc[c1] - xc[c2], yd = yc[c1] - yc[c2];
        d = pow(xd * xd + yd * yd, 0.5);
        if (kind == 0) d = (double)(int)d;
    }
    packed[(int64_t)c2 + (int64_t)c1 * N - (int64_t)(c1 + 2) * (c1 + 1) / 2] = d;
    D[(int64_t)c1 * N + c2] = D[(int64_t)c2 * N + c1] = (float)d;
    Dd[(int64_t)c1 * N + c2] = Dd[(int64_t)c2 * N + c1] = d;
}

// The largest distance (exact in any order).
__global__ void __launch_bounds__(256) k_tsp_max(const double *__restrict__ packed, int64_t nd, double *mx)
{
    double m = 0;
    for (int64_t k = threadIdx.x; k < nd; k += blockDim.x) m = fmax(m, packed[k]);
    for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(FULL, m, o));
    __shared__ double w[8];
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < (int)(blockDim.x >> 5); i++) m = fmax(m, w[i]);
        *mx = fmax(m, w[0]);
    }
}

// Per-city distance sums (src/tsp_gpu.cu:51-68 adds each pair to both of its
// cities walking the packed array, so city c receives its pairs in ascending
// order of the other city), then the linear field of src/kernels.cu:591-592,
// -1 (A rowsum + (N - 2)(B + C)) / 2 with B = C = scale * max distance,
// rounded per operation as the host states it.
__global__ void __launch_bounds__(128) k_tsp_rows(const double *__restrict__ Dd, int32_t N, double A,
                                                  double scale, const double *__restrict__ mx,
                                                  double *rowsum, double *I2d, float *I2)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= N) return;
    double r = 0;
    for (int k = 0; k < N; k++)
        if (k != c) r = __dadd_rn(r, Dd[(int64_t)c * N + k]);
    rowsum[c] = r;
    const double B = __dmul_rn(scale, *mx);
    const double v = __ddiv_rn(__dmul_rn(-1.0, __dadd_rn(__dmul_rn(A, r), __dmul_rn((double)(N - 2), __dadd_rn(B, B)))),
                               2.0);
    I2d[c] = v;
    I2[c] = (float)v;
}

}  // namespace

cudaError_t launch_tsp_setup(const double *xc, const double *yc, int32_t N, int32_t kind, double A, double scale,
                             double *packed, double *mx, double *rowsum, DevTsp &t, cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(t.D, 0, sizeof(float) * N * N, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(t.Dd, 0, sizeof(double) * N * N, s);
    if (e != cudaSuccess) return e;
    const int64_t nn = (int64_t)N * N;
    k_tsp_dist<<<(unsigned)((nn + 255) / 256), 256, 0, s>>>(xc, yc, N, kind, packed, t.D, t.Dd);
    k_tsp_max<<<1, 256, 0, s>>>(packed, (int64_t)N * (N - 1) / 2, mx);
    k_tsp_rows<<<(N + 127) / 128, 128, 0, s>>>(t.Dd, N, A, scale, mx, rowsum, t.I2d, t.I2);
    return cudaGetLastError();
}

cudaError_t launch_tsp_lengths(const DevTsp &t, const int32_t *tours, const int32_t *valid, int32_t A,
                               double *len, cudaStream_t s)
{
    if (A <= 0) return cudaSuccess;
    k_tsp_lengths<<<(A + 127) / 128, 128, 0, s>>>(tours, valid, t.Dd, t.N, A, len);
    return cudaGetLastError();
}

}  // namespace sbx
