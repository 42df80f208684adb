// k_resident_f64.cu -- resident MaxCut SB kernel in FP64 for small graphs, +-1
// weights: one CTA owns one agent of every row and keeps its x, y in shared
// memory for all the steps of a launch (agents never interact), with one
// __syncthreads() per step in the Jacobi order of the reference kernel
// (src/kernels.cu:211-269).  The arithmetic is the streaming kernel's FP64 path
// (separately rounded products and sums in the reference's order), so the
// states are identical.
//
// A launch per step takes 2.3 us however small the graph; here a step costs
// its latency and the SM's FP64 pipe (two lanes a cycle, about eight
// operations per spin), which is why one agent per CTA: it spreads the agents
// over the SMs.  The matrix is read in sliced form (engine.h, DevSell); a row's
// sign is a byte, four neighbours make a word, and a byte dot product counts
// them.
#include "k_step.cuh"

#include <algorithm>
#include <cmath>

namespace sbx {

namespace {

struct R64P {
    const int2 *__restrict__ off;      // sliced matrix, entries scaled by 1
    const float *__restrict__ deg;
    const uint2 *__restrict__ col;
    const int32_t *__restrict__ perm;
    const Coef4 *__restrict__ coef;    // per step: k1, k2 (clamped), k1, k2 (raw)
    double *x, *y;                     // global [n][Ap]
    uint32_t *Wp, *fin;                // global planes [n][W]
    int32_t *stab;
    uint8_t *bif, *prev;
    int32_t *ctl;
    int32_t *wincount;                 // bifurcated agents after each window
    int32_t n, A, Ap, W, period, threshold, uw, fused, step0, nsteps, first;
    double c0;
};

// Bit sh of a shared plane word.
__device__ __forceinline__ void bit_put(uint32_t *p, uint32_t bit, int sh)
{
    if (bit) atomicOr(p, 1u << sh);
    else atomicAnd(p, ~(1u << sh));
}

__global__ void __launch_bounds__(1024) k_res64(const R64P P)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int n = P.n, NT = blockDim.x, tid = threadIdx.x;
    double *xs = (double *)smem, *ys = xs + n;
    uint8_t *S0 = (uint8_t *)(ys + n), *S1 = S0 + n + 1;   // one byte a row, and the zero row
    uint8_t *Wb = S1 + n + 1;                              // window spins
    __shared__ int s_chg, s_new, s_stop;

    pdl_wait();
    const int a = blockIdx.x, wg = a >> 5, sh = a & 31;
    // early exit of the update-window mode (src/ising.cu:200-211)
    if (tid == 0) {
        s_stop = P.ctl[CTL_STOP];
        if (!s_stop && P.uw && P.step0 > 0 && P.wincount[P.step0 / P.period - 1] == P.A) s_stop = 1;
        s_chg = 0;
        S0[n] = 0;
        S1[n] = 0;
    }
    __syncthreads();
    if (s_stop) {
        if (a == 0 && tid == 0) P.ctl[CTL_STOP] = 1;
        return;
    }
    // the agent's window state, kept by thread 0
    int stab = 0;
    bool bif = false, prev = false;
    if (tid == 0) {
        stab = P.stab[a];
        bif = P.bif[a] != 0;
        prev = P.prev[a] != 0;
    }
    // the state: at step 0 after the pre-step Update_XY (src/ising.cu:188); the
    // unfused step begins with Update_XY of its own step
    const int32_t k0 = P.step0;
    const Coef4 cu = P.coef[k0];
    const int nxy = (P.first ? 1 : 0) + (P.fused ? 0 : 1);
    uint8_t *Sc = (k0 & 1) ? S1 : S0;
    for (int s = tid; s < n; s += NT) {
        const int64_t r = __ldg(&P.perm[s]);
        double x = P.x[r * P.Ap + a], y = P.y[r * P.Ap + a];
        for (int t = 0; t < nxy; t++) {
            y = madd(cu.w, x, y);
            x = madd(cu.z, y, x);
        }
        xs[s] = x;
        ys[s] = y;
        Sc[s] = (uint8_t)sbit(x);
        Wb[s] = (uint8_t)((P.Wp[r * P.W + wg] >> sh) & 1u);
    }
    __syncthreads();
    for (int32_t it = 0; it < P.nsteps; it++) {
        const int32_t k = k0 + it;
        const uint8_t *Sin = (k & 1) ? S1 : S0;
        uint8_t *Snx = (k & 1) ? S0 : S1;
        const bool win = (k + 1) % P.period == 0, last = it == P.nsteps - 1;
        const Coef4 c = P.coef[k], cn = P.coef[k + 1];
        bool chg = false;
        for (int s = tid; s < n; s += NT) {
            const int2 o = __ldg(&P.off[s >> 5]);
            const uint2 *cp = P.col + (int64_t)o.x * 32 + (s & 31);
            int cnt = 0;
            for (int b = 0; b < o.y; b++) {
                const uint2 e = __ldg(cp + b * 32);
                uint32_t w = __byte_perm(__byte_perm(Sin[e.x & 0x7fffu], Sin[(e.x >> 16) & 0x7fffu], 0x0040),
                                         __byte_perm(Sin[e.y & 0x7fffu], Sin[(e.y >> 16) & 0x7fffu], 0x0040), 0x5410);
                w ^= prmt<0xfdb9>(e.x, e.y) & 0x01010101u;   // the weights' signs
                cnt = __dp4a(w, 0x01010101u, (uint32_t)cnt);
            }
            const double tv = (double)(2 * cnt - (int)__ldg(&P.deg[s]));
            double x = xs[s], y = ys[s];
            // src/kernels.cu:236-262, or mat_mult + confine (:150-209)
            const bool out = fabs(x) > 1.0;
            const double xc = spin_of(x);
            y = out ? 0.0 : madd(P.c0, tv, y);
            x = out ? xc : x;
            if (P.fused) {
                x = madd(c.x, y, x);
                y = madd(c.y, x, y);
            }
            const uint32_t wb = sbit(x);   // the sign the window sees
            if (!P.fused && !last) {
                y = madd(cn.w, x, y);
                x = madd(cn.z, y, x);
            }
            xs[s] = x;
            ys[s] = y;
            Snx[s] = (uint8_t)sbit(x);
            if (win) {
                chg |= wb != Wb[s];
                Wb[s] = (uint8_t)wb;
            }
        }
        if (win) {
            // the agent's window bookkeeping, src/kernels.cu:46-79
            if (chg) s_chg = 1;
            __syncthreads();
            if (tid == 0) {
                const bool equal = !s_chg, nb = !bif;
                stab += (equal && nb);
                stab = (!equal && nb) ? 0 : stab;
                bif = stab == P.threshold - 1;
                s_new = bif != prev;
                prev = bif;
                if (P.uw && bif) atomicAdd(&P.wincount[(k + 1) / P.period - 1], 1);
            }
            __syncthreads();
            if (s_new)
                for (int s = tid; s < n; s += NT)
                    bit_put(&P.fin[(int64_t)__ldg(&P.perm[s]) * P.W + wg], Wb[s], sh);
            if (tid == 0) s_chg = 0;
        }
        __syncthreads();
    }
    // the state back (chunked runs continue from it; get_state reads it)
    for (int s = tid; s < n; s += NT) {
        const int64_t r = __ldg(&P.perm[s]);
        P.x[r * P.Ap + a] = xs[s];
        P.y[r * P.Ap + a] = ys[s];
        bit_put(&P.Wp[r * P.W + wg], Wb[s], sh);
    }
    if (tid == 0) {
        P.stab[a] = stab;
        P.bif[a] = bif;
        P.prev[a] = prev;
        if (a == 0) {
            P.ctl[CTL_STEP] = P.step0 + P.nsteps;
            P.ctl[CTL_WINDOWS] = (P.step0 + P.nsteps) / P.period;
        }
    }
}

size_t smem64(int64_t n) { return (size_t)n * 19 + 2; }
int threads64(int64_t n) { return (int)std::min<int64_t>(1024, std::max<int64_t>(64, (n + 31) / 32 * 32)); }

}  // namespace

bool resident64_pick(const SolveDims &d, const DevCsr &J)
{
    if (d.prec != P_F64 || !J.unit || J.n > 32767) return false;
    if (smem64(d.n) + 1024 > (size_t)dev_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin)) return false;
    // The shorter step (microseconds, both sides fitted on GB300, mean error 11%,
    // over 50 to 6,000 rows, mean degrees 2 to 900, stars and R-MAT, and 1 to
    // 1,024 agents): an SM's agents one after another through its FP64 pipe, and
    // its CTAs' walks over the neighbours, where one thread walks the longest
    // row, against a launch, the whole GPU's FP64 pipes and 32 agents a gathered
    // word, heavy rows in chunks.  300 rows of degree 12: 1.8 against 3.3 at 128
    // agents, 8.9 against 7.6 at 1,024; 128 agents and 1,000 rows of degree 900:
    // 34.5 against 19.6; a star of 1,000: 10.2 against 7.7.
    const double nsm = std::max(1, dev_attr(cudaDevAttrMultiProcessorCount));
    const double n = (double)d.n, deg = (double)J.nnz / n, more = std::max(0.0, deg - 12);
    const double waves = std::ceil(d.A / nsm), together = std::max(1, 1024 / threads64(d.n));   // CTAs of an SM
    const double walk = more / 4 * std::max(0.04, 0.13e-3 * n) + 6e-3 * ((double)J.max_deg - deg);
    return 0.75 + 3.7e-3 * n * waves + std::ceil(waves / together) * walk <
           2.4 + 17e-6 * n * d.Ap + more * (0.08e-6 * n * d.Ap) + std::min(more, kHeavy - 12.0) * 7e-3 +
               (J.max_deg > kHeavy ? 3.3 : 0.0);
}

cudaError_t launch_resident64(const SolveDims &d, const DevCsr &J, Work &w, int32_t step0, int32_t nsteps, bool first,
                              cudaStream_t s)
{
    if (!J.sell[1].base) return cudaErrorInvalidValue;
    R64P P;
    P.off = J.sell[1].off;
    P.deg = J.sell[1].deg;
    P.col = J.sell[1].col;
    P.perm = J.perm;
    P.coef = (const Coef4 *)w.coef64;
    P.x = (double *)w.x;
    P.y = (double *)w.y;
    P.Wp = w.Wp;
    P.fin = w.fin;
    P.stab = w.stab;
    P.bif = w.bif;
    P.prev = w.prev;
    P.ctl = w.ctl;
    P.wincount = w.wincount;
    P.n = (int32_t)d.n;
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
    P.c0 = d.c0;
    const size_t smem = smem64(d.n);
    cudaError_t e = cudaFuncSetAttribute(k_res64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return launch(k_res64, dim3((unsigned)d.A), dim3((unsigned)threads64(d.n)), smem, s, d.pdl, P);
}

}  // namespace sbx
