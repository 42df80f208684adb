// k_init.cu -- the reference's initial state, generated on the device.
//
// The reference fills X and Y on the host with glibc rand() after
// srand(seed), interleaved X[i], Y[i] (src/ising.cu:91-95), or Y only with
// X = 0 for TSP (src/ising_tsp.cu:55-59).  glibc's rand() (TYPE_3 additive
// feedback generator) is the linear recurrence over Z/2^32
//     u[i] = u[i-31] + u[i-3],   output_k = u[344+k] >> 1,
// seeded by u[0] = seed (0 -> 1), u[i] = 16807 u[i-1] mod (2^31-1) for
// i = 1..30, u[31..33] = u[0..2].  Its 31-word window therefore advances by a
// fixed 31x31 matrix M, and M^k jumps k outputs at once.  Each device thread
// jumps to the start of its own chunk of outputs with precomputed powers
// M^(L*2^b) and then runs the recurrence serially, so the whole stream is
// produced in parallel and equals, value for value, what rand() returns.
// The powers do not depend on the seed; one launch can fill many instances,
// each from its own seed (its own 31-word starting window).
#include "common.cuh"
#include "engine.h"

#include <algorithm>
#include <cstring>

namespace sbx {

namespace {

constexpr int R = 31;

void matmul31(const uint32_t *a, const uint32_t *b, uint32_t *c)
{
    uint32_t t[R * R];
    for (int i = 0; i < R; i++)
        for (int j = 0; j < R; j++) {
            uint32_t s = 0;
            for (int k = 0; k < R; k++) s += a[i * R + k] * b[k * R + j];
            t[i * R + j] = s;
        }
    memcpy(c, t, sizeof t);
}

}  // namespace

void rand_seed_window(uint32_t seed, uint32_t *V0)
{
    // the minimal-standard LCG, then the lag-31 recurrence up to the first
    // returned value; V0 = u[313..343], the window before output 0
    uint32_t u[344];
    uint64_t word = seed ? seed : 1u;
    u[0] = (uint32_t)word;
    for (int i = 1; i < 31; i++) {
        word = (16807u * word) % 2147483647u;
        u[i] = (uint32_t)word;
    }
    for (int i = 31; i < 34; i++) u[i] = u[i - 31];
    for (int i = 34; i < 344; i++) u[i] = u[i - 31] + u[i - 3];
    for (int i = 0; i < R; i++) V0[i] = u[313 + i];
}

void rand_jump_matrices(int64_t L, int nbits, std::vector<uint32_t> &out)
{
    // M: window (u[i-31..i-1]) -> (u[i-30..i]); out[b] = M^(L*2^b)
    uint32_t M[R * R] = {0}, P[R * R], Acc[R * R];
    for (int i = 0; i < R - 1; i++) M[i * R + i + 1] = 1;
    M[(R - 1) * R + 0] = 1;
    M[(R - 1) * R + 28] = 1;
    for (int i = 0; i < R * R; i++) Acc[i] = (i % (R + 1)) == 0;
    memcpy(P, M, sizeof P);
    for (int64_t e = L; e; e >>= 1) {
        if (e & 1) matmul31(Acc, P, Acc);
        matmul31(P, P, P);
    }
    out.assign((size_t)nbits * R * R, 0);
    for (int b = 0; b < nbits; b++) {
        memcpy(&out[(size_t)b * R * R], Acc, sizeof Acc);
        matmul31(Acc, Acc, Acc);
    }
}

namespace {

// (((double)rand() / RAND_MAX) * 2 - 1) / 10 with one FP64 rounding per
// operation, src/ising.cu:91-95.
__device__ __forceinline__ double init_value64(uint32_t r)
{
    return __ddiv_rn(__dsub_rn(__dmul_rn(__ddiv_rn((double)r, 2147483647.0), 2.0), 1.0), 10.0);
}

// The same value rounded to FP32, without FP64 arithmetic (two FP64 divisions
// per value bounded the init kernel): the exact value is t / (10 RAND_MAX)
// with t = 2 r - RAND_MAX an odd 32-bit integer, taken as a 64-bit product
// with 2^98 / (10 RAND_MAX).  The FP64 expression differs from it by less
// than 2^-38 of itself for |t| >= 2^18, so away from a rounding boundary of
// FP32 by more than that both round alike; the rest (1.8e-4 of the values)
// take the FP64 expression.  Compared with it for all 2^31 values of r.
__device__ __forceinline__ float init_value32(uint32_t r)
{
    constexpr uint32_t C1 = 0xccccccceu, C0 = 0x6666666au;   // 2^98 / (10 (2^31 - 1))
    const int32_t t = (int32_t)(2u * r - 2147483647u);
    const uint32_t u = (uint32_t)abs(t);
    const int lz = __clz((int)u);
    const uint32_t un = u << lz;
    uint64_t m = (uint64_t)un * C1 + (((uint64_t)un * C0) >> 32);
    int e = 61 - lz;   // biased FP32 exponent of a value m * 2^(-66 - lz) with m's top bit at 2^63
    if (!(m >> 63)) {
        m <<= 1;
        e--;
    }
    const uint64_t rem = m & ((1ull << 40) - 1);
    if (u < (1u << 18) || rem - ((1ull << 39) - (1ull << 25)) < (2ull << 25)) return (float)init_value64(r);
    const uint32_t man = (uint32_t)(m >> 40) + (uint32_t)(rem >> 39);   // may carry into the exponent
    return __uint_as_float((((uint32_t)(e + 63)) << 23) + (man - (1u << 23)) + ((uint32_t)t & 0x80000000u));
}

template <class T> __device__ __forceinline__ T init_value(uint32_t r) { return St<T>::st(init_value32(r)); }
template <> __device__ __forceinline__ double init_value<double>(uint32_t r) { return init_value64(r); }

// One thread: find its instance, jump to its chunk's start, emit L outputs in
// rounds of 62 (31 agents' x and y, or 62 y for TSP).  A round's raw values
// go through the warp's shared stage, and the warp converts and stores one
// thread's run at a time: consecutive lanes hold consecutive agents, so a
// store covers two or three sectors instead of one sector per lane.
// slot (MaxCut only, may be null): the row of the state that takes the
// instance's row r, as a global row (row_off + r -> slot[row_off + r]).
// Bound: issue (about 60 instructions per output, the jump included).
constexpr int kRound = 62;
constexpr int kInitNT = 64;

template <class T>
__global__ void __launch_bounds__(kInitNT) k_rand_init(T *x, T *y, int32_t Ap, int tsp, int64_t L, int shift,
                                                       const uint32_t *__restrict__ mats,
                                                       const RandInst *__restrict__ inst, int count,
                                                       int64_t total_threads,
                                                       const int32_t *__restrict__ slot)
{
    struct Run {
        int64_t row0, row;   // the instance's first row; the run's first row in it
        int32_t a, A, left;  // the run's first agent, agents per row, outputs of this round
    };
    __shared__ uint32_t stage[kInitNT / 32][32][kRound + 1];
    __shared__ Run s_run[kInitNT / 32][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t t = (int64_t)blockIdx.x * kInitNT + threadIdx.x;
    int64_t left = 0, row = 0, row0 = 0;
    int32_t a = 0, A = 1;
    uint32_t v[R];
    if (t < total_threads) {
        int lo = 0, hi = count - 1;   // last instance with thread_base <= t
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (inst[mid].thread_base <= t) lo = mid;
            else hi = mid - 1;
        }
        const RandInst &I = inst[lo];
        const int64_t lt = t - I.thread_base;
        A = I.A;
        row0 = I.row_off;
        const int64_t o0 = lt * L, outputs = I.n * I.A * (tsp ? 1 : 2);
        left = max((int64_t)0, min(L, outputs - o0));
        const int64_t e0 = tsp ? o0 : o0 >> 1;   // L is even: x and y of an agent stay together
        row = e0 / A;
        a = (int32_t)(e0 - row * A);
#pragma unroll
        for (int i = 0; i < R; i++) v[i] = I.V0[i];
        // chunk lt starts lt 2^shift rounds in
        for (int b = 0; left > 0 && (lt >> b) != 0; b++) {
            if (!((lt >> b) & 1)) continue;
            const uint32_t *P = mats + (size_t)(b + shift) * R * R;
            uint32_t nv[R];
#pragma unroll
            for (int i = 0; i < R; i++) {
                uint32_t s = 0;
#pragma unroll
                for (int k = 0; k < R; k++) s += __ldg(&P[i * R + k]) * v[k];
                nv[i] = s;
            }
#pragma unroll
            for (int i = 0; i < R; i++) v[i] = nv[i];
        }
    }
    const int per = tsp ? kRound : kRound / 2;   // agents of a round
    while (__any_sync(FULL, left > 0)) {
        if (left > 0) {
            // Circular window: at phase q, v[q] holds u[i-31] and v[(q+28)%31] u[i-3].
#pragma unroll 1
            for (int h = 0; h < kRound; h += R) {
#pragma unroll
                for (int q = 0; q < R; q++) {
                    v[q] += v[(q + 28) % R];
                    stage[warp][lane][h + q] = v[q] >> 1;
                }
            }
        }
        s_run[warp][lane] = Run{row0, row, a, A, (int32_t)min(left, (int64_t)kRound)};
        __syncwarp();
        for (int k = 0; k < 32; k++) {
            const Run rn = s_run[warp][k];
            for (int e = lane; e < per && (tsp ? e : 2 * e) < rn.left; e += 32) {
                int64_t rr = rn.row;
                int32_t aa = rn.a + e;
                while (aa >= rn.A) {
                    aa -= rn.A;
                    rr++;
                }
                const int64_t srow = slot ? (int64_t)__ldg(&slot[rn.row0 + rr]) : rn.row0 + rr;
                const int64_t idx = srow * Ap + aa;
                if (tsp) {
                    y[idx] = init_value<T>(stage[warp][k][e]);   // x stays zero
                } else {
                    x[idx] = init_value<T>(stage[warp][k][2 * e]);
                    y[idx] = init_value<T>(stage[warp][k][2 * e + 1]);
                }
            }
        }
        __syncwarp();
        left -= kRound;
        a += per;
        while (a >= A) {
            a -= A;
            row++;
        }
    }
}

template <class T>
cudaError_t launch_t(void *x, void *y, int32_t Ap, int tsp, int64_t L, int shift, const uint32_t *mats,
                     const RandInst *inst, int count, int64_t total_threads, const int32_t *slot,
                     cudaStream_t s)
{
    const int64_t grid = (total_threads + kInitNT - 1) / kInitNT;
    if (grid == 0) return cudaSuccess;
    k_rand_init<T><<<(unsigned)grid, kInitNT, 0, s>>>((T *)x, (T *)y, Ap, tsp, L, shift, mats, inst, count,
                                                      total_threads, slot);
    return cudaGetLastError();
}

}  // namespace

// Outputs per thread: kRound 2^shift, the largest of shifts 0..6 that leaves
// enough threads to fill the GPU.  Short chunks cost more jumps (each set bit
// of the thread's number is a 31 x 31 product), long ones leave SMs idle:
// 25,600 outputs in 26 threads of 992 took 1.0 ms, most of it one thread's
// serial FP64 divisions.
int rand_chunk_shift(int64_t outputs)
{
    const int64_t fill = 640 * (int64_t)std::max(1, dev_attr(cudaDevAttrMultiProcessorCount));
    int s = 6;
    while (s > 0 && (outputs / kRound >> s) < fill) s--;
    return s;
}
int64_t rand_round() { return kRound; }

cudaError_t launch_rand_init(int prec, void *x, void *y, int32_t Ap, bool tsp, int shift, const uint32_t *mats,
                             const RandInst *inst, int count, int64_t total_threads, const int32_t *slot,
                             cudaStream_t s)
{
    if (tsp) slot = nullptr;
    const int64_t L = (int64_t)kRound << shift;
    switch (prec) {
    case P_F32: return launch_t<float>(x, y, Ap, tsp, L, shift, mats, inst, count, total_threads, slot, s);
    case P_BF16: return launch_t<__nv_bfloat16>(x, y, Ap, tsp, L, shift, mats, inst, count, total_threads, slot, s);
    case P_F16: return launch_t<__half>(x, y, Ap, tsp, L, shift, mats, inst, count, total_threads, slot, s);
    default: return launch_t<double>(x, y, Ap, tsp, L, shift, mats, inst, count, total_threads, slot, s);
    }
}

}  // namespace sbx
