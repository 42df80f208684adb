// engine.h -- internal interface between the C-ABI host layer (api.cpp) and
// the CUDA launchers (k_*.cu).  Not part of the public ABI.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

namespace sbx {

enum Prec { P_F32 = 0, P_BF16 = 1, P_F16 = 2, P_F64 = 3 };

// One instance of the reference's init stream (k_init.cu): rows
// [row_off, row_off + n) x agents [0, A) of x, y from srand(seed)'s window V0;
// its device threads are thread_base .. thread_base + ceil(outputs/L) - 1.
struct RandInst {
    int64_t row_off, n, thread_base;
    int32_t A, pad;
    uint32_t V0[31];
};

// Rows with more neighbours than this are "heavy" (+-1 weights): the step
// kernel counts them in chunks of kHeavy; byte counters (2 per neighbour)
// never overflow.
constexpr int kHeavy = 127;

// Mixed count mode (kernels with heavy rows): light rows of at least this
// many neighbours are counted in bit planes, shorter ones in byte counters
// (R-MAT scale 20 on GB300: 8, 12 and 20 timed within 1%).
constexpr int kBitsMin = 12;

// Rows of 1 to kLight neighbours of a +-1 matrix whose rows are visited in
// degree order have a record of eight words: row, degree, column words.
constexpr int kLight = 6;

inline size_t prec_bytes(int p) { return p == P_F64 ? 8 : p == P_F32 ? 4 : 2; }

// An attribute of the calling thread's current device (0 when the query
// fails); queried each time, so contexts on different devices see their own.
inline int dev_attr(cudaDeviceAttr a)
{
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&v, a, dev) != cudaSuccess) return 0;
    return v;
}

struct DevBsm;

// A matrix in sliced form for the resident kernels: row s is the row of slot
// s (perm[s], decreasing degree), 32 consecutive slots a slice, a slice's
// entries in blocks of four per row, blocks as long as its longest row needs.
// Lane l of a warp reads its block as one 8-byte word next to its
// neighbours' (a row-by-row layout cost a cache line per lane and entry).
// An entry is its column's slot times `scale` (the byte offset of the slot in
// the kernel's sign array), bit 15 the sign of a -1 weight; entries past a
// row's end name slot n, whose signs are all zero.  val: the negated weights
// of other matrices, zero past a row's end.
struct DevSell {
    void *base = nullptr;              // one allocation holding the arrays below
    const int2 *off = nullptr;         // per slice: first block, blocks
    const float *deg = nullptr;        // per slot: entries
    const uint2 *col = nullptr;        // [blocks][32]
    const float4 *val = nullptr;       // [blocks][32], null for +-1 weights
};

// MaxCut / QUBO matrix on the device.  colw holds the column index; when every
// weight is +-1 ("unit"), bit 31 holds the weight's sign and no value array is
// read by the step kernels.
struct DevCsr {
    int64_t n = 0, nnz = 0;
    int32_t *rowptr = nullptr;
    uint32_t *colw = nullptr;
    double *vald = nullptr;
    float *valf = nullptr;
    int32_t *perm = nullptr; // rows in decreasing degree (resident kernel order)
    bool skewed = false;     // max degree > 8x mean: the step kernel visits rows in perm order
    int64_t nheavy = 0;      // heavy rows: the first nheavy entries of perm
    int64_t niso = 0;        // isolated rows (degree 0): the last niso entries of perm
    uint32_t *light = nullptr;   // records of the nlight rows before those (kLight)
    int32_t nlight = 0;
    // Heavy rows (unit weights, degree > kHeavy) are split into chunks of
    // kHeavy neighbours, each counted by its own work item of the step kernel.
    int32_t *hchunk = nullptr;    // per row: first chunk of a heavy row, else -1
    int32_t *chunk_row = nullptr; // per chunk: its row
    int32_t nchunks = 0;
    // Batched (block-diagonal) matrices: dt*xi0 of each row's instance, and
    // the instance of each row; null for a single problem.
    float *c0r32 = nullptr;
    double *c0r64 = nullptr;
    int32_t *rinst = nullptr;
    // batched: instances, their agent counts and weight sums (per-window trace)
    int32_t ninst = 0;
    int32_t *iagents = nullptr;
    double *iwsum = nullptr;
    bool weights_always = false;  // the device copy holds the weights even when all are +-1
    bool unit = false;       // all |w| == 1
    bool allpos = false;     // all w == +1 (unit, no sign bits)
    bool integer = false;    // all integer-valued, small enough for int32 sums
    double wsum = 0;         // reference csr.sum
    int32_t max_deg = 0;
    std::vector<double> hval;   // host copy of values (xi0)
    std::vector<int32_t> hrowptr, hcol, hperm;
    // The sliced forms of the resident kernels, built on first use: [0] entries
    // scaled by 4 (sign words), [1] by 1 (sign bytes).
    DevSell sell[2];
    // Batched: the plan of the shared-memory-plane step kernel, when the
    // solve uses it (k_batch_smem.cu)
    const DevBsm *bsm = nullptr;
};

// Control words shared by the kernels of one solve.
// CTL_ERR: a kernel gave up a bounded wait (1), or the on-chip batch kernel's
// layout does not fit (kErrMisfit); set, never cleared by kernels.
constexpr int kErrMisfit = 2;
enum Ctl { CTL_STEP = 0, CTL_STOP = 1, CTL_WINDOWS = 2, CTL_NBIF = 3, CTL_TRACED = 4, CTL_ERR = 5, CTL_N = 8 };

// One window of a traced solve: SB steps run, best cut over the agents of
// the window spins, nanoseconds since the loop began (device clock).
struct TraceRec {
    long long steps;
    double best;
    long long t_ns;
    long long pad;
};

// Device buffers of one solve (grown on demand, owned by the context).
struct Work {
    void *x = nullptr, *y = nullptr, *x2 = nullptr;
    uint32_t *S[2] = {nullptr, nullptr};
    uint32_t *Wp = nullptr, *fin = nullptr, *chg = nullptr, *newmask = nullptr;
    int32_t *stab = nullptr;
    uint8_t *bif = nullptr, *prev = nullptr;
    int32_t *ctl = nullptr;
    int32_t *wincount = nullptr;          // bifurcated agents after each window
    int32_t *visits = nullptr;            // TSP streaming window scratch
    double2 *ab = nullptr;                // TSP (a_t, b_t) per step, FP64
    float2 *sched = nullptr;              // TSP (b_t, dt*-(1-a_t)) per step
    uint32_t *part = nullptr;             // heavy-row partial counts
    int32_t *hcount = nullptr;            // heavy rows: finished chunks per (row, segment)
    int32_t *gbar = nullptr;              // window barrier of co-resident launches
    unsigned long long *eacc = nullptr;   // per-agent cut accumulators
    double *cut = nullptr;                // per-agent cuts
    double *stats = nullptr;              // k_stats output, 7 per problem
    double *cutrow = nullptr;             // non-integer cuts: a block of rows' halves [row][Ap]
    TraceRec *trace = nullptr;            // per-window records; trace_t0: loop start
    long long *trace_t0 = nullptr;
    double *btrace = nullptr;             // batched: best cut [window][instance]
    int32_t *tours = nullptr, *valid = nullptr;
    uint32_t *rjump = nullptr;            // rand jump matrices (computed once)
    RandInst *rinst = nullptr;            // init instances of the current solve
    float *coef32 = nullptr;              // per-step coefficients (float4 / step)
    double *coef64 = nullptr;             // the same in FP64 (double4 / step)
    size_t cap_x = 0, cap_y = 0, cap_x2 = 0, cap_S0 = 0, cap_S1 = 0, cap_Wp = 0, cap_fin = 0,
           cap_chg = 0, cap_new = 0, cap_stab = 0, cap_bif = 0, cap_prev = 0, cap_ctl = 0,
           cap_win = 0, cap_visits = 0, cap_ab = 0, cap_sched = 0, cap_eacc = 0, cap_cut = 0,
           cap_trace = 0, cap_t0 = 0, cap_btrace = 0, cap_tours = 0, cap_valid = 0, cap_rj = 0, cap_c32 = 0, cap_c64 = 0, cap_part = 0, cap_rinst = 0, cap_hcount = 0, cap_gbar = 0, cap_stats = 0, cap_cutrow = 0;
    bool rjump_ready = false;
};

// One solve's shape and scalars.
struct SolveDims {
    int64_t n = 0;
    int32_t A = 0, Ap = 0, W = 0;
    int prec = P_F32;
    int32_t steps = 0, period = 100, threshold = 25;
    int32_t nwin = 0;   // TSP: windows to run
    int fused = 1, uw = 0;
    double dt = 0.1, xi0 = 0, c0 = 0;
    bool pdl = true;
    // streaming step tile: agents per lane (0: widest vector that divides
    // Ap), lanes per row (32, 16, 8, 4), threads per CTA
    int32_t tv = 0, tlr = 32, tbt = 256;
    int32_t tcm = 0;         // +-1 rows: 0 byte counters per lane, 1 bit planes per word, 2 mixed
    int32_t tst = 0;         // 1: whole-warp rows staged through shared memory (bulk copies)
    int trace = 0;           // per-window best-cut records: 1 one problem, 2 batched
    int32_t steps_run = 0;   // resident batch: SB steps of the run
    int giveup = 0;          // SBX_FLAG_TEST_GIVEUP: bounded waits give up at once
    int tbsm = 0;            // batched: the shared-memory-plane step kernel (J.bsm),
                             // its CTA size (512 or 1024); 0: not used
};

// Agents that a row's lanes of the streaming step hold: the padded ones, up to
// the widest whole-warp tile in a power of two (rows sharing a warp), past it in
// whole tiles.
inline int tile_agents(const SolveDims &d)
{
    const int most = prec_bytes(d.prec) == 2 ? 256 : 128;
    int a = 32;
    while (a < most && a < d.Ap) a *= 2;
    return d.Ap > most ? (d.Ap + most - 1) / most * most : a;
}

// Plan of the batched step kernel with per-instance sign planes in shared
// memory (k_batch_smem.cu): the rows cut into one contiguous run per CTA,
// each run into segments at instance boundaries.
struct DevBsm {
    uint16_t *lcol = nullptr;     // per entry: local column | weight sign << 15; rows padded
                                  // to blocks of eight with the all-zero row (local row n_i)
    uint32_t *rinfo = nullptr;    // per row: first block of eight entries << 7 | degree
    int32_t *seg = nullptr;       // per segment: instance, first row, end row (global rows)
    int32_t *cta_seg = nullptr;   // per CTA: first segment; grid + 1 entries
    int32_t *ioff = nullptr;      // per instance: first row
    int32_t *in = nullptr;        // per instance: rows
    int32_t grid = 0;
    int64_t max_rows = 0;         // largest instance: the shared-memory plane's rows
};

// A batch class packed for the on-chip batch kernel (k_batch_res.cu), 16-bit or
// FP32 state: whole
// instances in bins, a bin's rows by decreasing degree ("slots") in slices of
// 32 (as DevSell); the bins listed by kind -- clusters of 1, 2 and 4 CTAs, and
// of 4 for bins past 16,383 rows -- each largest first.
struct DevBres {
    bool tried = false;          // planned (rows is null when the class does not fit)
    bool placed = false;         // entries placed by bank
    int64_t steps = 0;           // steps of its solves so far
    int32_t *bins = nullptr, *slot0 = nullptr, *slice0 = nullptr, *rows = nullptr, *off = nullptr;
    void *col = nullptr;         // [blocks][32] of four entries (batch_res_entry)
    void *cb = nullptr;          // per slot: dt * xi0, -degree
    int32_t *perm = nullptr;     // slot -> class row
    int32_t bin0[4] = {}, nbins[4] = {};
    std::vector<int32_t> hinst, hdeg;   // per slot: instance, degree
    double dt = -1;              // dt of the uploaded cb
};

// A batch class packed for the resident batch kernel (k_resident_batch.cu):
// whole instances in bins, rows of a bin by decreasing degree ("slots"), the
// matrix relabelled into slot order.
struct DevRb {
    int32_t *rowptr = nullptr;   // [slots + 1]
    uint32_t *colw = nullptr;    // columns as slots, bit 31 the weight sign
    float *valf = nullptr;
    float *c0 = nullptr;         // dt * xi0 per slot
    int32_t *perm = nullptr;     // slot -> row
    int32_t *bin_off = nullptr;  // [nbins + 1]
    int32_t *cta_bin = nullptr;  // bins, largest first
    int32_t nbins = 0;
    int64_t max_bin_rows = 0;
    bool unit = false;
    double dt = -1;              // dt of the uploaded c0
};

// ---- launchers (k_*.cu) ----

// glibc rand() on the device (k_init.cu).
void rand_seed_window(uint32_t seed, uint32_t *V0);
// out[b] = M^(L * 2^b), b < nbits (31x31 each): independent of the seed.
void rand_jump_matrices(int64_t L, int nbits, std::vector<uint32_t> &out);
// Each init thread emits rand_round() << shift outputs; the shift for a run of
// `outputs` outputs in all.
int64_t rand_round();
int rand_chunk_shift(int64_t outputs);
// mats: the jump matrices of rand_round() outputs.  slot: null, or (batched
// MaxCut) the state row of each instance row.
cudaError_t launch_rand_init(int prec, void *x, void *y, int32_t Ap, bool tsp, int shift, const uint32_t *mats,
                             const RandInst *inst, int count, int64_t total_threads, const int32_t *slot,
                             cudaStream_t s);

// Streaming MaxCut kernels (k_stream.cu).
cudaError_t launch_prestep(const SolveDims &d, const DevCsr &J, Work &w, cudaStream_t s,
                           int *launches);
// evs (optional): 2*period events recorded around each step kernel.
cudaError_t launch_chunk(const SolveDims &d, const DevCsr &J, Work &w, cudaStream_t s,
                         int *launches, cudaEvent_t *evs = nullptr);
cudaError_t launch_cut(const SolveDims &d, const DevCsr &J, Work &w, const uint32_t *plane,
                       cudaStream_t s, int *launches);
// Rows of w.cutrow that launch_cut needs (0 for integer weights).
int64_t cut_scratch_rows(const SolveDims &d, const DevCsr &J);
// count plain (non-window) steps of the solve's kind at step 0: the
// autotuner's timing runs.
cudaError_t launch_plain_steps(const SolveDims &d, const DevCsr &J, Work &w, int count, cudaStream_t s);
// Traced solves: stamp the loop start on the device clock.
cudaError_t launch_trace_start(Work &w, cudaStream_t s);
// The statistics of src/ising.cu:238-265 on the device (k_stats): out[7] =
// min, max, total and mean (agent order), sum of squared deviations (agent
// order), agents at the maximum, first agent at the maximum.
cudaError_t launch_stats(const double *v, int32_t A, double *out, cudaStream_t s);
// Batched: cut[agent_off[i] + a] from instance i's exact sums, and out[7 i..]
// its statistics.
cudaError_t launch_stats_batch(const unsigned long long *eacc, int32_t Ap, const int32_t *agents,
                               const int32_t *agent_off, const double *wsum, int32_t ninst, double *cut,
                               double *out, cudaStream_t s);
// Integer weights, block-diagonal J: eacc[instance][Ap] += s_r sum_j J_rj s_j.
cudaError_t launch_cut_batch(const SolveDims &d, const DevCsr &J, const uint32_t *plane,
                             unsigned long long *eacc, cudaStream_t s);

// Batched step with shared-memory sign planes (k_batch_smem.cu): bytes of
// dynamic shared memory for the largest instance; one launch of a fused or
// force + clamp step (kind K_FUSED / K_FC of k_step.cuh).
size_t bsm_smem_bytes(int64_t max_rows, int W);
struct StepP;
cudaError_t launch_batch_smem(const SolveDims &d, const DevBsm &M, const StepP &P, int kind, bool win,
                              int offset, cudaStream_t s);

// Resident MaxCut kernel (k_resident.cu): returns cudaErrorInvalidValue when the
// shape does not fit.
int resident_pick_ka(const SolveDims &d, const DevCsr &J, int requested);
size_t resident_smem_bytes(const SolveDims &d, int ka);
cudaError_t launch_resident(const SolveDims &d, const DevCsr &J, Work &w, int ka,
                            int32_t step0, int32_t nsteps, bool first, cudaStream_t s);
// Resident batch kernel (k_resident_batch.cu): bins hold at most this many
// rows; one launch runs d.steps_run fused steps of every instance.
int64_t resident_batch_max_rows();
cudaError_t launch_resident_batch(const SolveDims &d, const DevRb &B, Work &w, cudaStream_t s);

// Resident FP64 kernel for small graphs, +-1 weights (k_resident_f64.cu), one
// agent per CTA: whether it is the faster one, and nsteps steps of it.
bool resident64_pick(const SolveDims &d, const DevCsr &J);
cudaError_t launch_resident64(const SolveDims &d, const DevCsr &J, Work &w, int32_t step0, int32_t nsteps, bool first,
                              cudaStream_t s);

// On-chip batch kernel (k_batch_res.cu), kinds 0..3 of bins (DevBres): the
// CTAs of a bin's cluster, its most rows, the entry of a neighbour.  The
// launch runs all d.steps_run fused steps of every bin, the kinds on the side
// streams between fork and join.  agents: the class's largest count.
int batch_res_ctas(int kind);
int64_t batch_res_rows(int kind, bool f32);
uint32_t batch_res_entry(int kind, bool f32, bool allpos, uint32_t slot, bool neg);
cudaError_t launch_batch_res(const SolveDims &d, const DevBres &B, bool allpos, int32_t agents, Work &w,
                             cudaStream_t s, cudaStream_t *side, cudaEvent_t fork, cudaEvent_t *join,
                             int *launches);

// Tensor-memory + shared-memory resident kernel (k_resident_rs.cu), fused
// steps: its agents per CTA (8 of 16-bit state, 4 of FP32) when it is to run.
int resident_rs_pick(const SolveDims &d, const DevCsr &J, bool forced, bool tile);
// coop: the update-window mode's windows in one co-resident launch (a
// bounded barrier per window); cudaErrorCooperativeLaunchTooLarge when the
// CTAs cannot all be resident.
cudaError_t launch_resident_rs(const SolveDims &d, const DevCsr &J, Work &w, int ka, int32_t step0,
                               int32_t nsteps, bool first, bool coop, cudaStream_t s);

// TSP kernels (k_tsp.cu).
struct DevTsp {
    int32_t N = 0;
    double A = 1, B = 0, C = 0;
    std::vector<double> packed, rowsum, I2h;   // host
    float *D = nullptr;                   // device N x N distances (float)
    float *I2 = nullptr;                  // device per-city linear field (float)
    double *I2d = nullptr;                // the same in FP64
    double *Dd = nullptr;                 // device N x N distances (FP64, exact)
    DevCsr qubo;                          // the QUBO as CSR (streaming path)
};
int tsp_pick_ka(const SolveDims &d, const DevTsp &t, int requested);
cudaError_t launch_tsp_resident(const SolveDims &d, const DevTsp &t, Work &w, int ka,
                                cudaStream_t s);
cudaError_t launch_tsp_stream(const SolveDims &d, const DevTsp &t, Work &w, cudaStream_t s,
                              int *launches);
// Resident TSP kernel with the distance product on the tensor cores
// (k_tsp_tc.cu): 16-bit state, 3 <= N <= 32, 8 agents per CTA.
bool tsp_tensor_fits(const SolveDims &d, const DevTsp &t);
constexpr int kTspTensorAgents = 8;
// threads_per_row: 1, 2 or 4 threads share a (position, agent) row's
// cities; 0 picks the default.
int tsp_tensor_threads_per_row(int requested);
cudaError_t launch_tsp_tensor(const SolveDims &d, const DevTsp &t, Work &w, int threads_per_row, cudaStream_t s);
// TSP setup on the device from city coordinates (device xc, yc): packed
// distances (src/kernels.cu:404-442), the tables t.D / t.Dd, the largest
// distance *mx, per-city sums (src/tsp_gpu.cu:51-68) and the linear field
// t.I2d / t.I2 with B = C = scale * max distance.
cudaError_t launch_tsp_setup(const double *xc, const double *yc, int32_t N, int32_t kind, double A, double scale,
                             double *packed, double *mx, double *rowsum, DevTsp &t, cudaStream_t s);
// Tour length of every agent holding a valid tour (NaN otherwise) into len[A].
cudaError_t launch_tsp_lengths(const DevTsp &t, const int32_t *tours, const int32_t *valid, int32_t A,
                               double *len, cudaStream_t s);

}  // namespace sbx
