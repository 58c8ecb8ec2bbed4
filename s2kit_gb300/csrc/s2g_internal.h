// s2g_internal.h -- internal (non-exported) declarations of the GB300 seminaive SHT library.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <initializer_list>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/s2kit_gb300.h"

namespace s2g {

// Records a formatted message for s2g_last_error() and returns `code`.
int fail(int code, const char* fmt, ...);
// cudaError_t -> status (records the CUDA error string)
int cuda_fail(cudaError_t e, const char* what);

#define S2G_CUDA(call)                                           \
    do {                                                         \
        cudaError_t e_ = (call);                                 \
        if (e_ != cudaSuccess) return ::s2g::cuda_fail(e_, #call); \
    } while (0)

#define S2G_TRY(call)            \
    do {                         \
        int r_ = (call);         \
        if (r_ != S2G_OK) return r_; \
    } while (0)

// Kernel launch accounting: every launch is counted; when profiling is enabled
// (s2g_prof_enable) it is also bracketed by CUDA events on its own stream.
void prof_begin(const char* name, cudaStream_t st);
void prof_end(cudaStream_t st);

// Graph capture on this thread: launches counted into the graph (see launches_add for replays).
void capture_count_begin();
unsigned long long capture_count_end();
void launches_add(unsigned long long n);

struct ProfScope {
    cudaStream_t st;
    ProfScope(const char* name, cudaStream_t s) : st(s) { prof_begin(name, s); }
    ~ProfScope() { prof_end(st); }
};

// Allows kernel fn `bytes` of dynamic shared memory on the current device.  The allowance is the function's, shared by
// all threads, and a launch that asks for more than it fails: it only ever grows.
int set_smem(const void* fn, size_t bytes);

// Device tables and constants for one (bandwidth, cutoff) on one device.
struct Tables {
    int bw = 0, cutoff = 0, device = -1;
    int64_t total = 0;          // doubles in each of fwd / inv
    double* fwd = nullptr;      // reference layout: SemiNaive_Naive_Pml_Table (cospml.c:451-475)
    double* inv = nullptr;      // Transpose_SemiNaive_Naive_Pml_Table layout (cospml.c:490-518)
    int64_t* off = nullptr;     // bw offsets (device)
    int64_t* h_off = nullptr;   // same, host copy
    double* weights = nullptr;  // 4*bw (weights.c:32-47)
    double* sinv = nullptr;     // sin(theta_j), 2*bw
    double2* tw_S = nullptr;    // exp(2 pi i k / 2bw), k < 2bw   (cos, sin)
    double2* tw_D = nullptr;    // exp(i pi k / (2 * 2bw)), k < 2bw (DCT pre/post twiddle)
    // split-precision (tensor core) operands, built on first use
    void* split = nullptr;
    // digit tables of the tensor-core FP64 path (digit_gemm.cu), built on first use
    void* dg = nullptr;
    int dg_skip = 0;            // they did not fit in device memory: calls left before the next attempt
    void* dg32 = nullptr;       // the same for FP32 transforms
    int dg32_skip = 0;
    int refs = 0;               // references (cache, plans, groups, calls in flight); under the cache lock
};

// Whether st is being captured (or, for the legacy stream, another one).
bool capturing(cudaStream_t st);

// While it lives, this thread may allocate although another captures a graph in the global mode, whose capture the
// allocation would otherwise end (and the call fail).  Not for a stream that is itself captured.
struct RelaxCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// Device scratch owned by a plan; grown on demand.  A buffer handed to a captured call lives as long as the plan:
// the graph has its address, and calls of other kinds at the same batch may need more of it.
struct Scratch {
    void* ptr = nullptr;
    size_t bytes = 0;
    size_t nofit = 0;          // dg_scratch: what did not fit, and the calls left before the next attempt
    int skip = 0;
    bool held = false;         // a captured call has it
    std::vector<void*> kept;   // outgrown buffers that captured calls have
    int ensure(size_t need, cudaStream_t st);  // st: the stream of the call that it is for
    void release();
};

// The FP32 transforms move samples and coefficients as float4 and through TMA, so their device
// pointers must be 16-byte aligned (every cudaMalloc pointer is); others are rejected up front.
inline int check_aligned16(std::initializer_list<const void*> ps) {
    for (const void* q : ps)
        if ((uintptr_t)q & 15) return fail(S2G_ERR_ARG, "device pointer %p is not 16-byte aligned", q);
    return S2G_OK;
}

inline bool overlap(const void* a, size_t na, const void* b, size_t nb) {
    return (uintptr_t)a < (uintptr_t)b + nb && (uintptr_t)b < (uintptr_t)a + na;
}

// Build / fetch device tables (cached per device, bw, cutoff); the caller gets a reference and
// returns it with put_tables.  cutoff 0 gives the weights, nodes and twiddles of bw without any
// Legendre table (fwd, inv and off null), for the on-the-fly family.
int get_tables(int bw, int cutoff, Tables** out);
void put_tables(Tables* t);
struct TabRef {
    Tables* t;
    ~TabRef() { put_tables(t); }
};
// Build tables into caller-visible device buffers (used by the host table builders).
// Allocates and fills t's device tables; with h_fwd/h_inv (host copies of total doubles each,
// e.g. read from a table file) the Legendre tables are uploaded instead of generated.
int build_tables(Tables* t, cudaStream_t st, const double* h_fwd = nullptr, const double* h_inv = nullptr);
int generate_weights_device(int bw, double* d_weights, cudaStream_t st);
int generate_cos_pml_device(int bw, int m_begin, int m_end, double* d_fwd, const int64_t* d_off,
                            cudaStream_t st);
int transpose_cos_pml_device(int bw, int m_begin, int m_end, const double* d_fwd, double* d_inv,
                             const int64_t* d_off, cudaStream_t st);
int generate_pml_device(int bw, int m_begin, int m_end, double* d_fwd, const int64_t* d_off, cudaStream_t st);
int pmm_device(int m, const double* d_eval, int n, double* d_out, cudaStream_t st);
int nodes_device(int n, double* d_out, int acos_only, cudaStream_t st);

// ---- FP64 pipeline (sht_fp64.cu) ----
struct F64Work {
    double* Xr;  // [batch][rows][2bw]
    double* Xi;
    int rows;    // rows per function in X (bw for REAL, 2bw for COMPLEX)
};
size_t f64_work_bytes(int bw, int batch, int data_format);
// ---- FP64 transforms as exact digit products on the tensor cores (digit_gemm.cu) ----
// Their kernels' waits are bounded; `err` is the word of the plan, group or call that gets S2G_ERR_TIMEOUT
// where one expired (device memory, or the host's where host_direct).  The functions further down that may take
// this path take the word as `dg`: with it they run there, on tables and scratch that the caller has readied
// (dg_prepare, dg_scratch); null keeps them off it.
bool dg_takes(int bw);
int dg_chunk(int bw, int batch, int es);  // functions transformed at a time, es: 8 for FP64, 4
size_t dg_work_bytes(int bw, int batch, bool two);  // two: the data have imaginary parts
// Grows s to `need` bytes for the digit path; *yes false where that does not fit, or cannot be done under capture (as
// dg_prepare for the tables), and the caller takes the other kernels, whose scratch may fit or be there.
int dg_scratch(Scratch& s, size_t need, cudaStream_t st, bool* yes);
bool dg_no_scratch();  // the test hook's
// FP32 samples and coefficients (igrid null: real fields); readied by dg32_prepare into t->dg32.
// gmap, cmap: per-function grid and coefficient offsets (real fields), null for functions back to back.
bool dg32_takes(int bw);
size_t dg32_work_bytes(int bw, int batch, bool two);
int dg32_prepare(Tables* t, cudaStream_t st, bool* yes);
int fst_dg32(const Tables* t, const float* rgrid, const float* igrid, float* rc, float* ic, int batch, void* work,
             cudaStream_t st, int* err, const int64_t* gmap = nullptr, const int64_t* cmap = nullptr);
int inv_fst_dg32(const Tables* t, const float* rc, const float* ic, float* rgrid, float* igrid, int batch, void* work,
                 cudaStream_t st, int* err, const int64_t* gmap = nullptr, const int64_t* cmap = nullptr);
// On-the-fly family (tables of cutoff 0): real fields for which it pays, and the scratch, once prepared or at any time.
bool dg_fly_takes(int bw, int fields);
size_t dg_fly_bytes(const Tables* t, int batch, bool two);
size_t dg_fly_bytes(int bw, int batch, bool two);
int dg_prepare(Tables* t, cudaStream_t st, bool* yes);
void dg_put(void* dg);
int dg_status(int* err);    // reads the (device) word and clears it
int dg_expired(int code);  // records the failure
int fst_f64_dg(const Tables* t, const double* rdata, const double* idata, double* rc, double* ic, int batch,
               int data_format, void* work, cudaStream_t st, int* err);
int inv_fst_f64_dg(const Tables* t, const double* rc, const double* ic, double* rdata, double* idata, int batch,
                   int data_format, void* work, cudaStream_t st, int* err);
int fst_f64(const Tables* t, const double* rdata, const double* idata, double* rc, double* ic, int batch,
            int data_format, int cutoff, void* work, cudaStream_t st, int* dg = nullptr);
// fst_f64 with the DFT geometry of length 2bw (Bluestein tables included when 2bw is not a
// power of two) supplied by the caller instead of looked up in the per-device length cache,
// which builds missing tables with cudaMalloc.  Null `len_S` behaves like fst_f64.
struct Len;
int fst_f64_len(const Tables* t, const Len* len_S, const double* rdata, const double* idata, double* rc,
                double* ic, int batch, int data_format, int cutoff, void* work, cudaStream_t st);
int inv_fst_f64(const Tables* t, const double* rc, const double* ic, double* rdata, double* idata, int batch,
                int data_format, int cutoff, void* work, cudaStream_t st, int* dg = nullptr);
// On-the-fly family (FST_semi_fly.c): the Legendre functions are generated inside the
// contraction kernels, so `t` needs only its weights and twiddles (tables of cutoff 0, see
// get_tables); work as f64_work_bytes.
int fst_f64_fly(const Tables* t, const double* rdata, const double* idata, double* rc, double* ic, int batch,
                int data_format, void* work, cudaStream_t st);
int inv_fst_f64_fly(const Tables* t, const double* rc, const double* ic, double* rdata, double* idata, int batch,
                    int data_format, void* work, cudaStream_t st);
int fzt_f64_fly(const Tables* t, const double* rdata, const double* idata, double* rres, double* ires, int batch,
                int data_format, void* work, cudaStream_t st);
int fzt_f64(const Tables* t, const double* rdata, const double* idata, double* rres, double* ires, int batch,
            int data_format, void* work, cudaStream_t st);
int transmult_f64(const double* rd, const double* id, const double* rf, const double* iff, double* rr,
                  double* ir, int bw, int batch, cudaStream_t st);
// 1-D transforms with caller-provided (device) tables for a single order m
int dlt_semi_f64(const double* data, int bw, int m, double* result, const double* table, const double* weights,
                 const double2* tw_S, const double2* tw_D, cudaStream_t st);
int inv_dlt_semi_f64(const double* coeffs, int bw, int m, double* result, const double* ttable,
                     const double* sinv, const double2* tw_S, const double2* tw_D, cudaStream_t st);
int dlt_naive_f64(const double* data, int bw, int m, const double* weights, double* result, const double* ptable,
                  cudaStream_t st);
int inv_dlt_naive_f64(const double* coeffs, int bw, int m, double* result, const double* ptable,
                      cudaStream_t st);
int twiddles_device(int n, double2* d_tw_full, double2* d_tw_quarter, cudaStream_t st);

// ---- split-precision pipeline (sht_split.cu, czt_split.cu) ----
// Orders the split path computes with the naive transform: odd m below 32.  For these the cosine
// series of G = P/sin(theta) has large coefficients, and FP32 rounding of the DCT output is
// amplified by them (the reference's seminaive/naive hybrid, FST_semi_memo.c:96-120, makes the
// same trade at the other end of the order range).
constexpr int kSplitNaiveOddBelow = 32;
__host__ __device__ __forceinline__ bool split_naive_order(int m) { return (m & 1) && m < kSplitNaiveOddBelow; }
// Layout of the split path's intermediate arrays at bandwidth bw, per plane (re, im), function
// and order m < bw: X and F rows of SX floats (latitudes theta < 2bw; a naive order's folded
// halves at t BN, t = 0, 1), C and Fc rows of 2 BH floats (cosine frequency k = 2j + t at t BH + j).
// bw itself (BH = bw/2, BN = bw, SX = 2bw) where the warp FFTs take length 2bw; at the chirp-z
// bandwidths BN and BH are rounded up to multiples of 8, the padding held at zero.
struct SplitLayout {
    int BH, BN, SX;
};
SplitLayout split_layout(int bw);
// True where the split path's length-2bw DFTs run as chirp-z transforms (czt_split.cu): bw in
// [17, 256] and 2bw not a warp-FFT length.
bool split_czt(int bw);
// Length M of the chirp-z convolution at bandwidth bw, from 33 on (below, small_takes): the power of two >= 4 bw - 1.
int czt_len(int bw);
// Device tables of one chirp-z bandwidth (the first three from czt_build_tables, the rest the
// split path's FP32 weights, sin(theta) and DCT twiddles).
struct CztTabs {
    int B, M;
    const float2* h;     // exp(-i pi (n^2 mod 2S) / S), n < S = 2B
    const float2* K;     // DFT_M of b_j = conj(h_|j|) (|j| < S, j mod M), divided by M
    const float2* twM;   // exp(2 pi i k / M), k < M
    const float* w32;    // quadrature weights, 2S (even orders, then odd)
    const float* sin32;  // sin(theta_j), S
    const float2* twD;   // (cos, sin)(pi k / 2S), k < S
};
int czt_build_tables(int bw, float2** d_h, float2** d_K, float2** d_tw);
// One FFT stage (which: 0 rows forward, 1 weighted DCT-II, 2 DCT-III, 3 rows inverse) of N
// functions at a chirp-z bandwidth; in/out, scale and gmap as the warp-FFT stages.
int czt_stage(int which, const CztTabs& g, const void* in, void* out, int N, float scale, const int64_t* gmap,
              cudaStream_t st);
size_t split_work_bytes(int bw, int batch);  // off the digit path
int fst_split(Tables* t, const float* grid, float* rc, float* ic, int batch, int precision, void* work,
              cudaStream_t st, int* dg);
int inv_fst_split(Tables* t, const float* rc, const float* ic, float* grid, int batch, int precision, void* work,
                  cudaStream_t st, int* dg);
// COMPLEX data as two real fields (cwork: split_complex_bytes of scratch besides work, off the digit path).
size_t split_complex_bytes(int bw, int batch);
int fst_split_complex(Tables* t, const float* rgrid, const float* igrid, float* rc, float* ic, int batch,
                      int precision, void* work, void* cwork, cudaStream_t st, int* dg);
int inv_fst_split_complex(Tables* t, const float* rc, const float* ic, float* rgrid, float* igrid, int batch,
                          int precision, void* work, void* cwork, cudaStream_t st, int* dg);
// One FFT stage of several bandwidth classes (split path, power-of-two bw <= 512) in ONE launch:
// which 0 rows forward (grid -> X), 1 weighted DCT-II (X -> C), 2 DCT-III (Fc -> F), 3 rows
// inverse (F -> grid); in/out as the per-class kernels, gmap per-function grid offsets for the
// rows stages.  dct_ctas_per_sm bounds the resident blocks the DCT stages are sized for (0: as
// many as fit).
struct StageSpec {
    Tables* t;
    int N;
    const void* in;
    void* out;
    const int64_t* gmap;
    float *rc = nullptr, *ic = nullptr;  // rows stages, bw < 32 (small_takes): the whole transform, to or from these
    const int64_t* cmap = nullptr;       // (their coefficient offsets); out, in are then the grid or unused
};
int split_stage_group(int which, const StageSpec* spec, int ncls, int dct_ctas_per_sm, cudaStream_t st);
// The same stage for one class of any split-path bandwidth, as its own launch.
int split_stage_one(int which, Tables* t, int N, const void* in, void* out, const int64_t* gmap, cudaStream_t st);
// Bandwidths transformed whole by one kernel (small32.cuh), and those transforms: real fields, functions back to
// back or at the offsets gmap (samples) and cmap (coefficients).
bool small_takes(int bw);
int fst_small(Tables* t, const float* grid, float* rc, float* ic, int N, cudaStream_t st, const int64_t* gmap = nullptr,
              const int64_t* cmap = nullptr);
int inv_fst_small(Tables* t, const float* rc, const float* ic, float* grid, int N, cudaStream_t st,
                  const int64_t* gmap = nullptr, const int64_t* cmap = nullptr);
// Reads (and optionally clears) the device error word of the tensor-core kernels.
int split_device_status(Tables* t, int clear);

// One bandwidth class of a (grouped) tensor-core contraction launch.  Intermediate arrays are
// class-contiguous: X/F [2][N][B][SX], C/Fc [2][N][B][2 BH] floats (split_layout(B)).
struct LegSpec {
    Tables* t;
    int N;                    // functions of this class
    int NB;                   // table rows per work item (0: the largest the class needs)
    const float* C;           // forward: DCT output
    const float* X;           // forward: phi-DFT output (naive orders)
    const float* rc_in;       // inverse: input coefficients
    const float* ic_in;
    float* rc;                // forward: output coefficients
    float* ic;
    float* Fc;                // inverse: cosine-series output
    float* F;                 // inverse: naive-order output
    const int64_t* cmap;      // function -> coefficient offset (null: f * B * B)
};
// One persistent launch over every class; counter: one device int (zeroed on `st` here);
// table_stages: depth of the kernel's table-copy ring, 0 = as many stages as fit.
int split_leg(bool fwd, int precision, const LegSpec* cls, int ncls, int* counter, int table_stages,
              cudaStream_t st);
// Packs the tensor-core operands of `t` for `precision` now (they are otherwise packed on first use).
int split_prepare(Tables* t, int precision);
int split_fwd_head(Tables* t, const float* grid, float* X, float* C, int batch, const int64_t* gmap,
                   cudaStream_t st);
int split_inv_tail(Tables* t, float* F, float* Fc, float* grid, int batch, const int64_t* gmap, cudaStream_t st);

// What the split path would refuse (bandwidth, cutoff, precision).
int split_check(const Tables* t, int precision);

// ---- split transforms with one FP64-residual refinement step (refine.cu) ----
size_t refine_io_bytes(int bw, int batch);
size_t refine_work_bytes(int bw, int batch);
int fst_refined(Tables* t, const double* grid, double* rc, double* ic, int batch, int precision, void* io,
                void* work, cudaStream_t st);
int inv_fst_refined(Tables* t, const double* rc, const double* ic, double* grid, int batch, int precision, void* io,
                    void* work, cudaStream_t st);

}  // namespace s2g
