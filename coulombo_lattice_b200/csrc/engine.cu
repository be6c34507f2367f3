// Context, orchestration and the GPU half of the C ABI (include/coulombo_lattice.h).
#include <algorithm>
#include <array>
#include <memory>
#include <map>
#include <mutex>
#include <tuple>
#include <cmath>
#include <cstdlib>
#include <cstdio>
#include <cstring>
#include <numeric>
#include <string>
#include <thread>
#include <vector>

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include "coulombo_lattice.h"
#include "host/host_logic.hpp"
#include "host/status.hpp"
#include "kernels.cuh"
#include "pair_mma.cuh"
#include "passes.hpp"
#include "gram_dmma.cuh"
#include "gram_tc.cuh"
#include "sublattice.cuh"
#include "zmix_wht.cuh"

using clk::cx;
using clk::FftPlan;

namespace {

// ---------------------------------------------------------------------------------------
// CUDA helpers
// ---------------------------------------------------------------------------------------
#define CL_CUDA(call)                                                                           \
    do {                                                                                        \
        cudaError_t err_ = (call);                                                              \
        if (err_ != cudaSuccess)                                                                \
            cl::fail(err_ == cudaErrorMemoryAllocation ? CL_ERR_MEMORY : CL_ERR_CUDA,           \
                     "CUDA error %s at %s:%d: %s", cudaGetErrorName(err_), __FILE__, __LINE__,  \
                     cudaGetErrorString(err_));                                                 \
    } while (0)

#define CL_LAUNCHED() CL_CUDA(cudaGetLastError())

template <typename T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    unsigned moves = 0;  // how often the storage changed
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
    void alloc(size_t count) {
        if (count == n && p) return;
        release();
        ++moves;
        if (count == 0) return;
        CL_CUDA(cudaMalloc(&p, count * sizeof(T)));
        n = count;
    }
    void upload(const T* host, size_t count, cudaStream_t s) {
        alloc(count);
        if (count) CL_CUDA(cudaMemcpyAsync(p, host, count * sizeof(T), cudaMemcpyHostToDevice, s));
    }
};

int device_count() {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

void require_gpu() {
    if (device_count() == 0) cl::fail(CL_ERR_CUDA, "no CUDA device is available");
}

int grid_for(long long n, int threads = 256) {
    long long b = (n + threads - 1) / threads;
    return (int)std::max(1LL, std::min(b, 148LL * 32));
}

// ---------------------------------------------------------------------------------------
// FFT plans and host-built tables
// ---------------------------------------------------------------------------------------
bool smooth235(int n) {
    if (n < 1) return false;
    for (int p : {2, 3, 5})
        while (n % p == 0) n /= p;
    return n == 1;
}

FftPlan make_plan(int n) {
    FftPlan p{};
    p.n = n;
    int m = n;
    auto push = [&](int r) {
        if (p.nst >= 16) cl::fail(CL_ERR_UNSUPPORTED, "FFT length %d needs too many stages", n);
        p.radix[p.nst++] = r;
        m /= r;
    };
    // fewest shared-memory round trips: radix 16 first, then 8/4, a lone 2 joined with a
    // 3 (-> 6) or 5 (-> 10), a lone 4 with a 3 (-> 12), then 3s and 5s
    int twos = 0, threes = 0, fives = 0;
    for (; m % 2 == 0; m /= 2) ++twos;
    for (; m % 3 == 0; m /= 3) ++threes;
    for (; m % 5 == 0; m /= 5) ++fives;
    if (m != 1) cl::fail(CL_ERR_UNSUPPORTED, "FFT length %d is not a product of 2, 3 and 5", n);
    m = n;
    while (twos >= 4) { push(16); twos -= 4; }
    if (twos == 3) { push(8); twos = 0; }
    if (twos == 2) {
        if (threes > 0) { push(12); --threes; } else push(4);
        twos = 0;
    }
    if (twos == 1) {
        if (threes > 0) { push(6); --threes; }
        else if (fives > 0) { push(10); --fives; }
        else push(2);
        twos = 0;
    }
    while (threes-- > 0) push(3);
    while (fives-- > 0) push(5);
    int ns = 1;
    for (int s = 0; s < p.nst; ++s) {
        p.ns_magic[s] = clk::fdiv_magic(ns);
        ns *= p.radix[s];
    }
    return p;
}

// tw[t] = exp(-2 pi i t / n), built in extended precision and rounded once.
std::vector<cx<double>> twiddles64(int n) {
    std::vector<cx<double>> t(n);
    const long double pi = 3.141592653589793238462643383279502884L;
    for (int i = 0; i < n; ++i) {
        long double ang = -2.0L * pi * (long double)i / (long double)n;
        t[i].re = (double)std::cos(ang);
        t[i].im = (double)std::sin(ang);
    }
    return t;
}

// phase(i) = exp(i pi i / n) (CoulombCalculator.cpp:45-54).
std::vector<cx<double>> phases64(int n) {
    std::vector<cx<double>> t(n);
    const long double pi = 3.141592653589793238462643383279502884L;
    for (int i = 0; i < n; ++i) {
        long double ang = pi * (long double)i / (long double)n;
        t[i].re = (double)std::cos(ang);
        t[i].im = (double)std::sin(ang);
    }
    return t;
}

// Thomas-Fermi-Resta radius (Interaction.cpp:18-32, same Newton iteration and stop rule).
void thomas_fermi(double dielectric, double lattice, double* r_tf, double* q_tf) {
    const double eps = 1.0e-12;
    const double q = 2.0 / std::sqrt(M_PI) * std::cbrt(96.0 * M_PI * M_PI) / lattice;
    double x = std::sqrt(6.0 * (dielectric - 1.0)), dx;
    int guard = 0;
    do {
        double F = std::sinh(x) - dielectric * x;
        double dF = std::cosh(x) - dielectric;
        dx = (std::fabs(F) < eps) ? 0 : F / dF;
        x -= dx;
        if (++guard > 10000) cl::fail(CL_ERR_ARGUMENT, "Thomas-Fermi radius did not converge");
    } while (dx / q > eps);
    *q_tf = q;
    *r_tf = x / q;
}

struct Axis {
    FftPlan plan;
    DevBuf<cx<double>> tw64;
    DevBuf<cx<float>> tw32;
    DevBuf<cx<double>> phase;
};

// Per-launch geometry of the x passes and the y/z passes.
struct XTile {
    int rows, ld;
    size_t smem;
};
struct LTile {
    int W;
    size_t smem;
};

template <typename T>
XTile x_tile(int nx, int nrows) {
    const int elems = sizeof(T) == 4 ? 4096 : 2048;
    int rows = std::max(1, std::min(elems / std::max(nx, 1), 64));
    rows = std::min(rows, nrows);
    int ld = (rows % 2 == 0) ? rows + 1 : rows;
    XTile t{rows, ld, sizeof(cx<T>) * ((size_t)nx + 2ull * nx * ld)};
    return t;
}

template <typename T>
LTile l_tile(int n, bool with_khat) {
    int W = sizeof(T) == 4 ? 16 : 8;
    auto bytes = [&](int w) {
        return sizeof(cx<T>) * ((size_t)n + 2ull * n * w) + (with_khat ? sizeof(T) * (size_t)n * w : 0);
    };
    while (W > 1 && bytes(W) > 200 * 1024) W /= 2;
    return LTile{W, bytes(W)};
}

unsigned zgroups(long long zblocks, int cnt) { return clp::density_groups(zblocks, cnt); }

// Bytes of grids a chunk may hold so that consecutive passes meet in L2 (CL_L2_CHUNK_MB;
// off by default: measured on B200 it gave no gain at 96^3 over whole-request chunks).
size_t l2_chunk_bytes() {
    const char* e = std::getenv("CL_L2_CHUNK_MB");
    double mb = e ? std::atof(e) : 0.0;
    return (size_t)(std::max(0.0, mb) * 1024 * 1024);
}

// Allows launches of `kernel` with `bytes` of dynamic shared memory.  The limit is one per kernel, whatever the
// thread or context: all set the same, the most that fits beside the kernel's static shared memory, so that none lowers
// it between another's call and launch.
template <typename K>
void ensure_smem(K kernel, size_t bytes, size_t most = 227 * 1024) {
    if (bytes > most) cl::fail(CL_ERR_UNSUPPORTED, "tile needs %zu bytes of shared memory", bytes);
    CL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
}

}  // namespace

// ---------------------------------------------------------------------------------------
// The context
// ---------------------------------------------------------------------------------------
// State of the sub-lattice decomposition (sublattice.cuh) for the loaded structure.
struct Sublattice {
    bool active = false;  // the request paths use the decomposition (a sub-lattice mode whose structure qualifies)
    bool zb = false;      // the classes are the zinc-blende set: compiled mixing table, canonical class order
    int m = 0, S = 0;
    int off[clk::kSlMaxClasses][3] = {};  // offset (x, y, z) of each class, in the order used on the GPU
    int sub[3] = {0, 0, 0};               // sub-grid points per axis, n/m
    int pad[3] = {0, 0, 0};               // transform length per axis, 2n/m
    int vn[3] = {0, 0, 0};                // virtual grid of the x and y passes: (pad x, pad y, S * sub z)
    long long vM = 0;
    clk::SlTable table;
    Axis ax[3];                           // plans and twiddles of the transform lengths
    DevBuf<cx<double>> H64, phxy64, phz64;
    DevBuf<cx<float>> H32, phxy32, phz32;
    // zinc-blende or two classes: the tables of the z pass that mixes in registers (zmix_wht.cuh)
    bool zw = false;
    DevBuf<unsigned char> zw_tab, zw_col, zw_zph;  // of the form's precision
    long long tables_version = -1;        // kernel version the tables were built from
};

struct PairSetup;

struct cl_ctx {
    int device = 0;
    int mode = CL_MODE_FP64_PLAIN;
    Sublattice sl;
    long long kernel_version = 0;  // bumped at every kernel build
    // grid the register passes run on (the real grid, or the sub-lattice virtual grid), the key
    // of the autotuner's choices
    int tune_dims[3] = {0, 0, 0};
    int tune_form = 0;  // 2 on the virtual grid
    int n[3] = {0, 0, 0};
    long long M = 0;
    double step[3] = {1, 1, 1};
    cudaStream_t stream = nullptr;
    cudaEvent_t ev[5] = {};
    Axis ax[3];

    bool kernel_ready = false;
    DevBuf<double> ghat;
    DevBuf<double> khat64;  // the 8 rounds' Khat_kappa, one after another
    DevBuf<float> khat32;

    // grid API ("every cell is an atom")
    DevBuf<int> grid_cell, grid_row_ptr;
    DevBuf<cx<double>> grid_rho, grid_V, grid_rho2;
    DevBuf<cx<float>> grid_rho32;  // the grid density in the FP32 form
    bool grid_prepared = false;

    // states
    long long layout_version = 0;  // bumped when the atoms, the states' number or the orbitals change
    int n_states = 0, n_holes = 0, n_orb = 0;
    long long n_atoms = 0, n_sorted = 0;
    DevBuf<cx<double>> coeff;
    DevBuf<int> cell_sorted, orig_sorted, row_ptr;
    DevBuf<unsigned long long> row_mask;  // sub-lattice forms: the atoms of every row (k_row_masks)
    DevBuf<cx<double>> coeff_stage;  // two states of caller coefficients, input atom order
    long long live_rows = 0;           // rows (y, z) holding at least one atom
    std::vector<int> atom_slot;        // input atom -> sorted (deduplicated) slot
    std::vector<int64_t> cells_seen;   // the cells of the last load (an identical list skips the sort)
    cudaStream_t copy_stream = nullptr;  // coefficient uploads of cl_compute_states
    std::vector<cudaEvent_t> state_ev;   // one per state: its coefficients are on the device

    // work buffers, kept across requests (grown on demand)
    DevBuf<unsigned char> work;
    DevBuf<unsigned char> rounds;  // per-round values at the atoms of a chunk of densities
    DevBuf<cx<double>> req_rho, req_V;
    DevBuf<double> req_o4;
    DevBuf<int> req_rows;
    DevBuf<float> tc_buf;  // TF32 hi/lo operands of the tensor-core Gram
    std::unique_ptr<PairSetup, void (*)(PairSetup*)> eager_pairs{nullptr, nullptr};  // lists of the last eager call
    DevBuf<int> slot_of_atom;      // input atom -> sorted slot (the potentials' gather)
    DevBuf<double> pot;            // potentials in input atom order
    double timings[4] = {0, 0, 0, 0};

    // Changes whenever a buffer that a request's launches name gets other storage.
    unsigned long long buffer_moves() const {
        unsigned long long m = khat64.moves + khat32.moves + coeff.moves + cell_sorted.moves + row_ptr.moves + row_mask.moves;
        m += (unsigned long long)work.moves + rounds.moves + tc_buf.moves;
        m += (unsigned long long)sl.H64.moves + sl.phxy64.moves + sl.phz64.moves + sl.H32.moves + sl.phxy32.moves +
             sl.phz32.moves + sl.zw_tab.moves + sl.zw_col.moves + sl.zw_zph.moves;
        for (const Axis* a : {ax, sl.ax})
            for (int d = 0; d < 3; ++d) m += (unsigned long long)a[d].tw64.moves + a[d].tw32.moves + a[d].phase.moves;
        return m;
    }

    // per-kernel profiling (events recorded around launches on `stream`)
    struct ProfEntry {
        int cls;
        cudaEvent_t a, b;
        double bytes;
    };
    bool profiling = false;
    std::vector<cudaEvent_t> ev_pool;
    size_t ev_used = 0;
    std::vector<ProfEntry> prof_pending;
    // while a batch captures this context with profiling on: event pairs go to the batch
    std::vector<ProfEntry>* prof_sink = nullptr;
    std::vector<cudaEvent_t>* prof_owned = nullptr;
    double prof_ms[CL_NUM_KCLASS] = {};
    double prof_bytes[CL_NUM_KCLASS] = {};
    int64_t prof_launches[CL_NUM_KCLASS] = {};

    ~cl_ctx() {
        if (copy_stream) {
            cudaStreamSynchronize(copy_stream);
            for (auto& e : state_ev) cudaEventDestroy(e);
            cudaStreamDestroy(copy_stream);
        }
        if (stream) {
            cudaStreamSynchronize(stream);
            for (auto& e : ev)
                if (e) cudaEventDestroy(e);
            for (auto& e : ev_pool) cudaEventDestroy(e);
            cudaStreamDestroy(stream);
        }
    }
};

namespace {

// Precision of a form: the all-FP64 forms against the FP32-transform forms.
bool fp64_form(const cl_ctx* c) { return c->mode == CL_MODE_FP64_PLAIN || c->mode == CL_MODE_FP64_SUBLATTICE; }
bool sublattice_mode(const cl_ctx* c) {
    return c->mode == CL_MODE_FP64_SUBLATTICE || c->mode == CL_MODE_FP32_SUBLATTICE;
}

size_t free_device_bytes() {
    size_t fr = 0, tot = 0;
    CL_CUDA(cudaMemGetInfo(&fr, &tot));
    return fr;
}

cudaEvent_t prof_event(cl_ctx* c) {
    if (c->prof_owned) {  // captured into a graph: the event lives as long as the graph
        cudaEvent_t e;
        CL_CUDA(cudaEventCreate(&e));
        c->prof_owned->push_back(e);
        return e;
    }
    if (c->ev_used == c->ev_pool.size()) {
        cudaEvent_t e;
        CL_CUDA(cudaEventCreate(&e));
        c->ev_pool.push_back(e);
    }
    return c->ev_pool[c->ev_used++];
}

// Marks the start of a launch of class `cls`; returns the start event (or nullptr).
// Inside a capture an event must be recorded as an external event-record node, so that
// every replay of the graph records it.
void prof_record(cl_ctx* c, cudaEvent_t e) {
    if (c->prof_owned)
        CL_CUDA(cudaEventRecordWithFlags(e, c->stream, cudaEventRecordExternal));
    else
        CL_CUDA(cudaEventRecord(e, c->stream));
}

cudaEvent_t prof_begin(cl_ctx* c) {
    if (!c->profiling) return nullptr;
    cudaEvent_t a = prof_event(c);
    prof_record(c, a);
    return a;
}

void prof_end(cl_ctx* c, cudaEvent_t a, int cls, double bytes) {
    if (!a) return;
    cudaEvent_t b = prof_event(c);
    prof_record(c, b);
    (c->prof_sink ? *c->prof_sink : c->prof_pending).push_back({cls, a, b, bytes});
}

// After the stream has been synchronised: fold the pending pairs into the totals.
void prof_collect(cl_ctx* c) {
    for (const auto& e : c->prof_pending) {
        float ms = 0;
        CL_CUDA(cudaEventElapsedTime(&ms, e.a, e.b));
        c->prof_ms[e.cls] += ms;
        c->prof_bytes[e.cls] += e.bytes;
        c->prof_launches[e.cls] += 1;
    }
    c->prof_pending.clear();
    c->ev_used = 0;
}

void build_khat(cl_ctx* c) {
    const int nx = c->n[0], ny = c->n[1], nz = c->n[2];
    const double denom = (double)((unsigned long long)c->M * 8ull);
    for (int r = 0; r < 8; ++r) {
        const int kx = r & 1, ky = (r >> 1) & 1, kz = (r >> 2) & 1;
        if (fp64_form(c)) {
            c->khat64.alloc(8 * c->M);
            clk::k_khat<double><<<grid_for(c->M), 256, 0, c->stream>>>(c->ghat.p, nx, ny, nz, kx, ky, kz, denom,
                                                                       c->khat64.p + r * c->M);
        } else {
            c->khat32.alloc(8 * c->M);
            clk::k_khat<float><<<grid_for(c->M), 256, 0, c->stream>>>(c->ghat.p, nx, ny, nz, kx, ky, kz, denom,
                                                                      c->khat32.p + r * c->M);
        }
        CL_LAUNCHED();
    }
}

// 3D DCT-I of the octant held in c->ghat (three separable passes), then Khat per round.
void transform_kernel(cl_ctx* c) {
    const int n1[3] = {c->n[0] + 1, c->n[1] + 1, c->n[2] + 1};
    const long long total = (long long)n1[0] * n1[1] * n1[2];
    DevBuf<double> tmp;
    tmp.alloc(total);
    double* src = c->ghat.p;
    double* dst = tmp.p;
    long long inner = 1;
    for (int d = 0; d < 3; ++d) {
        const int L = n1[d];
        const int np = L - 1;
        std::vector<double> ct(2 * (size_t)np);
        const long double pi = 3.141592653589793238462643383279502884L;
        for (int t = 0; t < 2 * np; ++t) ct[t] = (double)std::cos(pi * (long double)t / (long double)np);
        DevBuf<double> dct;
        dct.upload(ct.data(), ct.size(), c->stream);
        const long long nlines = total / L;
        int nl = 16;
        while (nl > 1 && (size_t)(L * nl + 2 * np) * sizeof(double) > 160 * 1024) nl /= 2;
        const size_t smem = (size_t)(L * nl + 2 * np) * sizeof(double);
        ensure_smem(clk::k_dct1, smem);
        const long long blocks = (nlines + nl - 1) / nl;
        clk::k_dct1<<<(unsigned)blocks, 256, smem, c->stream>>>(src, dst, L, inner, nlines, nl, dct.p);
        CL_LAUNCHED();
        CL_CUDA(cudaStreamSynchronize(c->stream));  // dct table lifetime
        std::swap(src, dst);
        inner *= L;
    }
    if (src != c->ghat.p)
        CL_CUDA(cudaMemcpyAsync(c->ghat.p, src, total * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
    build_khat(c);
    CL_CUDA(cudaStreamSynchronize(c->stream));
    c->kernel_ready = true;
    ++c->kernel_version;
}

// ---------------------------------------------------------------------------------------
// Autotuner of the register passes (passes.hpp).  For each pass of a grid shape and
// precision, every compiled variant (radix split of the line length x lines per block) is
// timed with CUDA events on the request's own buffers, and the fastest is kept for the rest of
// the process.  Tuning runs at the first eager request of a shape (never inside a graph
// capture); CL_AUTOTUNE=0 keeps the default variants.
// ---------------------------------------------------------------------------------------
struct TuneKey {
    int pass, fp32, nx, ny, nz;
    bool operator<(const TuneKey& o) const {
        return std::tie(pass, fp32, nx, ny, nz) < std::tie(o.pass, o.fp32, o.nx, o.ny, o.nz);
    }
};
struct TuneEntry {
    clp::Variant v;
    int candidates = 0;
    double ms = 0, ms_default = 0;  // per launch of the tuning sample
};
std::mutex g_tune_mu;
std::map<TuneKey, TuneEntry> g_tune;

// Key of a pass on the grid the context's passes currently run on; fp32 carries the form: bit 0
// FP32 transforms, bit 1 the sub-lattice virtual grid.
TuneKey tune_key(const cl_ctx* c, int pass, bool fp32) {
    return TuneKey{pass, (fp32 ? 1 : 0) | c->tune_form, c->tune_dims[0], c->tune_dims[1], c->tune_dims[2]};
}
bool g_tune_loaded = false;

// CL_TUNE_FILE: choices persist across processes.  Lines "pass fp32 nx ny nz split half pad";
// the file is read once (before the first lookup) and every new choice is appended.
const char* tune_file() {
    const char* f = std::getenv("CL_TUNE_FILE");
    return (f && *f) ? f : nullptr;
}

void tune_load_locked() {  // g_tune_mu held
    if (g_tune_loaded) return;
    g_tune_loaded = true;
    const char* path = tune_file();
    if (!path) return;
    FILE* fh = std::fopen(path, "r");
    if (!fh) return;
    TuneKey k{};
    TuneEntry e;
    while (std::fscanf(fh, "%d %d %d %d %d %d %d %d", &k.pass, &k.fp32, &k.nx, &k.ny, &k.nz, &e.v.split, &e.v.half,
                       &e.v.pad) == 8) {
        if (k.pass < 0 || k.pass >= clp::kNumPasses) continue;
        e.candidates = 0;  // loaded, not timed in this process
        g_tune[k] = e;
    }
    std::fclose(fh);
}

void tune_save(const TuneKey& k, const TuneEntry& e) {
    const char* path = tune_file();
    if (!path) return;
    if (FILE* fh = std::fopen(path, "a")) {
        std::fprintf(fh, "%d %d %d %d %d %d %d %d\n", k.pass, k.fp32, k.nx, k.ny, k.nz, e.v.split, e.v.half,
                     e.v.pad);
        std::fclose(fh);
    }
}

bool autotune_enabled() {
    const char* e = std::getenv("CL_AUTOTUNE");
    return !(e && e[0] == '0');
}

bool register_passes_enabled() { return !std::getenv("CL_NO_REGISTER_FFT"); }

clp::Variant tuned_variant(const cl_ctx* c, int pass, bool fp32) {
    if (const char* f = std::getenv("CL_TUNE_FORCE")) {  // "split,half[,pad]": one variant for every pass
        clp::Variant v;
        if (std::sscanf(f, "%d,%d,%d", &v.split, &v.half, &v.pad) >= 2) return v;
    }
    std::lock_guard<std::mutex> g(g_tune_mu);
    tune_load_locked();
    auto it = g_tune.find(tune_key(c, pass, fp32));
    return it == g_tune.end() ? clp::Variant{} : it->second.v;
}

bool stream_capturing(cudaStream_t s) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    CL_CUDA(cudaStreamIsCapturing(s, &st));
    return st != cudaStreamCaptureStatusNone;
}

// Times launch(variant) -- one warm-up and three timed launches per candidate -- and records
// the fastest variant of the pass.  Candidates: the split variants of the line length `len`,
// each with the default and (FP32) the half lines per block; the default is tried first.
template <typename F>
void tune_pass(cl_ctx* c, int pass, bool fp32, int len, F&& launch) {
    const TuneKey key = tune_key(c, pass, fp32);
    {
        std::lock_guard<std::mutex> g(g_tune_mu);
        tune_load_locked();
        if (g_tune.count(key)) return;
    }
    std::vector<clp::Variant> cands;
    const int pads = (fp32 && pass == clp::kXFwd) ? 2 : 1;
    for (int sv = 0; sv < clp::split_variants(len); ++sv)
        for (int h = 0; h < (fp32 ? 2 : 1); ++h)
            for (int pd = 0; pd < pads; ++pd) cands.push_back(clp::Variant{sv, h, pd});
    TuneEntry best;
    best.candidates = (int)cands.size();
    if (cands.size() >= 2) {
        cudaEvent_t a, b;
        CL_CUDA(cudaEventCreate(&a));
        CL_CUDA(cudaEventCreate(&b));
        double best_ms = 1e30;
        for (size_t i = 0; i < cands.size(); ++i) {
            launch(cands[i]);
            CL_LAUNCHED();
            CL_CUDA(cudaEventRecord(a, c->stream));
            for (int k = 0; k < 3; ++k) launch(cands[i]);
            CL_LAUNCHED();
            CL_CUDA(cudaEventRecord(b, c->stream));
            CL_CUDA(cudaEventSynchronize(b));
            float ms = 0;
            CL_CUDA(cudaEventElapsedTime(&ms, a, b));
            const double per = ms / 3.0;
            if (i == 0) best.ms_default = per;
            if (per < best_ms) {
                best_ms = per;
                best.v = cands[i];
            }
        }
        best.ms = best_ms;
        cudaEventDestroy(a);
        cudaEventDestroy(b);
    }
    std::lock_guard<std::mutex> g(g_tune_mu);
    g_tune[key] = best;
    tune_save(key, best);
}

// Fused plane passes against the separate passes they replace: times launch() like
// tune_pass and records split = 1 (use the fused kernel) when it beats sep_ms, the sum of the
// tuned separate passes' times on the same sample.
template <typename F>
void tune_plane(cl_ctx* c, int pass, bool fp32, double sep_ms, F&& launch) {
    const TuneKey key = tune_key(c, pass, fp32);
    {
        std::lock_guard<std::mutex> g(g_tune_mu);
        tune_load_locked();
        if (g_tune.count(key)) return;
    }
    cudaEvent_t a, b;
    CL_CUDA(cudaEventCreate(&a));
    CL_CUDA(cudaEventCreate(&b));
    launch();
    CL_LAUNCHED();
    CL_CUDA(cudaEventRecord(a, c->stream));
    for (int k = 0; k < 3; ++k) launch();
    CL_LAUNCHED();
    CL_CUDA(cudaEventRecord(b, c->stream));
    CL_CUDA(cudaEventSynchronize(b));
    float ms = 0;
    CL_CUDA(cudaEventElapsedTime(&ms, a, b));
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    TuneEntry e;
    e.candidates = 2;
    e.ms = ms / 3.0;
    e.ms_default = sep_ms;
    e.v.split = (sep_ms <= 0 || e.ms < sep_ms) ? 1 : 0;  // ms: the fused pass; ms_default: separate
    std::lock_guard<std::mutex> g(g_tune_mu);
    g_tune[key] = e;
    tune_save(key, e);
}

double tuned_ms(const cl_ctx* c, int pass, bool fp32) {
    std::lock_guard<std::mutex> g(g_tune_mu);
    auto it = g_tune.find(tune_key(c, pass, fp32));
    return it == g_tune.end() ? 0.0 : it->second.ms;
}

// Whether the fused plane pass replaces the separate ones: CL_XY_PLANE=0/1 decides outright;
// with forced variants (CL_TUNE_FORCE) the separate passes run; otherwise the tuned choice,
// and the fused pass when nothing was tuned.
bool use_plane(const cl_ctx* c, int pass, bool fp32, bool supported) {
    if (!supported) return false;
    if (const char* e = std::getenv("CL_XY_PLANE")) return e[0] != '0';
    if (std::getenv("CL_TUNE_FORCE")) return false;
    std::lock_guard<std::mutex> g(g_tune_mu);
    tune_load_locked();
    auto it = g_tune.find(tune_key(c, pass, fp32));
    return it == g_tune.end() ? true : it->second.v.split != 0;
}

// Number of atoms listed by a row CSR (host-side copy kept with the CSR).
long long row_ptr_count(cl_ctx* c, const int* row_ptr) {
    return row_ptr == c->row_ptr.p ? c->n_sorted : c->M;
}

// One request's transforms: for every density p in [0, np) (rho rows), V[p] = the 8-round
// convolution (the rounds of round_mask) at the atoms of the row CSR.  For a chunk of densities,
// each round's inverse x pass writes its values at the atoms (type T) to a slot of the rounds
// buffer; k_round_sum then forms V in FP64.  buf holds `chunk` grids of type T.
template <typename T>
void run_rounds(cl_ctx* c, const cx<T>* rho, long long rho_stride, int np, const int* row_ptr,
                const int* cell, cx<double>* V, long long v_stride, int round_mask) {
    const int nx = c->n[0], ny = c->n[1], nz = c->n[2];
    const int nrows = ny * nz;
    const long long nxy = (long long)nx * ny;
    const size_t grid_bytes = sizeof(cx<T>) * (size_t)c->M;
    for (int d = 0; d < 3; ++d) c->tune_dims[d] = c->n[d];
    c->tune_form = 0;
    // Densities per chunk.  When a few grids fit in L2, chunks are sized so that the passes of
    // one round hand their output to the next pass through L2; otherwise chunks are as large
    // as 60% of the free memory allows (fewer, larger launches and Khat reuse in the z pass).
    const long long n_at = row_ptr_count(c, row_ptr);
    const int n_rounds = __builtin_popcount(round_mask & 0xFF);
    if (n_rounds == 0) {  // no round of this share (a split over more ranks than rounds)
        CL_CUDA(cudaMemset2DAsync(V, sizeof(cx<double>) * v_stride, 0, sizeof(cx<double>) * n_at, np, c->stream));
        return;
    }
    const size_t round_bytes = sizeof(cx<T>) * (size_t)n_at * n_rounds;  // per density
    const size_t l2_budget = l2_chunk_bytes();
    const size_t by_l2 = l2_budget / grid_bytes;
    const size_t all_rounds = (size_t)np * n_rounds * grid_bytes;
    const bool few = all_rounds <= (512ull << 20) && l2_budget == 0 && np * n_rounds <= 65535;  // gridDim.y
    int chunk = std::max(np, 1);
    size_t budget = SIZE_MAX;  // of this request; the free memory is asked for only when its buffers must grow
    if (l2_budget != 0 || c->work.n < (few ? all_rounds : np * grid_bytes) || c->rounds.n < np * round_bytes) {
        budget = (size_t)(0.6 * (double)(free_device_bytes() + c->work.n + c->rounds.n));
        const size_t by_mem = std::max<size_t>(1, budget / (grid_bytes + round_bytes));
        chunk = (int)std::max<size_t>(1, std::min<size_t>((size_t)chunk, by_l2 >= 2 ? by_l2 : by_mem));
    }
    // All rounds in one launch of each pass where their grids take at most 512 MB: 8 rounds of launches
    // become one, and a small grid's rounds fill the SMs together (B200, a request's kernels: 32^3 in FP64,
    // 10 densities, 0.388 -> 0.120 ms; 45^3 in FP32, 10 densities, 0.471 -> 0.183; 64^3 in FP64, one
    // density, 0.360 -> 0.127).  Larger grids fill the SMs round by round and keep one
    // round's buffers.
    const bool together = few && chunk == np && all_rounds <= budget / 2;
    const int per_launch = together ? n_rounds : 1;
    c->work.alloc(std::max(c->work.n, together ? all_rounds : (size_t)chunk * grid_bytes));
    c->rounds.alloc(std::max(c->rounds.n, (size_t)chunk * round_bytes));
    cx<T>* buf = reinterpret_cast<cx<T>*>(c->work.p);
    cx<T>* tr = reinterpret_cast<cx<T>*>(c->rounds.p);
    const T* kh = sizeof(T) == 4 ? (const T*)c->khat32.p : (const T*)c->khat64.p;

    const Axis& X = c->ax[0];
    const Axis& Y = c->ax[1];
    const Axis& Z = c->ax[2];
    const cx<T>* twx = sizeof(T) == 4 ? (const cx<T>*)X.tw32.p : (const cx<T>*)X.tw64.p;
    const cx<T>* twy = sizeof(T) == 4 ? (const cx<T>*)Y.tw32.p : (const cx<T>*)Y.tw64.p;
    const cx<T>* twz = sizeof(T) == 4 ? (const cx<T>*)Z.tw32.p : (const cx<T>*)Z.tw64.p;

    const XTile xt = x_tile<T>(nx, nrows);
    const LTile yt = l_tile<T>(ny, false);
    const LTile zt = l_tile<T>(nz, true);
    ensure_smem(clk::k_xfwd<T>, xt.smem);
    ensure_smem(clk::k_xinv<T>, xt.smem);
    ensure_smem(clk::k_ypass<-1, T>, yt.smem);
    ensure_smem(clk::k_ypass<+1, T>, yt.smem);
    ensure_smem(clk::k_zpass<T>, zt.smem);
    const int xblocks = (nrows + xt.rows - 1) / xt.rows;
    const int ychunks = (nx + yt.W - 1) / yt.W;
    const long long zblocks = (nxy + zt.W - 1) / zt.W;
    // Rows without atoms are skipped (not stored / not loaded) when the x and y passes are both
    // the register ones, which agree on it; CL_NO_ROW_SKIP turns it off.
    const bool reg_x = register_passes_enabled() && clp::split_variants(nx) > 0;
    const bool reg_y = register_passes_enabled() && clp::split_variants(ny) > 0;
    const bool reg_z = register_passes_enabled() && clp::split_variants(nz) > 0;
    const int skip_empty = (reg_x && reg_y && !std::getenv("CL_NO_ROW_SKIP")) ? 1 : 0;
    const bool fp32 = sizeof(T) == 4;
    const bool plane_ok = reg_x && reg_y && clp::plane_supported(fp32, nx, ny);

    // Autotuning at the first eager request of this shape: the variants run on the first
    // densities of the request (about 512 MB of grids) in the work and rounds buffers, which
    // the request's own passes overwrite afterwards.
    if (autotune_enabled() && !std::getenv("CL_TUNE_FORCE") && np > 0 && !stream_capturing(c->stream)) {
        const int cnt_t = (int)std::max<size_t>(1, std::min<size_t>((size_t)chunk, (512ull << 20) / grid_bytes));
        const clk::RoundPhase rp0{c->ax[0].phase.p, c->ax[1].phase.p, c->ax[2].phase.p, 0, 0, 0, 0, 1, 0};
        const int* rp_skip = skip_empty ? row_ptr : nullptr;
        if (reg_x)
            tune_pass(c, clp::kXFwd, fp32, nx, [&](clp::Variant v) {
                clp::xfwd<T>(c->stream, v, rho, rho_stride, row_ptr, cell, buf, c->M, twx, rp0, nx, ny, nrows, cnt_t,
                             skip_empty);
            });
        if (reg_y) {
            tune_pass(c, clp::kYFwd, fp32, ny, [&](clp::Variant v) {
                clp::ycol<-1, T>(c->stream, v, buf, c->M, twy, nx, ny, nz, cnt_t, rp_skip);
            });
            tune_pass(c, clp::kYInv, fp32, ny, [&](clp::Variant v) {
                clp::ycol<+1, T>(c->stream, v, buf, c->M, twy, nx, ny, nz, cnt_t, rp_skip);
            });
        }
        if (reg_z)
            tune_pass(c, clp::kZConv, fp32, nz, [&](clp::Variant v) {
                clp::zconv<T>(c->stream, v, buf, c->M, twz, kh, nxy, nz, cnt_t, clp::Rounds{});
            });
        if (reg_x)
            tune_pass(c, clp::kXInv, fp32, nx, [&](clp::Variant v) {
                clp::xinv<T>(c->stream, v, buf, c->M, twx, row_ptr, cell, tr, n_at, nx, nrows, cnt_t);
            });
        if (plane_ok && !std::getenv("CL_XY_PLANE")) {
            tune_plane(c, clp::kXYFwd, fp32, tuned_ms(c, clp::kXFwd, fp32) + tuned_ms(c, clp::kYFwd, fp32), [&] {
                clp::xyfwd<T>(c->stream, rho, rho_stride, row_ptr, cell, buf, c->M, twx, rp0, nx, ny, nz, cnt_t);
            });
            tune_plane(c, clp::kXYInv, fp32, tuned_ms(c, clp::kYInv, fp32) + tuned_ms(c, clp::kXInv, fp32), [&] {
                clp::xyinv<T>(c->stream, buf, c->M, twx, row_ptr, cell, tr, n_at, nx, ny, nz, cnt_t);
            });
        }
    }
    const bool xy_fwd = use_plane(c, clp::kXYFwd, fp32, plane_ok);
    const bool xy_inv = use_plane(c, clp::kXYInv, fp32, plane_ok);
    const clp::Variant v_xf = tuned_variant(c, clp::kXFwd, fp32), v_yf = tuned_variant(c, clp::kYFwd, fp32),
                       v_z = tuned_variant(c, clp::kZConv, fp32), v_yi = tuned_variant(c, clp::kYInv, fp32),
                       v_xi = tuned_variant(c, clp::kXInv, fp32);

    // algorithmic bytes per density of each pass (minimum HBM traffic of its work); with
    // skipped rows only the live fraction of a row-side sweep counts
    const double gbytes = (double)grid_bytes;
    const double atoms = (double)(row_ptr_count(c, row_ptr));
    const double live = (skip_empty && row_ptr == c->row_ptr.p) ? (double)c->live_rows / nrows : 1.0;
    const double row_side = (row_ptr == c->row_ptr.p) ? (double)c->live_rows / nrows : 1.0;
    for (int p0 = 0; p0 < np; p0 += chunk) {
        const int cnt = std::min(chunk, np - p0);
        const cx<T>* rho_c = rho + (long long)p0 * rho_stride;
        cx<double>* V_c = V + (long long)p0 * v_stride;
        const long long tr_slot = (long long)cnt * n_at;  // elements per round
        int done = 0;                                      // rounds of the mask launched so far
        for (int r = 0; r < 8; ++r) {
            if (!((round_mask >> r) & 1)) continue;
            clp::Rounds rounds{0, 0, (long long)cnt * c->M};
            for (; r < 8 && rounds.n < per_launch; ++r)
                if ((round_mask >> r) & 1) rounds.list |= (unsigned)r << (4 * rounds.n++);
            --r;
            const int grids = cnt * rounds.n;  // one after another, a round's densities together
            cx<T>* tr_r = tr + done * tr_slot;
            done += rounds.n;
            const clk::RoundPhase rp{c->ax[0].phase.p, c->ax[1].phase.p, c->ax[2].phase.p, 0, 0, 0,
                                     rounds.list,      rounds.n,          rounds.stride};
            cudaEvent_t e = prof_begin(c);
            if (xy_fwd) {
                clp::xyfwd<T>(c->stream, rho_c, rho_stride, row_ptr, cell, buf, c->M, twx, rp, nx, ny, nz, cnt);
            } else if (!(reg_x && clp::xfwd<T>(c->stream, v_xf, rho_c, rho_stride, row_ptr, cell, buf, c->M, twx,
                                                rp, nx, ny, nrows, cnt, skip_empty))) {
                clk::k_xfwd<T><<<dim3(xblocks, 1, rounds.n), 256, xt.smem, c->stream>>>(
                    rho_c, rho_stride, row_ptr, cell, buf, c->M, X.plan, twx, rp, nx, ny, nrows, xt.rows, xt.ld, cnt);
            }
            CL_LAUNCHED();
            prof_end(c, e, CL_KCLASS_XFWD,
                     grids * (atoms * (double)sizeof(cx<T>) + (xy_fwd ? 1.0 : live) * gbytes) + atoms * 4.0);
            if (!xy_fwd) {
                e = prof_begin(c);
                if (!(reg_y && clp::ycol<-1, T>(c->stream, v_yf, buf, c->M, twy, nx, ny, nz, grids,
                                                 skip_empty ? row_ptr : nullptr)))
                    clk::k_ypass<-1, T><<<dim3(ychunks * nz, grids), 256, yt.smem, c->stream>>>(
                        buf, c->M, Y.plan, twy, nx, ny, yt.W, ychunks);
                CL_LAUNCHED();
                prof_end(c, e, CL_KCLASS_YPASS, grids * (1.0 + live) * gbytes);
            }
            e = prof_begin(c);
            if (!(reg_z && clp::zconv<T>(c->stream, v_z, buf, c->M, twz, kh, nxy, nz, cnt, rounds)))
                clk::k_zpass<T><<<dim3((unsigned)zblocks, zgroups(zblocks * rounds.n, cnt), rounds.n), 256, zt.smem,
                                  c->stream>>>(buf, c->M, Z.plan, twz, kh, nxy, nz, zt.W, cnt, 0, rounds.list,
                                               rounds.stride);
            CL_LAUNCHED();
            prof_end(c, e, CL_KCLASS_ZPASS, grids * 2.0 * gbytes + rounds.n * (double)c->M * sizeof(T));
            if (!xy_inv) {
                e = prof_begin(c);
                if (!(reg_y && clp::ycol<+1, T>(c->stream, v_yi, buf, c->M, twy, nx, ny, nz, grids,
                                                 skip_empty ? row_ptr : nullptr)))
                    clk::k_ypass<+1, T><<<dim3(ychunks * nz, grids), 256, yt.smem, c->stream>>>(
                        buf, c->M, Y.plan, twy, nx, ny, yt.W, ychunks);
                CL_LAUNCHED();
                prof_end(c, e, CL_KCLASS_YPASS, grids * (1.0 + live) * gbytes);
            }
            e = prof_begin(c);
            if (xy_inv) {
                clp::xyinv<T>(c->stream, buf, c->M, twx, row_ptr, cell, tr_r, n_at, nx, ny, nz, grids);
            } else if (!(reg_x && clp::xinv<T>(c->stream, v_xi, buf, c->M, twx, row_ptr, cell, tr_r, n_at, nx, nrows,
                                                grids))) {
                clk::k_xinv<T><<<xblocks, 256, xt.smem, c->stream>>>(buf, c->M, X.plan, twx, row_ptr, cell, tr_r,
                                                                     n_at, nx, nrows, xt.rows, xt.ld, grids);
            }
            CL_LAUNCHED();
            prof_end(c, e, CL_KCLASS_XINV,
                     grids * ((xy_inv ? 1.0 : row_side) * gbytes + atoms * (double)sizeof(cx<T>)) + atoms * 4.0);
        }
        if (n_rounds > 0) {
            const clk::RoundPhase base{c->ax[0].phase.p, c->ax[1].phase.p, c->ax[2].phase.p, 0, 0, 0, 0, 1, 0};
            const long long blocks = std::min<long long>((n_at + 255) / 256, 148LL * 16);
            cudaEvent_t e = prof_begin(c);
            clk::k_round_sum<T><<<dim3((unsigned)blocks, zgroups(blocks, cnt)), 256, 0, c->stream>>>(
                tr, tr_slot, n_at, round_mask & 0xFF, base, cell, nx, ny, n_at, V_c, v_stride, cnt);
            CL_LAUNCHED();
            prof_end(c, e, CL_KCLASS_ROUND_SUM,
                     cnt * atoms * (n_rounds * (double)sizeof(cx<T>) + 16.0) + atoms * 4.0);
        }
    }
}

// Pair densities are complex128 in the plain form and complex64 in the FP32 form (rounded
// once from their FP64 sums); buffers are addressed in elements of the form's type.
size_t rho_bytes(const cl_ctx* c) { return fp64_form(c) ? sizeof(cx<double>) : sizeof(cx<float>); }
void* rho_at(const cl_ctx* c, void* base, long long elems) {
    return static_cast<unsigned char*>(base) + elems * (long long)rho_bytes(c);
}

void run_rounds_mode(cl_ctx* c, const void* rho, long long rho_stride, int np, const int* row_ptr, const int* cell,
                     cx<double>* V, long long v_stride, int round_mask = 0xFF) {
    if (fp64_form(c))
        run_rounds<double>(c, static_cast<const cx<double>*>(rho), rho_stride, np, row_ptr, cell, V, v_stride,
                           round_mask);
    else
        run_rounds<float>(c, static_cast<const cx<float>*>(rho), rho_stride, np, row_ptr, cell, V, v_stride,
                          round_mask);
}


// ---------------------------------------------------------------------------------------
// Sub-lattice decomposition (sublattice.cuh)
// ---------------------------------------------------------------------------------------

// Plans and twiddles of the transform lengths, the class kernels H (from the kernel spectrum in
// c->ghat) and the class phases, built once per kernel and class set.  Not during a capture.
void ensure_sl_tables(cl_ctx* c) {
    Sublattice& sl = c->sl;
    if (sl.tables_version == c->kernel_version) return;
    if (stream_capturing(c->stream))
        cl::fail(CL_ERR_STATE, "the sub-lattice tables must be built by an eager call before a capture");
    const bool fp32 = !fp64_form(c);
    for (int d = 0; d < 3; ++d) {
        Axis& A = sl.ax[d];
        A.plan = make_plan(sl.pad[d]);
        auto t64 = twiddles64(sl.pad[d]);
        std::vector<cx<float>> t32(t64.size());
        for (size_t i = 0; i < t64.size(); ++i) t32[i] = cx<float>{(float)t64[i].re, (float)t64[i].im};
        A.tw64.upload(t64.data(), t64.size(), c->stream);
        A.tw32.upload(t32.data(), t32.size(), c->stream);
    }
    const int px = sl.pad[0], py = sl.pad[1], pz = sl.pad[2];
    const long long nxy = (long long)px * py, nq = nxy * pz;
    // class kernels H_r(q): the residue representatives and the m-th roots of unity
    clk::SlRes res{};
    res.nh = sl.table.nh;
    res.m = sl.m;
    for (int h = 0; h < res.nh; ++h)
        for (int d = 0; d < 3; ++d) res.rep[h][d] = sl.table.rep[h][d];
    for (int e = 0; e < 4; ++e) {  // exact: m is 2 or 4
        const int q = (sl.m == 4) ? e : 2 * e;  // quarter turns
        static const double cq[4] = {1.0, 0.0, -1.0, 0.0}, sq[4] = {0.0, 1.0, 0.0, -1.0};
        res.wc[e] = cq[q & 3];
        res.ws[e] = sq[q & 3];
    }
    const double denom = (double)((unsigned long long)c->M * 8ull);
    const int blocks = grid_for(nq);
    sl.zw = sl.zb ? clp::zw_zb_supported(pz) : sl.S == 2 && clp::zw_pair_supported(pz);
    if (sl.zb || sl.zw) {
        // raw class kernels in FP64, then their Walsh-Hadamard form (sublattice.cuh) rounded once
        DevBuf<cx<double>> raw;
        raw.alloc((size_t)res.nh * nq);
        clk::k_sl_build_h<double><<<blocks, 256, 0, c->stream>>>(c->ghat.p, c->n[0], c->n[1], c->n[2], px, py, pz,
                                                                 res, denom, raw.p);
        CL_LAUNCHED();
        clk::SlWht w{};
        for (int k = 0; k < sl.S; ++k) {
            w.src[k] = sl.table.h[k * clk::kSlMaxClasses];  // (class k, class 0): alpha_k, then beta_k
            w.cj[k] = sl.table.cj[k * clk::kSlMaxClasses];
        }
        if (sl.zw) {
            const int half = sl.S / 2;  // class 0 of the second half
            clk::ZwBuild zb{};
            std::memcpy(zb.src, w.src, sizeof zb.src);
            std::memcpy(zb.cj, w.cj, sizeof zb.cj);
            for (int d = 0; d < 3; ++d) {
                zb.delta[d] = sl.off[half][d] - sl.off[0][d];
                zb.n[d] = c->n[d];
                zb.p[d] = sl.pad[d];
                // the half's offsets along the axis are its class 0's and that +- 2 (zinc-blende, mod 4)
                for (int h = 0; h < 2; ++h) zb.sgn[h][d] = sl.off[h * half][d] < 2 ? 1 : -1;
            }
            const auto build = [&](auto tag) {
                using T = decltype(tag);
                sl.zw_tab.alloc(sizeof(clk::Quad<T>) * (sl.zb ? 3 : 1) * nq);
                auto* tab = reinterpret_cast<clk::Quad<T>*>(sl.zw_tab.p);
                if (sl.zb) {
                    sl.zw_col.alloc(sizeof(cx<T>) * 7 * nxy);
                    sl.zw_zph.alloc(sizeof(cx<T>) * 2 * pz);
                    clk::k_zw_table<T, clk::kZwZb><<<blocks, 256, 0, c->stream>>>(raw.p, zb, tab);
                    CL_LAUNCHED();
                    clk::k_zw_columns<T><<<grid_for(nxy), 256, 0, c->stream>>>(
                        zb, reinterpret_cast<cx<T>*>(sl.zw_col.p), reinterpret_cast<cx<T>*>(sl.zw_zph.p));
                } else {
                    clk::k_zw_table<T, clk::kZwPair><<<blocks, 256, 0, c->stream>>>(raw.p, zb, tab);
                }
            };
            if (fp32)
                build(float{});
            else
                build(double{});
        } else if (fp32) {
            sl.H32.alloc((size_t)8 * nq);
            clk::k_sl_zb_wht<float><<<blocks, 256, 0, c->stream>>>(raw.p, nq, w, sl.H32.p);
        } else {
            sl.H64.alloc((size_t)8 * nq);
            clk::k_sl_zb_wht<double><<<blocks, 256, 0, c->stream>>>(raw.p, nq, w, sl.H64.p);
        }
        CL_LAUNCHED();
        CL_CUDA(cudaStreamSynchronize(c->stream));  // raw goes out of scope
    } else if (fp32) {
        sl.H32.alloc((size_t)res.nh * nq);
        clk::k_sl_build_h<float><<<blocks, 256, 0, c->stream>>>(c->ghat.p, c->n[0], c->n[1], c->n[2], px, py, pz, res,
                                                                denom, sl.H32.p);
    } else {
        sl.H64.alloc((size_t)res.nh * nq);
        clk::k_sl_build_h<double><<<blocks, 256, 0, c->stream>>>(c->ghat.p, c->n[0], c->n[1], c->n[2], px, py, pz,
                                                                 res, denom, sl.H64.p);
    }
    CL_LAUNCHED();
    if (sl.zw) {
        sl.tables_version = c->kernel_version;
        return;
    }
    // phases: phxy[s][ky][kx] = exp(-i pi (kx bx/nx + ky by/ny)), phz[b][kz] = exp(-i pi kz b/nz) (b < m;
    // rows up to 4), in extended precision and rounded once
    const long double pi = 3.141592653589793238462643383279502884L;
    std::vector<cx<double>> phxy((size_t)sl.S * nxy), phz((size_t)4 * pz, cx<double>{0.0, 0.0});
    for (int s2 = 0; s2 < sl.S; ++s2)
        for (int ky = 0; ky < py; ++ky)
            for (int kx = 0; kx < px; ++kx) {
                const long double a = -pi * ((long double)kx * sl.off[s2][0] / c->n[0] +
                                             (long double)ky * sl.off[s2][1] / c->n[1]);
                phxy[(size_t)s2 * nxy + (size_t)ky * px + kx] = cx<double>{(double)std::cos(a), (double)std::sin(a)};
            }
    for (int b = 0; b < sl.m; ++b)
        for (int kz = 0; kz < pz; ++kz) {
            const long double a = -pi * (long double)kz * b / c->n[2];
            phz[(size_t)b * pz + kz] = cx<double>{(double)std::cos(a), (double)std::sin(a)};
        }
    if (fp32) {
        std::vector<cx<float>> f1(phxy.size()), f2(phz.size());
        for (size_t i = 0; i < phxy.size(); ++i) f1[i] = cx<float>{(float)phxy[i].re, (float)phxy[i].im};
        for (size_t i = 0; i < phz.size(); ++i) f2[i] = cx<float>{(float)phz[i].re, (float)phz[i].im};
        sl.phxy32.upload(f1.data(), f1.size(), c->stream);
        sl.phz32.upload(f2.data(), f2.size(), c->stream);
        CL_CUDA(cudaStreamSynchronize(c->stream));
    } else {
        sl.phxy64.upload(phxy.data(), phxy.size(), c->stream);
        sl.phz64.upload(phz.data(), phz.size(), c->stream);
        CL_CUDA(cudaStreamSynchronize(c->stream));
    }
    sl.tables_version = c->kernel_version;
}

// One request's transforms in the sub-lattice form: for every density p in [0, np), V[p] at the
// atoms (virtual-grid order).  Per chunk of densities: x and y forward passes on the virtual
// grid (fused plane pass where compiled and faster), the z pass with class mixing, the y and x
// inverse passes writing the values at the atoms; in the FP32 form they are widened to V.
template <typename T>
void run_sublattice(cl_ctx* c, const cx<T>* rho, long long rho_stride, int np, void* V_any, long long v_stride,
                    bool v32) {
    cx<double>* V = static_cast<cx<double>*>(V_any);
    ensure_sl_tables(c);
    const Sublattice& sl = c->sl;
    const int nx = sl.vn[0], ny = sl.vn[1], nz = sl.vn[2];
    const int nrows = ny * nz;
    const long long nxy = (long long)nx * ny;
    const long long vM = sl.vM;
    const size_t grid_bytes = sizeof(cx<T>) * (size_t)vM;
    const bool fp32 = sizeof(T) == 4;
    for (int d = 0; d < 3; ++d) c->tune_dims[d] = sl.vn[d];
    c->tune_form = 2;
    const int* row_ptr = c->row_ptr.p;
    const int* cell = c->cell_sorted.p;
    const long long n_at = c->n_sorted;
    // values at the atoms: straight into V in FP64, and in FP32 when the reductions read FP32
    // potentials (v32); otherwise through the rounds buffer, widened to V
    const bool via_tr = fp32 && !v32;
    const size_t at_bytes = via_tr ? sizeof(cx<T>) * (size_t)n_at : 0;
    // the whole request where the buffers kept from the last one hold it (asking the driver for the free
    // memory takes longer than a small request's launches), else as much as 60% of the free memory holds
    int chunk = std::max(np, 1);
    if (c->work.n < chunk * grid_bytes || (via_tr && c->rounds.n < chunk * at_bytes)) {
        const size_t budget = (size_t)(0.6 * (double)(free_device_bytes() + c->work.n + c->rounds.n));
        chunk = (int)std::max<size_t>(1, std::min<size_t>((size_t)chunk, budget / (grid_bytes + at_bytes)));
    }
    c->work.alloc(std::max(c->work.n, (size_t)chunk * grid_bytes));
    if (via_tr) c->rounds.alloc(std::max(c->rounds.n, (size_t)chunk * at_bytes));
    cx<T>* buf = reinterpret_cast<cx<T>*>(c->work.p);
    cx<T>* tr = reinterpret_cast<cx<T>*>(c->rounds.p);
    const cx<T>* twx = fp32 ? (const cx<T>*)sl.ax[0].tw32.p : (const cx<T>*)sl.ax[0].tw64.p;
    const cx<T>* twy = fp32 ? (const cx<T>*)sl.ax[1].tw32.p : (const cx<T>*)sl.ax[1].tw64.p;
    const cx<T>* twz = fp32 ? (const cx<T>*)sl.ax[2].tw32.p : (const cx<T>*)sl.ax[2].tw64.p;
    const cx<T>* H = fp32 ? (const cx<T>*)sl.H32.p : (const cx<T>*)sl.H64.p;
    const cx<T>* phxy = fp32 ? (const cx<T>*)sl.phxy32.p : (const cx<T>*)sl.phxy64.p;
    const cx<T>* phz = fp32 ? (const cx<T>*)sl.phz32.p : (const cx<T>*)sl.phz64.p;
    clk::SlMix mix{};
    mix.S = sl.S;
    for (int s2 = 0; s2 < clk::kSlMaxClasses; ++s2) mix.offz[s2] = s2 < sl.S ? sl.off[s2][2] : 0;
    for (int i = 0; i < clk::kSlMaxClasses * clk::kSlMaxClasses; ++i) {
        mix.h[i] = sl.table.h[i];
        mix.cj[i] = sl.table.cj[i];
    }
    const XTile xt = x_tile<T>(nx, nrows);
    const LTile yt = l_tile<T>(ny, false);
    ensure_smem(clk::k_xfwd<T>, xt.smem);
    ensure_smem(clk::k_xinv<T>, xt.smem);
    ensure_smem(clk::k_ypass<-1, T>, yt.smem);
    ensure_smem(clk::k_ypass<+1, T>, yt.smem);
    const int xblocks = (nrows + xt.rows - 1) / xt.rows;
    const int ychunks = (nx + yt.W - 1) / yt.W;
    const bool reg_x = register_passes_enabled() && clp::split_variants(nx) > 0;
    const bool reg_y = register_passes_enabled() && clp::split_variants(ny) > 0;
    const int skip_empty = (reg_x && reg_y && !std::getenv("CL_NO_ROW_SKIP")) ? 1 : 0;
    const bool plane_ok = reg_x && reg_y && clp::plane_supported(fp32, nx, ny);
    // Class planes: the quadrant plane passes, at every length compiled the fastest measured
    // (36 densities of 128 x 128 planes: 0.57 ms forward and 0.74 inverse, the general plane passes 0.94
    // and 0.89; 820 of 64 x 64: 1.37 and 1.58, 1.94 and 1.89; 78 of 48 x 48: 0.082 and 0.081, the
    // separate passes 0.159 and 0.165); CL_NO_QPLANE=1 keeps the general ones
    const bool qplane = clp::quadrant_supported(fp32, nx, ny) && !std::getenv("CL_NO_QPLANE");
    // no phase in any pass: the rounds' phase tables are never read with kappa = 0
    const clk::RoundPhase rp0{c->ax[0].phase.p, c->ax[1].phase.p, c->ax[2].phase.p, 0, 0, 0, 0, 1, 0};
    cx<T>* out0 = via_tr ? tr : static_cast<cx<T>*>(V_any);
    const long long out_stride = via_tr ? n_at : v_stride;
    if (autotune_enabled() && !std::getenv("CL_TUNE_FORCE") && np > 0 && !qplane && !stream_capturing(c->stream)) {
        const int cnt_t = (int)std::max<size_t>(1, std::min<size_t>((size_t)chunk, (512ull << 20) / grid_bytes));
        const int* rp_skip = skip_empty ? row_ptr : nullptr;
        if (reg_x)
            tune_pass(c, clp::kXFwd, fp32, nx, [&](clp::Variant v) {
                clp::xfwd<T>(c->stream, v, rho, rho_stride, row_ptr, cell, buf, vM, twx, rp0, nx, ny, nrows, cnt_t,
                             skip_empty);
            });
        if (reg_y) {
            tune_pass(c, clp::kYFwd, fp32, ny, [&](clp::Variant v) {
                clp::ycol<-1, T>(c->stream, v, buf, vM, twy, nx, ny, nz, cnt_t, rp_skip);
            });
            tune_pass(c, clp::kYInv, fp32, ny, [&](clp::Variant v) {
                clp::ycol<+1, T>(c->stream, v, buf, vM, twy, nx, ny, nz, cnt_t, rp_skip);
            });
        }
        if (reg_x)
            tune_pass(c, clp::kXInv, fp32, nx, [&](clp::Variant v) {
                clp::xinv<T>(c->stream, v, buf, vM, twx, row_ptr, cell, out0, out_stride, nx, nrows, cnt_t);
            });
        if (plane_ok && !std::getenv("CL_XY_PLANE")) {
            tune_plane(c, clp::kXYFwd, fp32, tuned_ms(c, clp::kXFwd, fp32) + tuned_ms(c, clp::kYFwd, fp32), [&] {
                clp::xyfwd<T>(c->stream, rho, rho_stride, row_ptr, cell, buf, vM, twx, rp0, nx, ny, nz, cnt_t);
            });
            tune_plane(c, clp::kXYInv, fp32, tuned_ms(c, clp::kYInv, fp32) + tuned_ms(c, clp::kXInv, fp32), [&] {
                clp::xyinv<T>(c->stream, buf, vM, twx, row_ptr, cell, out0, out_stride, nx, ny, nz, cnt_t);
            });
        }
    }
    const bool xy_fwd = use_plane(c, clp::kXYFwd, fp32, plane_ok);
    const bool xy_inv = use_plane(c, clp::kXYInv, fp32, plane_ok);
    const clp::Variant v_xf = tuned_variant(c, clp::kXFwd, fp32), v_yf = tuned_variant(c, clp::kYFwd, fp32),
                       v_yi = tuned_variant(c, clp::kYInv, fp32), v_xi = tuned_variant(c, clp::kXInv, fp32);
    const double gbytes = (double)grid_bytes;
    const double atoms = (double)n_at;
    const double live = skip_empty ? (double)c->live_rows / nrows : 1.0;
    const double row_side = (double)c->live_rows / nrows;
    const double h_bytes = sl.zw ? (sl.zb ? 12.0 : 4.0) * sizeof(T) * sl.pad[2] * nxy
                                 : (double)sl.table.nh * sl.pad[2] * nxy * sizeof(cx<T>);
    for (int p0 = 0; p0 < np; p0 += chunk) {
        const int cnt = std::min(chunk, np - p0);
        const cx<T>* rho_c = rho + (long long)p0 * rho_stride;
        cx<T>* out_c = via_tr ? tr : static_cast<cx<T>*>(V_any) + (long long)p0 * v_stride;
        cudaEvent_t e = prof_begin(c);
        if (qplane) {
            if (nx == ny)
                clp::pfwd<T>(c->stream, rho_c, rho_stride, row_ptr, c->row_mask.p, buf, vM, twx, nx, nz, cnt);
            else
                clp::pfwd_xy<T>(c->stream, rho_c, rho_stride, row_ptr, c->row_mask.p, buf, vM, twx, twy, nx, ny, nz, cnt);
        } else if (xy_fwd) {
            clp::xyfwd<T>(c->stream, rho_c, rho_stride, row_ptr, cell, buf, vM, twx, rp0, nx, ny, nz, cnt);
        } else if (!(reg_x && clp::xfwd<T>(c->stream, v_xf, rho_c, rho_stride, row_ptr, cell, buf, vM, twx, rp0, nx,
                                            ny, nrows, cnt, skip_empty))) {
            clk::k_xfwd<T><<<xblocks, 256, xt.smem, c->stream>>>(rho_c, rho_stride, row_ptr, cell, buf, vM,
                                                                 sl.ax[0].plan, twx, rp0, nx, ny, nrows, xt.rows,
                                                                 xt.ld, cnt);
        }
        CL_LAUNCHED();
        prof_end(c, e, CL_KCLASS_XFWD,
                 cnt * (atoms * (double)sizeof(cx<T>) + (xy_fwd || qplane ? 1.0 : live) * gbytes) + atoms * 4.0);
        if (!xy_fwd && !qplane) {
            e = prof_begin(c);
            if (!(reg_y && clp::ycol<-1, T>(c->stream, v_yf, buf, vM, twy, nx, ny, nz, cnt,
                                             skip_empty ? row_ptr : nullptr)))
                clk::k_ypass<-1, T><<<dim3(ychunks * nz, cnt), 256, yt.smem, c->stream>>>(buf, vM, sl.ax[1].plan, twy,
                                                                                          nx, ny, yt.W, ychunks);
            CL_LAUNCHED();
            prof_end(c, e, CL_KCLASS_YPASS, cnt * (1.0 + live) * gbytes);
        }
        e = prof_begin(c);
        bool mixed;
        if (sl.zw) {
            const auto* tab = reinterpret_cast<const clk::Quad<T>*>(sl.zw_tab.p);
            mixed = sl.zb ? clp::zw_zb<T>(c->stream, buf, vM, twz, tab, reinterpret_cast<const cx<T>*>(sl.zw_col.p),
                                          reinterpret_cast<const cx<T>*>(sl.zw_zph.p), nxy, sl.pad[2], cnt)
                          : clp::zw_pair<T>(c->stream, buf, vM, twz, tab, nxy, sl.pad[2], cnt);
        } else {
            mixed = clp::zmix<T>(c->stream, buf, vM, twz, H, phxy, phz, mix, sl.zb, nxy, sl.pad[2], cnt);
        }
        if (!mixed)
            cl::fail(CL_ERR_UNSUPPORTED, "no sub-lattice z pass for %d points", sl.pad[2]);
        CL_LAUNCHED();
        prof_end(c, e, CL_KCLASS_ZPASS, cnt * 2.0 * gbytes + h_bytes);
        if (!xy_inv && !qplane) {
            e = prof_begin(c);
            if (!(reg_y && clp::ycol<+1, T>(c->stream, v_yi, buf, vM, twy, nx, ny, nz, cnt,
                                             skip_empty ? row_ptr : nullptr)))
                clk::k_ypass<+1, T><<<dim3(ychunks * nz, cnt), 256, yt.smem, c->stream>>>(buf, vM, sl.ax[1].plan, twy,
                                                                                          nx, ny, yt.W, ychunks);
            CL_LAUNCHED();
            prof_end(c, e, CL_KCLASS_YPASS, cnt * (1.0 + live) * gbytes);
        }
        e = prof_begin(c);
        if (qplane) {
            if (nx == ny)
                clp::pinv<T>(c->stream, buf, vM, twx, row_ptr, c->row_mask.p, out_c, out_stride, nx, nz, cnt);
            else
                clp::pinv_xy<T>(c->stream, buf, vM, twx, twy, row_ptr, c->row_mask.p, out_c, out_stride, nx, ny, nz, cnt);
        } else if (xy_inv) {
            clp::xyinv<T>(c->stream, buf, vM, twx, row_ptr, cell, out_c, out_stride, nx, ny, nz, cnt);
        } else if (!(reg_x && clp::xinv<T>(c->stream, v_xi, buf, vM, twx, row_ptr, cell, out_c, out_stride, nx, nrows,
                                            cnt))) {
            clk::k_xinv<T><<<xblocks, 256, xt.smem, c->stream>>>(buf, vM, sl.ax[0].plan, twx, row_ptr, cell, out_c,
                                                                 out_stride, nx, nrows, xt.rows, xt.ld, cnt);
        }
        CL_LAUNCHED();
        prof_end(c, e, CL_KCLASS_XINV,
                 cnt * ((xy_inv || qplane ? 1.0 : row_side) * gbytes + atoms * (double)sizeof(cx<T>)) + atoms * 4.0);
        if (via_tr) {
            e = prof_begin(c);
            clk::k_sl_widen<T><<<dim3((unsigned)std::min<long long>((n_at + 255) / 256, 148LL * 8), cnt), 256, 0,
                                 c->stream>>>(tr, n_at, V + (long long)p0 * v_stride, v_stride, n_at);
            CL_LAUNCHED();
            prof_end(c, e, CL_KCLASS_ROUND_SUM, cnt * atoms * ((double)sizeof(cx<T>) + 16.0));
        }
    }
}

// The transforms of a request on the context's loaded atoms: the sub-lattice decomposition when
// it is in use, else the 8 rounds (of the rounds in round_mask).
// V is complex128 [np][v_stride], or complex64 when v32 (the FP32 sub-lattice form whose
// reductions read FP32 potentials, see v_fp32).
void run_transforms(cl_ctx* c, const void* rho, long long rho_stride, int np, void* V, long long v_stride, bool v32,
                    int round_mask = 0xFF) {
    if (c->sl.active) {
        if ((round_mask & 0xFF) != 0xFF)
            cl::fail(CL_ERR_UNSUPPORTED, "the sub-lattice form has no rounds to split (use an 8-round form)");
        if (fp64_form(c))
            run_sublattice<double>(c, static_cast<const cx<double>*>(rho), rho_stride, np, V, v_stride, false);
        else
            run_sublattice<float>(c, static_cast<const cx<float>*>(rho), rho_stride, np, V, v_stride, v32);
        return;
    }
    if (v32) cl::fail(CL_ERR_STATE, "the 8-round forms write FP64 potentials");
    run_rounds_mode(c, rho, rho_stride, np, c->row_ptr.p, c->cell_sorted.p, static_cast<cx<double>*>(V), v_stride,
                    round_mask);
}

// ---------------------------------------------------------------------------------------
// Tensor-core Gram (FP32 form): TF32 split pass + tcgen05 GEMM, see gram_tc.cuh.
// ---------------------------------------------------------------------------------------
bool use_tc_gram(const cl_ctx* c) { return !fp64_form(c) && !std::getenv("CL_NO_TC_GRAM"); }

// The FP32 sub-lattice form keeps the potentials at the atoms in FP32 (as the inverse passes
// produce them) when the tensor-core Gram reads them: its split rounds them to TF32 parts
// directly, with no FP64 copy in between.
bool v_fp32(const cl_ctx* c) { return c->sl.active && !fp64_form(c) && use_tc_gram(c); }
void* v_at(void* base, long long elems, bool v32) {
    return static_cast<unsigned char*>(base) + elems * (long long)(v32 ? sizeof(cx<float>) : sizeof(cx<double>));
}

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    if (!fn) cl::fail(CL_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    return fn;
}

// 3D FP32 tensor [2 parts][rows][k_pad] viewed in boxes of 32 atoms x box_rows rows x 1 part,
// 128-byte swizzle; rows of a box beyond `rows` are zero-filled by the copy (not read).
CUtensorMap tc_tensor_map(float* base, long long k_pad, long long rows, int box_rows) {
    CUtensorMap m;
    const cuuint64_t dims[3] = {(cuuint64_t)k_pad, (cuuint64_t)rows, 2};
    const cuuint64_t strides[2] = {(cuuint64_t)k_pad * sizeof(float), (cuuint64_t)(rows * k_pad) * sizeof(float)};
    const cuuint32_t box[3] = {(cuuint32_t)clk::tc::BK, (cuuint32_t)box_rows, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = tensor_map_encoder()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims, strides, box, estr,
                                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) cl::fail(CL_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return m;
}

struct TcShape {
    int rowsA = 0, rowsB = 0;        // real operand rows: re and im of each density
    long long chunk = 0, k_pad = 0;  // atoms per operand chunk, chunk rounded up to a k-tile
};

long long tc_bytes_per_atom(int rowsA, int rowsB) { return 2LL * (rowsA + rowsB) * (long long)sizeof(float); }

TcShape tc_shape(const cl_ctx* c, int nl, int nr, long long n_atoms) {
    TcShape s;
    s.rowsA = 2 * nl;
    s.rowsB = 2 * nr;
    const long long per_atom = tc_bytes_per_atom(s.rowsA, s.rowsB);
    const long long fit = (long long)(c->tc_buf.n * sizeof(float)) / per_atom / clk::tc::BK * clk::tc::BK;
    const long long full = (n_atoms + clk::tc::BK - 1) / clk::tc::BK * clk::tc::BK;
    s.k_pad = std::min(full, fit);
    s.chunk = std::min(n_atoms, s.k_pad);
    return s;
}

// Reductions of the FP32 forms over fewer than 65,536 atoms (CL_TC_MIN_ATOMS) are summed in
// FP64 (k_gram_dmma).  The TF32x3 Gram's error is ~2^-23 of each product, random in sign, so relative to
// the sum of the terms' magnitudes it falls as 1/sqrt(atoms): at 2M atoms it is far below the
// FP32 gate even where the terms cancel 1000:1, while on a box of a hundred atoms it can reach
// the 1e-9 eV floor on integrals that small.  Below the threshold the FP64 Gram costs little.
long long tc_min_atoms() {
    const char* e = std::getenv("CL_TC_MIN_ATOMS");
    return e ? std::atoll(e) : 65536LL;
}
bool small_gram(const cl_ctx* c, long long n_atoms) {
    return !fp64_form(c) && n_atoms < tc_min_atoms() && !std::getenv("CL_TC_FUSED") && !std::getenv("CL_TC_SPLIT");
}

// Pairs of densities a request reduces: the result is [nl][nr], its needed part a few blocks
// (gram_blocks.hpp), which can also be taken as one block.
struct GramPlan {
    int nl = 0, nr = 0;
    std::vector<clk::GramBlock> blocks;  // at most clk::kGramBlocks
    clk::GramBlock whole{};
};
GramPlan whole_gram(int nl, int nr, bool sym) {
    GramPlan g;
    g.nl = nl;
    g.nr = nr;
    g.whole = clk::GramBlock{0, nl, 0, nr, sym ? 1 : 0};
    g.blocks = {g.whole};
    return g;
}
// The plan's tiles of at most max_l x max_r densities: as separate blocks, or as one block where that
// gives fewer (a tensor-core tile costs nearly the same whatever it holds).
clk::GramTiles tc_tiles(const GramPlan& g, int max_l, int max_r) {
    const clk::GramTiles parts = clk::gram_tiles(g.blocks.data(), (int)g.blocks.size(), g.nr, max_l, max_r, 1);
    const clk::GramTiles one = clk::gram_tiles(&g.whole, 1, g.nr, max_l, max_r, 1);
    return clk::gram_tile_count(one) <= clk::gram_tile_count(parts) ? one : parts;
}

// How a request's reductions are computed.
enum class GramKind {
    kFp64,   // FP64 tensor cores (k_gram_dmma)
    kFused,  // TF32x3, operands split inside the kernel (k_gram_tc_ws)
    kSplit,  // TF32x3 after the split pass (k_tf32_split, k_gram_tc)
};
// One tile of at most 40 right densities holds the whole request: the fused Gram may sum k-tiles in pairs (see
// k_gram_tc_ws).
bool paired_gram(const GramPlan& g) { return g.nl <= clk::tc::BM / 2 && g.nr <= clk::tc::WS_MAX_NB8 / 2; }
// FP32 potentials and densities can take either TF32x3 Gram: the fused one splits the operands of its
// tile (at most 64 x 48 densities) itself, once per tile, the other reads split operands that a pass of
// their own writes.  Per k-tile of 32 atoms an SM takes 1.06 us for a fused tile that sums k-tiles in pairs, 1.25 us
// for one that does not and 1.10 us for a 64 x 64 tile after the split, whose pass costs 0.0167 us a density
// (110,592 atoms, all pairs of 16 states: 0.213 ms fused, 0.180 + 0.126 split; of 20: 0.464, 0.294 + 0.187; of 24:
// 0.785, 0.433 + 0.261).  CL_TC_SPLIT=1 keeps the split pass everywhere; CL_TC_FUSED=1 takes the fused Gram at
// any tile count.
GramKind gram_kind(const cl_ctx* c, const GramPlan& g, bool v_f32, bool rho_f32, long long n_atoms) {
    if (!use_tc_gram(c) || small_gram(c, n_atoms)) return GramKind::kFp64;
    if (!v_f32 || !rho_f32 || std::getenv("CL_TC_SPLIT")) return GramKind::kSplit;
    if (std::getenv("CL_TC_FUSED")) return GramKind::kFused;
    const double fused = (paired_gram(g) ? 1.06 : 1.25) *
                         clk::gram_tile_count(tc_tiles(g, clk::tc::BM / 2, clk::tc::WS_MAX_NB / 2));
    const double split = 1.10 * clk::gram_tile_count(tc_tiles(g, clk::tc::BM / 2, clk::tc::BN / 2)) +
                         0.0167 * (g.nl + g.nr);
    return fused <= split ? GramKind::kFused : GramKind::kSplit;
}

// Operand buffer of the split pass: whole atom range when it fits in a quarter of the free
// device memory (at most 8 GiB), else chunks of the atom range.  Called outside any capture.
void tc_reserve(cl_ctx* c, const GramPlan& g, long long n_atoms, bool v_f32, bool rho_f32) {
    if (g.nl <= 0 || g.nr <= 0 || n_atoms <= 0 || gram_kind(c, g, v_f32, rho_f32, n_atoms) != GramKind::kSplit) return;
    const int rowsA = 2 * g.nl, rowsB = 2 * g.nr;
    const long long per_atom = tc_bytes_per_atom(rowsA, rowsB);
    const long long full = (n_atoms + clk::tc::BK - 1) / clk::tc::BK * clk::tc::BK;
    const long long have = (long long)(c->tc_buf.n * sizeof(float)) / per_atom;
    if (have >= full) return;
    const long long budget = std::min<long long>(8LL << 30, (long long)(free_device_bytes() / 4));
    long long atoms = std::min(full, std::max<long long>(budget / per_atom, 64LL * clk::tc::BK));
    if (const char* e = std::getenv("CL_TC_MAX_ATOMS"))  // cap per chunk (exercises the chunked path)
        atoms = std::min(atoms, std::max<long long>(clk::tc::BK, std::atoll(e)));
    atoms = atoms / clk::tc::BK * clk::tc::BK;
    if (atoms <= have) return;
    c->tc_buf.alloc((size_t)(atoms * per_atom / (long long)sizeof(float)));
}

// Atom splits of a Gram launch: whole waves of 148 blocks, each split at least 16 k-tiles long.
int gram_splits(int tiles, int kt_total) {
    int best_s = 1;
    double best = -1e30;
    const int s_max = std::max(1, std::min(256, kt_total / 16));
    for (int s = 1; s <= s_max; ++s) {
        const int per = (kt_total + s - 1) / s;
        const int used = (kt_total + per - 1) / per;
        const long long items = (long long)tiles * used;
        const long long waves = (items + 147) / 148;
        const double score = (double)items / (double)(waves * 148) - 0.01 * (double)waves;
        if (score > best) {
            best = score;
            best_s = used;
        }
    }
    return best_s;
}

// Register tile (A x B MMA tiles a warp) and warp grid of an FP64 Gram over C tiles of ta x tb MMA tiles:
// the least work of a warp per k-step -- 16 cycles of its FP64 pipe an MMA, about 5 a fragment -- times
// the warps that share it.
struct DmmaShape {
    int reg = 0, wr = 1, wc = 1;
    double cost = 1e300;
};
constexpr int kDmmaReg[8][2] = {{1, 1}, {2, 2}, {3, 3}, {4, 4}, {5, 5}, {6, 6}, {7, 4}, {8, 4}};
DmmaShape dmma_shape(int ta, int tb) {
    DmmaShape best;
    for (int wr = 1; wr <= clk::dm::WARPS; wr *= 2)
        for (int wc = 1; wr * wc <= clk::dm::WARPS; wc *= 2)
            for (int r = 0; r < 8; ++r) {
                const int A = kDmmaReg[r][0], B = kDmmaReg[r][1];
                if (wr * A < ta || wc * B < tb) continue;
                const double t = (16.0 * A * B + 5.0 * (A + B)) * wr * wc;
                if (t < best.cost) best = DmmaShape{r, wr, wc, t};
            }
    return best;
}

// The FP64 tensor-core Gram over the whole atom range (see k_gram_dmma).  Tile sides of at most 24, 48
// or 64 densities, whichever takes the fewest MMAs over all tiles (smaller ones follow a symmetric
// block's diagonal closer), in whole 8-row tiles of the MMA.
template <typename SV, typename SR>
void gram_dmma(cl_ctx* c, const cx<SV>* V, long long v_stride, const cx<SR>* rho, long long r_stride,
               const int* rows_dev, const GramPlan& plan, long long n_atoms, double* out4_dev) {
    using namespace clk::dm;
    GramArgs<SV> g{};
    g.V = V;
    g.v_stride = v_stride;
    g.lidx = rows_dev;
    g.ridx = rows_dev ? rows_dev + plan.nl : nullptr;
    g.r_stride = r_stride;
    g.na = n_atoms;
    g.out4 = out4_dev;
    DmmaShape shape;
    for (int width : {WIDTH, 48, 24}) {
        const clk::GramTiles t = clk::gram_tiles(plan.blocks.data(), (int)plan.blocks.size(), plan.nr, width, width, 4);
        int a = 0, b = 0;
        for (int k = 0; k < t.n; ++k) {
            a = std::max(a, t.wl[k]);
            b = std::max(b, t.wr[k]);
        }
        DmmaShape sh = dmma_shape(a / 4, b / 4);
        sh.cost *= clk::gram_tile_count(t);
        if (sh.cost < 0.9 * shape.cost) {
            shape = sh;
            g.tiles = t;
            g.nd_a = a;
            g.nd_b = b;
        }
    }
    g.wr = shape.wr;
    g.wc = shape.wc;
    g.align_v = reinterpret_cast<uintptr_t>(V) % 16 == 0 && v_stride * sizeof(cx<SV>) % 16 == 0;
    g.align_r = reinterpret_cast<uintptr_t>(rho) % 16 == 0 && r_stride * sizeof(cx<SR>) % 16 == 0;
    const int tiles = clk::gram_tile_count(g.tiles);
    const int kc = g.wr * g.wc == 1 && n_atoms / 64 * tiles >= 148 * 4 ? 64 : 32;
    const int chunks = (int)std::min<long long>((n_atoms + kc - 1) / kc, 1LL << 30);
    // small boxes: enough atom splits to occupy the SMs in one wave (at least 2 chunks a block)
    const int splits0 = std::max(1, std::max(gram_splits(tiles, chunks), std::min(chunks / 2, 148 / tiles)));
    const long long per_chunks = (chunks + splits0 - 1) / splits0;
    g.atoms_per_split = per_chunks * kc;
    const int splits = (int)((n_atoms + g.atoms_per_split - 1) / g.atoms_per_split);
    const size_t stage = stage_bytes<SV, SR>(kc, g.nd_a, g.nd_b);
    g.stages = 4 * stage <= 220 * 1024 ? 4 : 3 * stage <= 224 * 1024 ? 3 : 2;
    const size_t smem = std::max(g.stages * stage, reduce_bytes(kDmmaReg[shape.reg][0], kDmmaReg[shape.reg][1],
                                                                 WARPS / (g.wr * g.wc)));
    cudaEvent_t e = prof_begin(c);
    const dim3 grid(tiles, splits);
    const auto launch = [&](auto kern) {
        ensure_smem(kern, 226 * 1024, 226 * 1024);  // beside 512 bytes of static shared memory
        kern<<<grid, THREADS, smem, c->stream>>>(rho, g);
    };
    const auto square = [&](auto k) {
        constexpr int KC = decltype(k)::value;
        switch (shape.reg) {
            case 0: launch(k_gram_dmma<SV, SR, KC, 1, 1>); break;
            case 1: launch(k_gram_dmma<SV, SR, KC, 2, 2>); break;
            case 2: launch(k_gram_dmma<SV, SR, KC, 3, 3>); break;
            case 3: launch(k_gram_dmma<SV, SR, KC, 4, 4>); break;
            case 4: launch(k_gram_dmma<SV, SR, KC, 5, 5>); break;
            default: launch(k_gram_dmma<SV, SR, KC, 6, 6>); break;
        }
    };
    if (shape.reg == 6)
        launch(k_gram_dmma<SV, SR, 32, 7, 4>);
    else if (shape.reg == 7)
        launch(k_gram_dmma<SV, SR, 32, 8, 4>);
    else if (kc == 64)
        square(std::integral_constant<int, 64>{});
    else
        square(std::integral_constant<int, 32>{});
    CL_LAUNCHED();
    prof_end(c, e, CL_KCLASS_GRAM,
             (double)n_atoms * (plan.nl * (double)sizeof(cx<SV>) + plan.nr * (double)sizeof(cx<SR>)));
}

// The fused Gram on FP32 operands over the whole atom range (see k_gram_tc_ws).
void gram_tc_fused(cl_ctx* c, const cx<float>* V, long long v_stride, const cx<float>* rho, long long r_stride,
                   const int* rows_dev, const GramPlan& plan, long long n_atoms, double* out4_dev) {
    using namespace clk::tc;
    // up to 48 right densities a tile, with 8 drain warps up to 40 (96^3, blocks of 42 and 36 densities: two tiles of
    // 48 0.077 ms; with k-tiles summed in pairs they took 0.070, three tiles of 40 0.087)
    FusedGram g{};
    g.tiles = tc_tiles(plan, BM / 2, WS_MAX_NB8 / 2);
    const clk::GramTiles wider = tc_tiles(plan, BM / 2, WS_MAX_NB / 2);
    const bool wide = clk::gram_tile_count(wider) < clk::gram_tile_count(g.tiles);
    if (wide) g.tiles = wider;
    int nA = 1, nB = 1;
    for (int b = 0; b < g.tiles.n; ++b) {
        nA = std::max(nA, std::min(g.tiles.wl[b], g.tiles.b[b].nl));
        nB = std::max(nB, std::min(g.tiles.wr[b], g.tiles.b[b].nr));
    }
    const int nb = std::max(16, (2 * nB + 15) / 16 * 16);
    g.V = reinterpret_cast<const float2*>(V);
    g.v_stride = v_stride;
    g.rho = reinterpret_cast<const float2*>(rho);
    g.r_stride = r_stride;
    g.lidx = rows_dev;
    g.ridx = rows_dev ? rows_dev + plan.nl : nullptr;
    g.na = n_atoms;
    g.out4 = out4_dev;
    g.err = out4_dev + (size_t)4 * plan.nl * plan.nr;
    g.kt_total = (int)((n_atoms + BK - 1) / BK);
    g.stage_bytes = (uint32_t)(2 * BM * 128 + 2 * nb * 128);
    g.raw_slot_bytes = (uint32_t)((nA + nB) * BK * 8);
    // CL_TC_COPY8=1: 8-byte copies even where the rows allow 16 (zinc-blende boxes always do)
    g.aligned16 = (reinterpret_cast<uintptr_t>(V) % 16 == 0 && reinterpret_cast<uintptr_t>(rho) % 16 == 0 &&
                   v_stride % 2 == 0 && r_stride % 2 == 0 && !std::getenv("CL_TC_COPY8"))
                      ? 1
                      : 0;
    const int tiles = clk::gram_tile_count(g.tiles);
    const int splits0 = gram_splits(tiles, g.kt_total);
    g.kt_per = (g.kt_total + splits0 - 1) / splits0;
    const int splits = (g.kt_total + g.kt_per - 1) / g.kt_per;
    // the deepest copy ring that fits: 5 k-tiles ahead (6 slots) at the 2.1M-atom box's 72 densities
    const size_t smem5 = ws_smem_bytes(g.stage_bytes, g.raw_slot_bytes, 5);
    const size_t smem3 = ws_smem_bytes(g.stage_bytes, g.raw_slot_bytes, 3);
    const size_t smem2 = ws_smem_bytes(g.stage_bytes, g.raw_slot_bytes, 2);
    if (smem2 > 227 * 1024) cl::fail(CL_ERR_UNSUPPORTED, "fused Gram needs %zu bytes of shared memory", smem2);
    cudaEvent_t e = prof_begin(c);
    const dim3 grid(tiles, splits);
    // k-tiles leave the tensor cores in pairs summed in FP32 only for requests in one tile of up to 40 right
    // densities (36 a side over 2.1M atoms: 0.47 ms); every k-tile of the others, with CL_TC_NO_WS=1 of all, goes
    // to FP64 by itself
    const bool pairs = paired_gram(plan) && !std::getenv("CL_TC_NO_WS");
    const auto launch_ws = [&](auto ahead, size_t smem) {
        constexpr int AHEAD = decltype(ahead)::value;
        const auto go = [&](auto kern, int threads) {
            ensure_smem(kern, 227 * 1024);
            kern<<<grid, threads, smem, c->stream>>>(g);
        };
        if (wide)
            go(k_gram_tc_ws<AHEAD, 12, false>, ws_threads(12));
        else if (pairs)
            go(k_gram_tc_ws<AHEAD, 8, true>, ws_threads(8));
        else
            go(k_gram_tc_ws<AHEAD, 8, false>, ws_threads(8));
    };
    if (smem5 <= 227 * 1024)
        launch_ws(std::integral_constant<int, 5>{}, smem5);
    else if (smem3 <= 227 * 1024)
        launch_ws(std::integral_constant<int, 3>{}, smem3);
    else
        launch_ws(std::integral_constant<int, 2>{}, smem2);
    CL_LAUNCHED();
    prof_end(c, e, CL_KCLASS_GRAM, (double)n_atoms * (plan.nl + plan.nr) * (double)sizeof(cx<float>));
}

// The split pass and the TF32x3 Gram on its operands, in chunks of the atom range.
void gram_tc_split(cl_ctx* c, const void* V, bool v_f32, long long v_stride, const void* rho, bool rho_f32,
                   long long r_stride, const int* rows_dev, const GramPlan& plan, long long n_atoms, double* out4_dev) {
    using namespace clk::tc;
    const int nl = plan.nl, nr = plan.nr;
    const TcShape sh = tc_shape(c, nl, nr, n_atoms);
    if (sh.k_pad < BK) cl::fail(CL_ERR_STATE, "tensor-core Gram operands not reserved");
    ensure_smem(clk::tc::k_gram_tc, SMEM_BYTES);
    float* A = c->tc_buf.p;
    float* B = A + 2LL * sh.rowsA * sh.k_pad;
    const CUtensorMap mapA = tc_tensor_map(A, sh.k_pad, sh.rowsA, BM);
    const CUtensorMap mapB = tc_tensor_map(B, sh.k_pad, sh.rowsB, BN);
    const clk::GramTiles gt = tc_tiles(plan, BM / 2, BN / 2);
    const int tiles = clk::gram_tile_count(gt);
    for (long long a0 = 0; a0 < n_atoms; a0 += sh.chunk) {
        const long long na = std::min(sh.chunk, n_atoms - a0);
        const long long kp = (na + BK - 1) / BK * BK;  // k-tiles that hold atoms of this chunk
        const int kt_total = (int)(kp / BK);
        cudaEvent_t e0 = prof_begin(c);
        const int xblocks = (int)std::min<long long>((kp + 255) / 256, 64);
        if (v_f32)
            clk::tc::k_tf32_split<float><<<dim3(xblocks, nl), 256, 0, c->stream>>>(
                static_cast<const cx<float>*>(V), v_stride, rows_dev, nl, a0, na, sh.k_pad, A);
        else
            clk::tc::k_tf32_split<double><<<dim3(xblocks, nl), 256, 0, c->stream>>>(
                static_cast<const cx<double>*>(V), v_stride, rows_dev, nl, a0, na, sh.k_pad, A);
        CL_LAUNCHED();
        if (rho_f32)
            clk::tc::k_tf32_split<float><<<dim3(xblocks, nr), 256, 0, c->stream>>>(
                static_cast<const cx<float>*>(rho), r_stride, rows_dev ? rows_dev + nl : nullptr, nr, a0, na, sh.k_pad, B);
        else
            clk::tc::k_tf32_split<double><<<dim3(xblocks, nr), 256, 0, c->stream>>>(
                static_cast<const cx<double>*>(rho), r_stride, rows_dev ? rows_dev + nl : nullptr, nr, a0, na, sh.k_pad, B);
        CL_LAUNCHED();
        prof_end(c, e0, CL_KCLASS_GRAM_SPLIT,
                 (double)na * (nl * (v_f32 ? 8.0 : 16.0) + nr * (rho_f32 ? 8.0 : 16.0)) +
                     (double)tc_bytes_per_atom(sh.rowsA, sh.rowsB) * kp);
        const int best_s = gram_splits(tiles, kt_total);
        const int kt_per = (kt_total + best_s - 1) / best_s;
        const int splits = (kt_total + kt_per - 1) / kt_per;
        cudaEvent_t e1 = prof_begin(c);
        clk::tc::k_gram_tc<<<dim3(tiles, splits), THREADS, SMEM_BYTES, c->stream>>>(
            mapA, mapB, kt_total, kt_per, gt, out4_dev, out4_dev + (size_t)4 * nl * nr);
        CL_LAUNCHED();
        prof_end(c, e1, CL_KCLASS_GRAM, (double)tc_bytes_per_atom(sh.rowsA, sh.rowsB) * kp);
    }
}

// Error slot after the 4 * nl * nr results: non-zero when a device-side wait gave up.
void check_gram_slot(double slot) {
    if (slot != 0.0) cl::fail(CL_ERR_TIMEOUT, "tensor-core Gram: a device-side wait timed out");
}

// out4[l][r] = {sum ac, bd, ad, bc} over atoms for the pairs of the plan's blocks; out4 holds
// 4 * nl * nr + 1 doubles, the last one an error slot.  rows_dev: the nl rows of V, then the nr rows of rho
// (null: row l, row r).  rho: the right densities, complex64 when rho_f32
// (the FP32 form's pair densities), else complex128 (the plain form's, and the grid API's caller-given
// density).
void gram(cl_ctx* c, const void* V_any, bool v_f32, long long v_stride, const void* rho_any, bool rho_f32,
          long long r_stride, const int* rows_dev, const GramPlan& plan, long long n_atoms, double* out4_dev) {
    CL_CUDA(cudaMemsetAsync(out4_dev, 0, sizeof(double) * (4 * (size_t)plan.nl * plan.nr + 1), c->stream));
    const auto* v32 = static_cast<const cx<float>*>(V_any);
    const auto* v64 = static_cast<const cx<double>*>(V_any);
    const auto* r32 = static_cast<const cx<float>*>(rho_any);
    const auto* r64 = static_cast<const cx<double>*>(rho_any);
    switch (gram_kind(c, plan, v_f32, rho_f32, n_atoms)) {
        case GramKind::kFused:
            if (!v_f32 || !rho_f32) cl::fail(CL_ERR_STATE, "the fused Gram needs FP32 operands");
            gram_tc_fused(c, v32, v_stride, r32, r_stride, rows_dev, plan, n_atoms, out4_dev);
            break;
        case GramKind::kSplit:
            gram_tc_split(c, V_any, v_f32, v_stride, rho_any, rho_f32, r_stride, rows_dev, plan, n_atoms, out4_dev);
            break;
        case GramKind::kFp64:
            if (v_f32 && rho_f32)
                gram_dmma(c, v32, v_stride, r32, r_stride, rows_dev, plan, n_atoms, out4_dev);
            else if (v_f32)
                cl::fail(CL_ERR_STATE, "FP32 potentials go with FP32 densities");
            else if (rho_f32)
                gram_dmma(c, v64, v_stride, r32, r_stride, rows_dev, plan, n_atoms, out4_dev);
            else
                gram_dmma(c, v64, v_stride, r64, r_stride, rows_dev, plan, n_atoms, out4_dev);
            break;
    }
}

// Pair densities rho[p][atom] for products (fl[p], fr[p]) (0-based state indices): the
// device lists and launch shape are set up once (setup synchronises), the launch itself only
// enqueues (it can be captured in a CUDA graph).
}  // namespace
struct PairSetup {
    DevBuf<clk::PairSeg> segs;  // products grouped by left state, indices into `states` (FP64 kernel)
    // FP64 tensor cores (at most 40 used states, see k_pair_mma)
    bool mma_ok = false, mma_sliced = false;
    clk::pm::PairMmaArgs mma{};
    DevBuf<int> mma_prod;
    int mma_grid = 1;  // thread blocks
    size_t mma_smem = 0;
    // tiles of 4 x 4 states (see k_pair_density_tile)
    bool tile_ok = false;
    DevBuf<int> tile_states, tiles, tile_prod;
    int ns_pad = 0, n_tiles = 0, tile_atoms = 0, tile_threads = 0, tile_blocks = 0;
    size_t tile_smem = 0;
    DevBuf<int> states;
    int np = 0, n_segs = 0, n_used = 0, chunk = 1, blocks = 1;
    size_t smem = 0;
};
namespace {

// Tables of the 4 x 4-state tile kernel: used states ascending, padded to a multiple of 4
// (-1: zero rows); the requested tiles (bi | bj << 16, bi >= bj); and per ordered state pair
// (i >= j) the density row 2p (rho_p = conj(c_i) c_j) or 2p + 1 (rho_p = conj(c_j) c_i).  The
// atoms a block stages (A) are the most, of 64, 32, 16, 8, whose coefficients fit 110 KB (two
// blocks an SM), else 8 atoms in up to 227 KB; beyond that, or when two products name the same
// pair of states both ways, the segment kernel runs instead (as it does with CL_NO_PAIR_TILE=1).
void pair_tile_setup(cl_ctx* c, const std::vector<int2>& fl, const std::vector<int>& used,
                     const std::vector<int>& where, PairSetup& ps) {
    const int n = (int)used.size();
    std::vector<int> order(n);
    std::iota(order.begin(), order.end(), 0);
    std::sort(order.begin(), order.end(), [&](int a, int b) { return used[a] < used[b]; });
    std::vector<int> pos(n);
    const int ns_pad = (n + clk::kPairTile - 1) / clk::kPairTile * clk::kPairTile;
    std::vector<int> st(ns_pad, -1);
    for (int k = 0; k < n; ++k) {
        pos[order[k]] = k;
        st[k] = used[order[k]];
    }
    std::vector<int> prod((size_t)ns_pad * ns_pad, -1);
    const int nblk = ns_pad / clk::kPairTile;
    std::vector<char> want((size_t)nblk * nblk, 0);
    for (int p = 0; p < ps.np; ++p) {
        int i = pos[where[fl[p].x]], j = pos[where[fl[p].y]];
        int code = 2 * p;
        if (i < j) {
            std::swap(i, j);
            code += 1;
        }
        int& slot = prod[(size_t)i * ns_pad + j];
        if (slot >= 0) return;  // the same pair both ways: the segment kernel
        slot = code;
        want[(size_t)(i / clk::kPairTile) * nblk + j / clk::kPairTile] = 1;
    }
    std::vector<int> tiles;
    for (int bi = 0; bi < nblk; ++bi)
        for (int bj = 0; bj <= bi; ++bj)
            if (want[(size_t)bi * nblk + bj]) tiles.push_back(bi | (bj << 16));
    const size_t per_atom = sizeof(cx<double>) * (size_t)ns_pad * (size_t)(c->n_orb | 1);
    int A = 0;
    for (int cand : {64, 32, 16, 8})
        if (per_atom * cand <= 110 * 1024) {
            A = cand;
            break;
        }
    if (A == 0 && per_atom * 8 <= 227 * 1024) A = 8;
    if (A == 0) return;
    ps.tile_ok = true;
    ps.ns_pad = ns_pad;
    ps.n_tiles = (int)tiles.size();
    ps.tile_atoms = A;
    ps.tile_smem = per_atom * A;
    ps.tile_threads = (int)std::min<long long>(256, ((long long)ps.n_tiles * A + 31) / 32 * 32);
    ps.tile_blocks = (int)std::max<long long>(1, std::min<long long>((c->n_sorted + A - 1) / A, 148LL * 8));
    ps.tile_states.upload(st.data(), st.size(), c->stream);
    ps.tiles.upload(tiles.data(), tiles.size(), c->stream);
    ps.tile_prod.upload(prod.data(), prod.size(), c->stream);
}

// f(NB, PACKED, FOLD, SLICED) as integral constants for n states: FOLD from 16 orbitals on, where the products
// it leaves out outweigh its shuffles (20 states, 10 orbitals: 0.31 ms without, 0.33 with; 20 orbitals:
// 0.57 and 0.56; 12 states: 0.139 and 0.126), of 5 to 8 states from 10 on (5 states, 8 orbitals: 0.031 and 0.032; 10
// orbitals: 0.039 and 0.038); orbitals in slices come in at more than that.
template <typename F>
void with_pair_mma(int n, int n_orb, bool sliced, F&& f) {
    const auto blocks = [&](auto fold, auto cut) {
        const std::false_type whole{};
        switch ((n + 7) / 8) {
            case 1:
                if (n <= 4)
                    f(std::integral_constant<int, 1>{}, std::true_type{}, fold, cut);
                else
                    f(std::integral_constant<int, 1>{}, whole, fold, cut);
                break;
            case 2: f(std::integral_constant<int, 2>{}, whole, fold, cut); break;
            case 3: f(std::integral_constant<int, 3>{}, whole, fold, cut); break;
            case 4: f(std::integral_constant<int, 4>{}, whole, fold, cut); break;
            default: f(std::integral_constant<int, 5>{}, whole, fold, cut); break;
        }
    };
    if (sliced)
        blocks(std::true_type{}, std::true_type{});
    else if (n_orb >= (n > 4 && n <= 8 ? 10 : 16))
        blocks(std::true_type{}, std::false_type{});
    else
        blocks(std::false_type{}, std::false_type{});
}

// Whether np products of n states with t4 of their 4 x 4 tiles named go to the tile kernel, which forms those tiles
// alone and takes orbitals one by one; the tensor-core kernel forms every 8 x 8 tile over steps of 4 orbitals.  Of 1
// orbital from 9 states on it does (32,768 atoms, FP32: 9 states 0.020 ms on the tensor cores, 0.017 in tiles; 20 states
// 0.033 and 0.028), beyond 10 orbitals or up to 16 states it does not (12 orbitals, 40 potentials: 0.137 and 0.163; 16
// states of 5 orbitals, all products: 0.030 and 0.042).  Between them the two costs decide, us at 32,768 atoms fitted to
// 17 to 40 states, 2 to 10 orbitals, and products from potentials to all (the choice costs 0.4 % on average, at most 15 %):
// the tile kernel's coefficients, tiles and products; the tensor-core kernel's steps, by its blocks, and products.
// Measured, 5 orbitals: FP32 potentials of 24 states 0.043 ms on the tensor cores and 0.039, of 40 0.092 and 0.059; all
// products of 24, 0.052 and 0.067, of 40, 0.134 and 0.138; FP64 of 40, 0.183 and 0.153.
bool pair_tiles_faster(int n, int n_orb, int np, int t4, bool fp64) {
    const int nb = (n + 7) / 8;
    if (n_orb == 1) return n > 8;
    if (nb <= 2 || n_orb > (nb == 3 ? 8 : 10)) return false;
    const int pad = (n + 3) / 4 * 4;
    const double tiles = 4 + 0.25 * pad + n_orb * (0.185 * pad + 0.2 * t4) + np * (fp64 ? 0.05 : 0.035);
    static const double steps[3][3] = {{32, 43, 56}, {58, 76, 108}, {69, 93, 138}};
    const double product = nb == 3 ? (fp64 ? 0.02 : 0.01) : (fp64 ? 0.08 : 0.04);
    return tiles < 0.97 * (steps[nb - 3][(n_orb + 3) / 4 - 1] + np * product);
}

// Tables and launch shape of the tensor-core kernel: used states ascending, the density row of each
// product (i, j), i >= j in that order (rows are conj(c_x) c_y, x >= y).  Batches hold about 160 values a
// state of 8 states, more of fewer (1,280 in all), in powers of two from one tile a warp group up, while enough blocks
// share an SM and the atoms make a batch for each (12 states, 1 orbital, FP64: 64 atoms, one block an SM, 0.066 ms,
// 32 atoms 0.051, 16 atoms 0.050; 2 states, 5 orbitals: 32 atoms 0.016, 128 0.014) -- more where one block an SM runs
// anyway (30 states: 8 atoms 0.53 ms, 4 atoms 0.60) -- two of them in shared memory; when even the smallest does not
// fit beside the products (many orbitals), it comes in slices of orbitals, as many as let those blocks fit.
void pair_mma_setup(cl_ctx* c, const std::vector<int2>& fl, const std::vector<int>& used,
                    const std::vector<int>& where, PairSetup& ps) {
    using namespace clk::pm;
    const int n = (int)used.size(), nb = (n + 7) / 8;
    if (n == 0 || nb > MAX_BLOCKS || ps.np > 32767) return;
    std::vector<int> order(n), pos(n);
    std::iota(order.begin(), order.end(), 0);
    std::sort(order.begin(), order.end(), [&](int x, int y) { return used[x] < used[y]; });
    for (int k = 0; k < n; ++k) pos[order[k]] = k;
    std::vector<int> prod((size_t)64 * nb * nb, -1);
    std::array<std::array<bool, 2 * MAX_BLOCKS>, 2 * MAX_BLOCKS> named{};  // tiles of 4 x 4 states
    int t4 = 0;
    for (int p = 0; p < ps.np; ++p) {
        const int i = pos[where[fl[p].x]], j = pos[where[fl[p].y]];
        if (i < j) cl::fail(CL_ERR_STATE, "pair density with its lower state first");
        int& row = prod[(size_t)i * 8 * nb + j];
        if (row >= 0) return;  // the same product twice: the kernels with a row per product
        row = p;
        t4 += !named[i / 4][j / 4];
        named[i / 4][j / 4] = true;
    }
    if (pair_tiles_faster(n, c->n_orb, ps.np, t4, fp64_form(c)) && !std::getenv("CL_NO_PAIR_TILE")) return;
    PairMmaArgs& g = ps.mma;
    g = PairMmaArgs{};
    g.n_orb = c->n_orb;
    g.n = c->n_sorted;
    g.np = ps.np;
    g.n_used = n;
    // rows of a tile an atom takes: of up to 4 states, several atoms share a tile
    g.rows_log2 = n == 1 ? 0 : n == 2 ? 1 : n <= 4 ? 2 : 3;
    const auto bytes = [&](int at, int orbitals) {
        const int pitch = state_pitch(at, orbitals);
        return fp64_form(c) ? pair_mma_smem<double>(nb, n, pitch, ps.np, at)
                            : pair_mma_smem<float>(nb, n, pitch, ps.np, at);
    };
    const size_t most = 227 * 1024, share = 228 * 1024 / min_blocks(nb) - 1024;  // a block's, of those an SM is to hold
    // batches may grow until one block fewer than that fits, but not below two
    const size_t room = min_blocks(nb) == 1 ? most : 228 * 1024 / std::max(2, min_blocks(nb) - 1) - 1024;
    int at = warps(nb) / warps_per_atom(nb) * (8 >> g.rows_log2), staged = c->n_orb;
    const bool sliced = bytes(at, staged) > most;
    if (sliced) {
        g.slice_log2 = 5;
        while (g.slice_log2 > 3 && bytes(at, 1 << g.slice_log2) > share) --g.slice_log2;
        staged = 1 << g.slice_log2;
        if (bytes(at, staged) > most) return;
    } else {
        const auto larger = [&] {
            const bool few = std::min(n, 8) * 2 * at * staged <= 1280 && c->n_sorted >= 2LL * at * 148 * min_blocks(nb);
            return at < 256 && (few || (min_blocks(nb) == 1 && at < 16)) && bytes(2 * at, staged) <= room;
        };
        while (larger()) at *= 2;
    }
    g.at = at;
    while ((1 << g.at_log2) < at) ++g.at_log2;
    g.state_pitch = state_pitch(at, staged);
    for (int k = 0; k < n; ++k) g.state[k] = used[order[k]];
    ps.mma_prod.upload(prod.data(), prod.size(), c->stream);
    ps.mma_ok = true;
    ps.mma_sliced = sliced;
    ps.mma_smem = bytes(at, staged);
    const long long batches = (g.n + at - 1) / at;
    int resident = 1;
    with_pair_mma(n, c->n_orb, sliced, [&](auto k, auto pack, auto fold, auto cut) {
        constexpr int NB = decltype(k)::value;
        constexpr bool PACKED = decltype(pack)::value, FOLD = decltype(fold)::value, SLICED = decltype(cut)::value;
        const auto count = [&](auto kern) {
            ensure_smem(kern, most);
            CL_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kern, 32 * warps(NB), ps.mma_smem));
        };
        if (fp64_form(c))
            count(k_pair_mma<NB, PACKED, FOLD, SLICED, double>);
        else
            count(k_pair_mma<NB, PACKED, FOLD, SLICED, float>);
    });
    ps.mma_grid = (int)std::max<long long>(1, std::min<long long>(batches, 148LL * std::max(1, resident)));
}

void pair_setup(cl_ctx* c, const std::vector<int2>& fl, PairSetup& ps) {
    ps.np = (int)fl.size();
    std::vector<int> used;
    std::vector<int> where(c->n_states, -1);
    for (const auto& f : fl)
        for (int s : {f.x, f.y})
            if (where[s] < 0) { where[s] = (int)used.size(); used.push_back(s); }
    // segments: the products of each left state, kPairSeg at a time (product order kept)
    std::vector<std::vector<int>> by_left(used.size());
    for (int p = 0; p < ps.np; ++p) by_left[where[fl[p].x]].push_back(p);
    std::vector<clk::PairSeg> segs;
    for (int u = 0; u < (int)used.size(); ++u)
        for (size_t k0 = 0; k0 < by_left[u].size(); k0 += clk::kPairSeg) {
            clk::PairSeg sg{};
            sg.left = u;
            sg.cnt = (int)std::min<size_t>(clk::kPairSeg, by_left[u].size() - k0);
            for (int j = 0; j < sg.cnt; ++j) {
                const int p = by_left[u][k0 + j];
                sg.right[j] = where[fl[p].y];
                sg.prod[j] = p;
            }
            segs.push_back(sg);
        }
    ps.n_segs = (int)segs.size();
    ps.segs.upload(segs.data(), segs.size(), c->stream);
    // CL_NO_PAIR_REG12=1: the 4 x 4-state tile kernel instead of the tensor cores; CL_NO_PAIR_TILE=1 with it:
    // the segment kernel
    if (!std::getenv("CL_NO_PAIR_REG12")) pair_mma_setup(c, fl, used, where, ps);
    if (!ps.mma_ok && !used.empty() && !std::getenv("CL_NO_PAIR_TILE")) pair_tile_setup(c, fl, used, where, ps);
    ps.states.upload(used.data(), used.size(), c->stream);
    ps.n_used = (int)used.size();
    // two stages of `chunk` atoms, each up to 48 KB (about two blocks per SM)
    const int os = c->n_orb | 1;
    const size_t per_atom = sizeof(cx<double>) * (size_t)used.size() * os;
    // the chunk (at most the 48 KB stage) whose item rounds -- segments x atoms over the 256
    // threads of a block -- cost least per atom
    const int max_chunk = (int)std::max<size_t>(1, std::min<size_t>(64, (48 * 1024) / per_atom));
    ps.chunk = max_chunk;
    double best = 1e300;
    for (int ch = max_chunk; ch >= std::max(1, max_chunk / 2); --ch) {
        const double rounds = (double)(((long long)ps.n_segs * ch + 255) / 256);
        if (rounds / ch < best - 1e-12) {
            best = rounds / ch;
            ps.chunk = ch;
        }
    }
    ps.smem = 2 * per_atom * ps.chunk;
    ensure_smem(clk::k_pair_density<double>, ps.smem);
    ensure_smem(clk::k_pair_density<float>, ps.smem);
    const long long chunks = (c->n_sorted + ps.chunk - 1) / ps.chunk;
    ps.blocks = (int)std::min<long long>(chunks, 148LL * 8);
    CL_CUDA(cudaStreamSynchronize(c->stream));
}

void pair_launch(cl_ctx* c, const PairSetup& ps, void* rho) {
    cudaEvent_t e = prof_begin(c);
    if (ps.mma_ok) {
        clk::pm::PairMmaArgs g = ps.mma;
        g.coeff = c->coeff.p;
        g.prod = ps.mma_prod.p;
        with_pair_mma(g.n_used, g.n_orb, ps.mma_sliced, [&](auto k, auto pack, auto fold, auto cut) {
            constexpr int NB = decltype(k)::value;
            constexpr bool PACKED = decltype(pack)::value, FOLD = decltype(fold)::value, SLICED = decltype(cut)::value;
            const int threads = 32 * clk::pm::warps(NB);
            if (fp64_form(c))
                clk::pm::k_pair_mma<NB, PACKED, FOLD, SLICED, double><<<ps.mma_grid, threads, ps.mma_smem, c->stream>>>(
                    g, static_cast<cx<double>*>(rho));
            else
                clk::pm::k_pair_mma<NB, PACKED, FOLD, SLICED, float><<<ps.mma_grid, threads, ps.mma_smem, c->stream>>>(
                    g, static_cast<cx<float>*>(rho));
        });
    } else if (fp64_form(c) && !ps.tile_ok) {
        ensure_smem(clk::k_pair_density<double>, ps.smem);
        clk::k_pair_density<double><<<ps.blocks, 256, ps.smem, c->stream>>>(
            c->coeff.p, c->n_sorted, c->n_orb, nullptr, c->n_sorted, ps.segs.p, ps.n_segs, ps.states.p,
            ps.n_used, ps.chunk, static_cast<cx<double>*>(rho));
    } else if (ps.tile_ok) {  // 4 x 4-state tiles (FP64 sums, rounded once)
        const auto go = [&](auto tag) {
            using RT = decltype(tag);
            ensure_smem(clk::k_pair_density_tile<RT>, ps.tile_smem);
            clk::k_pair_density_tile<RT><<<ps.tile_blocks, ps.tile_threads, ps.tile_smem, c->stream>>>(
                c->coeff.p, c->n_sorted, c->n_orb, nullptr, c->n_sorted, ps.tile_states.p, ps.ns_pad,
                ps.tiles.p, ps.n_tiles, ps.tile_prod.p, ps.tile_atoms, static_cast<cx<RT>*>(rho));
        };
        if (fp64_form(c))
            go(double{});
        else
            go(float{});
    } else {  // the segment kernel (FP64 sums, rounded once)
        ensure_smem(clk::k_pair_density<float>, ps.smem);
        clk::k_pair_density<float><<<ps.blocks, 256, ps.smem, c->stream>>>(
            c->coeff.p, c->n_sorted, c->n_orb, nullptr, c->n_sorted, ps.segs.p, ps.n_segs, ps.states.p,
            ps.n_used, ps.chunk, static_cast<cx<float>*>(rho));
    }
    CL_LAUNCHED();
    prof_end(c, e, CL_KCLASS_DENSITY,
             (double)ps.n_used * c->n_sorted * c->n_orb * 16.0 + (double)ps.np * c->n_sorted * rho_bytes(c));
}

void pair_densities(cl_ctx* c, const std::vector<int2>& fl, void* rho) {
    // the lists stay with the context until its next eager call (stream-ordered after this one's launch)
    if (!c->eager_pairs) c->eager_pairs = {new PairSetup(), [](PairSetup* p) { delete p; }};
    PairSetup& ps = *c->eager_pairs;
    ps.mma_ok = ps.tile_ok = false;
    pair_setup(c, fl, ps);
    pair_launch(c, ps, rho);
}

// Device buffer of at least `count` elements, reallocated only when it must grow.
template <typename T>
void grow(DevBuf<T>& b, size_t count) {
    if (b.n >= count && b.p) return;
    b.alloc(count);
}

void check_ctx(cl_ctx* c) {
    if (!c) cl::fail(CL_ERR_ARGUMENT, "null context");
    CL_CUDA(cudaSetDevice(c->device));
}

void check_kernel(cl_ctx* c) {
    if (!c->kernel_ready) cl::fail(CL_ERR_STATE, "the Coulomb kernel is not initialised (call cl_set_kernel_*)");
}

void identity_atoms(cl_ctx* c) {
    if (c->grid_cell.p) return;
    const int nrows = c->n[1] * c->n[2];
    std::vector<int> cell((size_t)c->M), rp((size_t)nrows + 1);
    std::iota(cell.begin(), cell.end(), 0);
    for (int r = 0; r <= nrows; ++r) rp[r] = r * c->n[0];
    c->grid_cell.upload(cell.data(), cell.size(), c->stream);
    c->grid_row_ptr.upload(rp.data(), rp.size(), c->stream);
    CL_CUDA(cudaStreamSynchronize(c->stream));
}

}  // namespace

// =======================================================================================
// C ABI
// =======================================================================================
extern "C" {

int cl_create(cl_ctx** out, int nx, int ny, int nz, double sx, double sy, double sz, int mode) {
    if (out) *out = nullptr;
    cl_ctx* c = nullptr;
    int st = cl::guarded([&] {
        if (!out) cl::fail(CL_ERR_ARGUMENT, "null output pointer");
        if (nx <= 0 || ny <= 0 || nz <= 0) cl::fail(CL_ERR_ARGUMENT, "dimensions must be positive");
        if (mode < CL_MODE_FP64_PLAIN || mode > CL_MODE_FP32_SUBLATTICE) cl::fail(CL_ERR_ARGUMENT, "unknown mode %d", mode);
        const int dims[3] = {nx, ny, nz};
        for (int d = 0; d < 3; ++d) {
            if (!smooth235(dims[d]))
                cl::fail(CL_ERR_UNSUPPORTED, "grid size %d is not a product of 2, 3 and 5", dims[d]);
            if (dims[d] > 4096) cl::fail(CL_ERR_UNSUPPORTED, "grid size %d exceeds 4096", dims[d]);
        }
        const long long M = (long long)nx * ny * nz;
        if (M >= (1LL << 31)) cl::fail(CL_ERR_UNSUPPORTED, "grid of %lld cells exceeds 2^31", M);
        if (!(sx > 0 && sy > 0 && sz > 0)) cl::fail(CL_ERR_ARGUMENT, "step lengths must be positive");
        require_gpu();
        c = new cl_ctx();
        CL_CUDA(cudaGetDevice(&c->device));
        c->mode = mode;
        c->n[0] = nx;
        c->n[1] = ny;
        c->n[2] = nz;
        c->M = M;
        c->step[0] = sx;
        c->step[1] = sy;
        c->step[2] = sz;
        CL_CUDA(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
        for (auto& e : c->ev) CL_CUDA(cudaEventCreate(&e));
        for (int d = 0; d < 3; ++d) {
            Axis& A = c->ax[d];
            A.plan = make_plan(dims[d]);
            auto t64 = twiddles64(dims[d]);
            std::vector<cx<float>> t32(t64.size());
            for (size_t i = 0; i < t64.size(); ++i) {
                t32[i].re = (float)t64[i].re;
                t32[i].im = (float)t64[i].im;
            }
            A.tw64.upload(t64.data(), t64.size(), c->stream);
            A.tw32.upload(t32.data(), t32.size(), c->stream);
            auto ph = phases64(dims[d]);
            A.phase.upload(ph.data(), ph.size(), c->stream);
        }
        CL_CUDA(cudaStreamSynchronize(c->stream));
        *out = c;
    });
    if (st != CL_OK) delete c;
    return st;
}

void cl_destroy(cl_ctx* ctx) {
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    delete ctx;
}

int cl_set_kernel_coulomb(cl_ctx* c, double dielectric, double onsite, double tf_lattice) {
    return cl::guarded([&] {
        check_ctx(c);
        clk::KernelModel km{dielectric, onsite, 0, 0.0, 0.0};
        if (tf_lattice > 0) {
            if (!(dielectric > 1.0)) cl::fail(CL_ERR_ARGUMENT, "dielectric constant must be >1 to use Thomas-Fermi model");
            km.thomas_fermi = 1;
            thomas_fermi(dielectric, tf_lattice, &km.r_tf, &km.q_tf);
        }
        const int n1x = c->n[0] + 1, n1y = c->n[1] + 1, n1z = c->n[2] + 1;
        const long long total = (long long)n1x * n1y * n1z;
        c->kernel_ready = false;
        c->ghat.alloc(total);
        cudaEvent_t pe = prof_begin(c);
        clk::k_kernel_octant<<<grid_for(total), 256, 0, c->stream>>>(c->ghat.p, n1x, n1y, n1z, c->step[0], c->step[1],
                                                                     c->step[2], km);
        CL_LAUNCHED();
        transform_kernel(c);
        prof_end(c, pe, CL_KCLASS_KERNEL, (double)total * 8.0 * 7.0 + (double)c->M * 8.0 * (fp64_form(c) ? 8.0 : 4.0));
        CL_CUDA(cudaStreamSynchronize(c->stream));
        prof_collect(c);
    });
}

int cl_set_kernel_grid(cl_ctx* c, const double* G) {
    return cl::guarded([&] {
        check_ctx(c);
        if (!G) cl::fail(CL_ERR_ARGUMENT, "null kernel grid");
        const long long total = (long long)(c->n[0] + 1) * (c->n[1] + 1) * (c->n[2] + 1);
        c->kernel_ready = false;
        c->ghat.upload(G, total, c->stream);
        transform_kernel(c);
    });
}

int cl_prepare_grid(cl_ctx* c, const double* rho) {
    return cl::guarded([&] {
        check_ctx(c);
        check_kernel(c);
        if (!rho) cl::fail(CL_ERR_ARGUMENT, "null density");
        identity_atoms(c);
        c->grid_rho.upload(reinterpret_cast<const cx<double>*>(rho), c->M, c->stream);
        c->grid_V.alloc(c->M);
        const void* rho_in = c->grid_rho.p;
        if (!fp64_form(c)) {  // the FP32 forms' densities are complex64
            c->grid_rho32.alloc(c->M);
            clk::k_narrow<float><<<grid_for(c->M), 256, 0, c->stream>>>(c->grid_rho.p, c->grid_rho32.p, c->M);
            CL_LAUNCHED();
            rho_in = c->grid_rho32.p;
        }
        run_rounds_mode(c, rho_in, c->M, 1, c->grid_row_ptr.p, c->grid_cell.p, c->grid_V.p, c->M);
        CL_CUDA(cudaStreamSynchronize(c->stream));
        c->grid_prepared = true;
    });
}

int cl_calculate_grid(cl_ctx* c, const double* rho2, double out[2]) {
    return cl::guarded([&] {
        check_ctx(c);
        if (!c->grid_prepared) cl::fail(CL_ERR_STATE, "calculate() called before prepare()");
        if (!rho2 || !out) cl::fail(CL_ERR_ARGUMENT, "null argument");
        c->grid_rho2.upload(reinterpret_cast<const cx<double>*>(rho2), c->M, c->stream);
        DevBuf<double> o4;
        o4.alloc(5);
        const GramPlan dot = whole_gram(1, 1, false);
        tc_reserve(c, dot, c->M, false, false);
        gram(c, c->grid_V.p, false, c->M, c->grid_rho2.p, false, c->M, nullptr, dot, c->M, o4.p);
        double h[5];
        CL_CUDA(cudaMemcpyAsync(h, o4.p, sizeof h, cudaMemcpyDeviceToHost, c->stream));
        CL_CUDA(cudaStreamSynchronize(c->stream));
        check_gram_slot(h[4]);
        out[0] = h[0] - h[1];
        out[1] = h[2] + h[3];
    });
}

int cl_potential_grid(cl_ctx* c, double* V) {
    return cl::guarded([&] {
        check_ctx(c);
        if (!c->grid_prepared) cl::fail(CL_ERR_STATE, "potential() called before prepare()");
        if (!V) cl::fail(CL_ERR_ARGUMENT, "null argument");
        CL_CUDA(cudaMemcpyAsync(V, c->grid_V.p, sizeof(cx<double>) * c->M, cudaMemcpyDeviceToHost, c->stream));
        CL_CUDA(cudaStreamSynchronize(c->stream));
    });
}

}  // extern "C"

namespace {

void check_states_args(int n_states, int n_holes, int64_t n_atoms, int n_orb, const double* coeff,
                       const int64_t* cells) {
    if (n_states <= 0 || n_holes < 0 || n_holes > n_states || n_atoms <= 0 || n_orb <= 0 || !coeff || !cells)
        cl::fail(CL_ERR_ARGUMENT, "invalid states description");
    if (n_atoms >= (1LL << 31)) cl::fail(CL_ERR_UNSUPPORTED, "too many atoms");
}

// Sub-lattice decomposition for the (deduplicated) atom cells, in the sub-lattice modes: the
// modulus m in {4, 2} dividing every grid size whose classes need the least transform work,
// S / m^3 of the 8 rounds' (S occupied classes, each transformed at (2n/m)^3 points), kept when
// at most half of it, with at most 8 classes and a compiled z-mix length.  Classes go in
// class-id order, or in the canonical zinc-blende order when they are that set (shifted).
// CL_NO_SUBLATTICE=1 keeps the 8 rounds.
void plan_sublattice(cl_ctx* c, const std::vector<int>& cell_s) {
    Sublattice& sl = c->sl;
    const int old_m = sl.m, old_S = sl.S;
    int old_off[clk::kSlMaxClasses][3];
    std::memcpy(old_off, sl.off, sizeof old_off);
    sl.active = false;
    sl.zb = false;
    if (!sublattice_mode(c) || std::getenv("CL_NO_SUBLATTICE")) return;
    const int nx = c->n[0], ny = c->n[1], nz = c->n[2];
    double best = 0.5;
    int best_m = 0;
    std::vector<int> best_ids;
    for (int m : {4, 2}) {
        if (nx % m || ny % m || nz % m) continue;
        if (!clp::zmix_supported(2 * nz / m)) continue;
        std::vector<char> seen((size_t)m * m * m, 0);
        for (int cs : cell_s) {
            const int x = cs % nx, y = (cs / nx) % ny, z = cs / (nx * ny);
            seen[((z % m) * m + y % m) * m + x % m] = 1;
        }
        std::vector<int> ids;
        for (int id = 0; id < m * m * m; ++id)
            if (seen[id]) ids.push_back(id);
        if (ids.empty() || (int)ids.size() > clk::kSlMaxClasses) continue;
        const double cost = (double)ids.size() / (double)(m * m * m);
        if (cost <= best) {
            best = cost;
            best_m = m;
            best_ids = ids;
        }
    }
    if (!best_m) return;
    const int m = best_m, S = (int)best_ids.size();
    sl.m = m;
    sl.S = S;
    for (int s = 0; s < S; ++s) {
        sl.off[s][0] = best_ids[s] % m;
        sl.off[s][1] = (best_ids[s] / m) % m;
        sl.off[s][2] = best_ids[s] / (m * m);
    }
    if (m == 4 && S == 8) {  // the zinc-blende set, shifted by t?
        for (int t = 0; t < 64 && !sl.zb; ++t) {
            const int tx = t % 4, ty = (t / 4) % 4, tz = t / 16;
            int cand[8][3];
            bool all = true;
            for (int s = 0; s < 8 && all; ++s) {
                cand[s][0] = (clk::ZincBlende::off[s][0] + tx) % 4;
                cand[s][1] = (clk::ZincBlende::off[s][1] + ty) % 4;
                cand[s][2] = (clk::ZincBlende::off[s][2] + tz) % 4;
                all = std::binary_search(best_ids.begin(), best_ids.end(),
                                         (cand[s][2] * 4 + cand[s][1]) * 4 + cand[s][0]);
            }
            if (all) {
                sl.zb = true;
                std::memcpy(sl.off, cand, sizeof cand);
            }
        }
    }
    for (int d = 0; d < 3; ++d) {
        sl.sub[d] = c->n[d] / m;
        sl.pad[d] = 2 * c->n[d] / m;
    }
    sl.vn[0] = sl.pad[0];
    sl.vn[1] = sl.pad[1];
    sl.vn[2] = S * sl.sub[2];
    sl.vM = (long long)sl.vn[0] * sl.vn[1] * sl.vn[2];
    sl.table = clk::sl_table(sl.off, S, m);
    if (m != old_m || S != old_S || std::memcmp(old_off, sl.off, sizeof old_off) != 0) sl.tables_version = -1;
    sl.active = true;
}

// Atoms sorted by cell; where several atoms share a cell the one listed last wins, as with
// F[cell] = value in atom order (Product.cpp:16-30).  Builds the sorted cell list, the input
// atom of each slot, the row CSR and the live-row count, and uploads them (synchronously).  With
// the sub-lattice decomposition the atoms are then ordered by their cell of the virtual grid
// (class-stacked sub-grids), which is the order every later pass and reduction uses.  A list
// identical to the previous load's is not processed again.
void load_cells(cl_ctx* c, int64_t n_atoms, const int64_t* cells) {
    if ((int64_t)c->cells_seen.size() == n_atoms && c->n_sorted > 0 &&
        std::memcmp(c->cells_seen.data(), cells, sizeof(int64_t) * (size_t)n_atoms) == 0)
        return;
    c->cells_seen.clear();
    ++c->layout_version;
    std::vector<int> order((size_t)n_atoms);
    std::iota(order.begin(), order.end(), 0);
    for (int64_t a = 0; a < n_atoms; ++a)
        if (cells[a] < 0 || cells[a] >= c->M) cl::fail(CL_ERR_ARGUMENT, "atom %lld lies outside the grid", (long long)a);
    bool sorted = true;
    for (int64_t a = 1; a < n_atoms && sorted; ++a) sorted = cells[a - 1] < cells[a];
    if (!sorted) std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return cells[x] < cells[y]; });
    std::vector<int> cell_s, orig_s;
    cell_s.reserve((size_t)n_atoms);
    orig_s.reserve((size_t)n_atoms);
    c->atom_slot.assign((size_t)n_atoms, 0);
    for (size_t i = 0; i < order.size(); ++i) {
        const int a = order[i];
        if (!cell_s.empty() && cell_s.back() == (int)cells[a]) {
            orig_s.back() = a;  // later atom of the same cell replaces the earlier one
        } else {
            cell_s.push_back((int)cells[a]);
            orig_s.push_back(a);
        }
        c->atom_slot[a] = (int)cell_s.size() - 1;
    }
    plan_sublattice(c, cell_s);
    int nx = c->n[0];
    int nrows = c->n[1] * c->n[2];
    if (c->sl.active) {
        const Sublattice& sl = c->sl;
        const int m = sl.m, gx = c->n[0], gy = c->n[1];
        int cls_of[64];
        for (int s = 0; s < sl.S; ++s) cls_of[(sl.off[s][2] * m + sl.off[s][1]) * m + sl.off[s][0]] = s;
        std::vector<int> vcell(cell_s.size()), perm(cell_s.size());
        for (size_t i = 0; i < cell_s.size(); ++i) {
            const int cs = cell_s[i];
            const int x = cs % gx, y = (cs / gx) % gy, z = cs / (gx * gy);
            const int s = cls_of[((z % m) * m + y % m) * m + x % m];
            vcell[i] = ((s * sl.sub[2] + z / m) * sl.pad[1] + y / m) * sl.pad[0] + x / m;
        }
        std::iota(perm.begin(), perm.end(), 0);
        std::sort(perm.begin(), perm.end(), [&](int a, int b) { return vcell[a] < vcell[b]; });
        std::vector<int> new_pos(cell_s.size());
        std::vector<int> vc(cell_s.size()), vo(cell_s.size());
        for (size_t k = 0; k < perm.size(); ++k) {
            new_pos[perm[k]] = (int)k;
            vc[k] = vcell[perm[k]];
            vo[k] = orig_s[perm[k]];
        }
        for (auto& slot : c->atom_slot) slot = new_pos[slot];
        cell_s.swap(vc);
        orig_s.swap(vo);
        nx = sl.vn[0];
        nrows = sl.vn[1] * sl.vn[2];
    }
    std::vector<int> rp((size_t)nrows + 1, 0);
    for (int cs : cell_s) rp[cs / nx + 1]++;
    for (int r = 0; r < nrows; ++r) rp[r + 1] += rp[r];
    long long live = 0;
    for (int r = 0; r < nrows; ++r) live += rp[r + 1] > rp[r];
    c->live_rows = live;
    c->n_sorted = (long long)cell_s.size();
    c->cell_sorted.upload(cell_s.data(), cell_s.size(), c->stream);
    c->orig_sorted.upload(orig_s.data(), orig_s.size(), c->stream);
    c->row_ptr.upload(rp.data(), rp.size(), c->stream);
    c->slot_of_atom.upload(c->atom_slot.data(), c->atom_slot.size(), c->stream);
    if (c->sl.active && c->sl.sub[0] <= 64) {
        c->row_mask.alloc((size_t)nrows);
        CL_CUDA(cudaMemsetAsync(c->row_mask.p, 0, sizeof(unsigned long long) * nrows, c->stream));
        clk::k_row_masks<<<grid_for(c->n_sorted), 256, 0, c->stream>>>(c->cell_sorted.p, (int)c->n_sorted, nx,
                                                                       c->row_mask.p);
        CL_LAUNCHED();
    }
    CL_CUDA(cudaStreamSynchronize(c->stream));
    c->cells_seen.assign(cells, cells + n_atoms);
}

// Uploads state s of the caller's coefficients ([state][atom][orb], input atom order) through
// a staging slot and stores it in the cell-sorted atom order the pair-density kernels read
// (k_gather_atoms): consecutive slots of a block are then contiguous rows in HBM.  Both on
// `stream`, so slot s & 1 is free again once the gather of state s - 2 has run.
void upload_state_sorted(cl_ctx* c, int s, const double* coeff, cudaStream_t stream) {
    const size_t per_in = (size_t)c->n_atoms * c->n_orb, per_s = (size_t)c->n_sorted * c->n_orb;
    cx<double>* slot = c->coeff_stage.p + (size_t)(s & 1) * per_in;
    CL_CUDA(cudaMemcpyAsync(slot, coeff + 2 * (size_t)s * per_in, sizeof(cx<double>) * per_in, cudaMemcpyHostToDevice,
                            stream));
    const int blocks = (int)std::max<long long>(1, std::min<long long>(((long long)per_s + 255) / 256, 148LL * 16));
    clk::k_gather_atoms<<<blocks, 256, 0, stream>>>(slot, c->orig_sorted.p, c->n_sorted, c->n_orb,
                                                    c->coeff.p + (size_t)s * per_s);
    CL_LAUNCHED();
}
// Makes room for the states' coefficients on the loaded cells; no states are loaded when that fails.
void reserve_states(cl_ctx* c, int n_states, int n_holes, int64_t n_atoms, int n_orb) {
    if (n_states != c->n_states || n_orb != c->n_orb) ++c->layout_version;
    c->n_states = 0;
    c->n_atoms = n_atoms;
    grow(c->coeff, (size_t)n_states * c->n_sorted * n_orb);
    grow(c->coeff_stage, 2 * (size_t)n_atoms * n_orb);
    c->n_states = n_states;
    c->n_holes = n_holes;
    c->n_orb = n_orb;
}

}  // namespace

extern "C" {

int cl_set_states(cl_ctx* c, int n_states, int n_holes, int64_t n_atoms, int n_orb, const double* coeff,
                  const int64_t* cells) {
    return cl::guarded([&] {
        check_ctx(c);
        check_states_args(n_states, n_holes, n_atoms, n_orb, coeff, cells);
        load_cells(c, n_atoms, cells);
        reserve_states(c, n_states, n_holes, n_atoms, n_orb);
        for (int s = 0; s < n_states; ++s) upload_state_sorted(c, s, coeff, c->stream);
        CL_CUDA(cudaStreamSynchronize(c->stream));
    });
}

}  // extern "C"

namespace {

// The densities of a request: rows (the left densities, then those only on the right, in ascending product
// order: ascending higher states), the Gram's columns block by block, and the blocks that its steps read
// (gram_blocks.hpp).
struct DensityLayout {
    std::vector<int> prods;       // product of each row
    std::vector<int> columns;     // row of each left, then of each right column of the Gram
    std::vector<int> lcol, rcol;  // left and right column of each product, -1: none
    std::vector<char> sym;          // per product: pairs with it are read with the larger product on the left
    GramPlan gram;
    // (state, state) of every row, 0-based, the higher first
    std::vector<int2> states() const {
        std::vector<int2> fl(prods.size());
        for (size_t i = 0; i < prods.size(); ++i) {
            int a, b;
            cl::product_states(prods[i], &a, &b);
            fl[i] = make_int2(a - 1, b - 1);
        }
        return fl;
    }
};

// Symmetry needs the whole convolution (all 8 rounds).  The FP64 forms use it at any size (2); the FP32
// forms, whose V_l rho_r and V_r rho_l differ by the transforms' rounding, only where it leaves out whole
// 64 x 64 tiles (1), so that up to 64 densities a shard's integrals equal the full request's.
int symmetric_blocks(const cl_ctx* c, int round_mask = 0xFF) {
    return (round_mask & 0xFF) != 0xFF ? 0 : fp64_form(c) ? 2 : 1;
}

// Columns go in ascending product order within a block.  `symmetric`: which blocks are treated as symmetric
// (symmetric_blocks).
DensityLayout layout_densities(const std::vector<cl::PlanStep>& plan, int n_states, int symmetric) {
    const int P = n_states * (n_states + 1) / 2;
    std::vector<char> is_left(P, 0), is_right(P, 0);
    for (const auto& st : plan) {
        is_left[st.left.product] = 1;
        is_right[st.right.product] = 1;
    }
    // connected components of the pairing (union-find; over as soon as one is left)
    std::vector<int> root(P);
    std::iota(root.begin(), root.end(), 0);
    const auto find = [&](int p) {
        while (root[p] != p) p = root[p] = root[root[p]];
        return p;
    };
    int parts = 0;
    for (int p = 0; p < P; ++p) parts += is_left[p] || is_right[p];
    for (size_t i = 0; i < plan.size() && parts > 1; ++i) {
        const int a = find(plan[i].left.product), b = find(plan[i].right.product);
        if (a == b) continue;
        root[std::max(a, b)] = std::min(a, b);
        --parts;
    }
    struct Part {
        std::vector<int> lefts, rights;
    };
    std::vector<Part> found;
    std::vector<int> id(P, -1);
    for (int p = 0; p < P; ++p) {
        if (!is_left[p] && !is_right[p]) continue;
        int& k = id[find(p)];
        if (k < 0) {
            k = (int)found.size();
            found.emplace_back();
        }
        if (is_left[p]) found[k].lefts.push_back(p);
        if (is_right[p]) found[k].rights.push_back(p);
    }
    // parts of fewer than 4 densities (half an MMA tile) share one block, and so do the smallest beyond
    // the blocks a launch can hold
    std::stable_sort(found.begin(), found.end(), [](const Part& a, const Part& b) {
        return a.lefts.size() + a.rights.size() > b.lefts.size() + b.rights.size();
    });
    const auto small = [](const Part& q) { return q.lefts.size() < 4 && q.rights.size() < 4; };
    while (found.size() > 1 && ((int)found.size() > clk::kGramBlocks || (small(found.back()) && small(found[found.size() - 2])))) {
        Part last = std::move(found.back());
        found.pop_back();
        Part& into = found.back();
        into.lefts.insert(into.lefts.end(), last.lefts.begin(), last.lefts.end());
        into.rights.insert(into.rights.end(), last.rights.begin(), last.rights.end());
    }
    DensityLayout d;
    std::vector<int> row(P, -1);
    for (const auto* side : {&is_left, &is_right}) {
        for (int p = 0; p < P; ++p) {
            if (!(*side)[p] || row[p] >= 0) continue;
            row[p] = (int)d.prods.size();
            d.prods.push_back(p);
        }
    }
    d.lcol.assign(P, -1);
    d.rcol.assign(P, -1);
    d.sym.assign(P, 0);
    std::vector<char> part_sym;
    for (Part& q : found) {
        std::sort(q.lefts.begin(), q.lefts.end());
        std::sort(q.rights.begin(), q.rights.end());
        const bool sym = (symmetric == 2 || (symmetric == 1 && q.lefts.size() > 64)) && q.lefts == q.rights;
        part_sym.push_back(sym);
        if (sym)
            for (int p : q.lefts) d.sym[p] = 1;
    }
    const bool all_sym = std::find(part_sym.begin(), part_sym.end(), 0) == part_sym.end();
    std::vector<int> right_rows;
    for (size_t k = 0; k < found.size(); ++k) {
        const Part& q = found[k];
        d.gram.blocks.push_back(clk::GramBlock{(int)d.columns.size(), (int)q.lefts.size(), (int)right_rows.size(),
                                               (int)q.rights.size(), part_sym[k]});
        for (int p : q.lefts) {
            d.lcol[p] = (int)d.columns.size();
            d.columns.push_back(row[p]);
        }
        for (int p : q.rights) {
            d.rcol[p] = (int)right_rows.size();
            right_rows.push_back(row[p]);
        }
    }
    d.gram.nl = (int)d.columns.size();
    d.gram.nr = (int)right_rows.size();
    d.gram.whole = clk::GramBlock{0, d.gram.nl, 0, d.gram.nr, all_sym};
    d.columns.insert(d.columns.end(), right_rows.begin(), right_rows.end());
    return d;
}

// f(begin, end) over [0, n) on several host threads where there is enough to share.
template <typename F>
void share_range(size_t n, F&& f) {
    const size_t hw = std::max(1u, std::thread::hardware_concurrency());
    const size_t nt = std::min<size_t>(std::min<size_t>(hw, 32), n / 65536 + 1);
    if (nt <= 1) {
        f(size_t{0}, n);
        return;
    }
    std::vector<std::thread> pool;
    for (size_t t = 0; t < nt; ++t) pool.emplace_back([&, t] { f(n * t / nt, n * (t + 1) / nt); });
    for (auto& th : pool) th.join();
}

// Where a step's value comes from (coulombo.cpp:199-207): the Gram entry of its (left, right) pair,
// combined for the pair's conjugation flags and conjugated when the left product is.
struct StepValue {
    uint64_t entry : 61, turned : 1, mixed : 1, conj : 1;
};
std::vector<StepValue> step_values(const std::vector<cl::PlanStep>& plan, const DensityLayout& d) {
    std::vector<StepValue> v(plan.size());
    share_range(plan.size(), [&](size_t i0, size_t i1) {
        for (size_t i = i0; i < i1; ++i) {
            const auto& st = plan[i];
            // a symmetric block holds the pairs with the larger product on the left
            const bool turned = d.sym[st.left.product] && st.left.product < st.right.product;
            const int l = d.lcol[turned ? st.right.product : st.left.product];
            const int r = d.rcol[turned ? st.left.product : st.right.product];
            v[i] = StepValue{(uint64_t)l * d.gram.nr + r, turned, st.left.conjugate != st.right.conjugate,
                             st.left.conjugate != 0};
        }
    });
    return v;
}
void map_step_values(const std::vector<cl::PlanStep>& plan, const std::vector<StepValue>& from, const double* h,
                     double* out) {
    share_range(plan.size(), [&](size_t i0, size_t i1) {
        for (size_t i = i0; i < i1; ++i) {
            const StepValue v = from[i];
            const double* q = h + 4 * v.entry;
            const double ad = v.turned ? q[3] : q[2], bc = v.turned ? q[2] : q[3];
            const double im = v.mixed ? bc - ad : ad + bc;
            double* o = out + 2 * (size_t)plan[i].id;
            o[0] = v.mixed ? q[0] + q[1] : q[0] - q[1];
            o[1] = v.conj ? -im : im;
        }
    });
}

// The steps of shard `shard` of `n_shards`: the plan's prepared (left) densities, in ascending
// product order, are dealt round-robin, and a step belongs to the shard of its left density.
// Every step is in exactly one shard, so the shards' integrals add up to the whole request's.
std::vector<cl::PlanStep> shard_steps(std::vector<cl::PlanStep> plan, int n_states, int shard, int n_shards) {
    if (n_shards < 1 || shard < 0 || shard >= n_shards) cl::fail(CL_ERR_ARGUMENT, "invalid shard %d of %d", shard, n_shards);
    if (n_shards == 1) return plan;
    const int P = n_states * (n_states + 1) / 2;
    std::vector<int> owner(P, -1);
    for (const auto& st : plan) owner[st.left.product] = 0;
    int k = 0;
    for (int p = 0; p < P; ++p)
        if (owner[p] == 0) owner[p] = k++ % n_shards;
        else owner[p] = -1;
    std::vector<cl::PlanStep> mine;
    for (const auto& st : plan)
        if (owner[st.left.product] == shard) mine.push_back(st);
    return mine;
}

void compute_impl(cl_ctx* c, int64_t n_int, const int16_t* spec, double* out, int round_mask, int shard = 0,
                  int n_shards = 1) {
    {
        check_ctx(c);
        check_kernel(c);
        if (c->n_states == 0) cl::fail(CL_ERR_STATE, "no states loaded (call cl_set_states)");
        if (n_int < 0 || (n_int && (!spec || !out))) cl::fail(CL_ERR_ARGUMENT, "invalid integral list");
        std::memset(c->timings, 0, sizeof c->timings);
        if (n_int == 0) return;
        std::vector<std::array<int16_t, 4>> specs((size_t)n_int);
        for (int64_t i = 0; i < n_int; ++i)
            for (int k = 0; k < 4; ++k) specs[i][k] = spec[4 * i + k];
        const auto plan = shard_steps(cl::orient_steps(c->n_states, specs), c->n_states, shard, n_shards);
        if (n_shards > 1) std::memset(out, 0, sizeof(double) * 2 * (size_t)n_int);
        if (plan.empty()) return;
        const DensityLayout lay = layout_densities(plan, c->n_states, symmetric_blocks(c, round_mask));
        const std::vector<int>& columns = lay.columns;
        const std::vector<int2> fl = lay.states();
        const int nu = (int)lay.prods.size(), nl = lay.gram.nl, nr = lay.gram.nr;
        const long long As = c->n_sorted;
        DevBuf<int>& dr = c->req_rows;
        grow(dr, columns.size());
        CL_CUDA(cudaMemcpyAsync(dr.p, columns.data(), columns.size() * sizeof(int), cudaMemcpyHostToDevice, c->stream));
        DevBuf<cx<double>>& rho = c->req_rho;
        DevBuf<cx<double>>& V = c->req_V;
        grow(rho, (size_t)nu * As);
        grow(V, (size_t)nl * As);
        DevBuf<double>& o4 = c->req_o4;
        grow(o4, (size_t)4 * nl * nr + 1);
        tc_reserve(c, lay.gram, As, v_fp32(c), rho_bytes(c) == sizeof(cx<float>));
        CL_CUDA(cudaEventRecord(c->ev[0], c->stream));
        pair_densities(c, fl, rho.p);
        CL_CUDA(cudaEventRecord(c->ev[1], c->stream));
        const bool v32 = v_fp32(c);
        run_transforms(c, rho.p, As, nl, V.p, As, v32, round_mask);
        CL_CUDA(cudaEventRecord(c->ev[2], c->stream));
        gram(c, V.p, v32, As, rho.p, rho_bytes(c) == sizeof(cx<float>), As, dr.p, lay.gram, As, o4.p);
        CL_CUDA(cudaEventRecord(c->ev[3], c->stream));
        std::vector<double> h((size_t)4 * nl * nr + 1);
        CL_CUDA(cudaMemcpyAsync(h.data(), o4.p, h.size() * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
        CL_CUDA(cudaStreamSynchronize(c->stream));
        check_gram_slot(h.back());
        float t01, t12, t23, t03;
        CL_CUDA(cudaEventElapsedTime(&t01, c->ev[0], c->ev[1]));
        CL_CUDA(cudaEventElapsedTime(&t12, c->ev[1], c->ev[2]));
        CL_CUDA(cudaEventElapsedTime(&t23, c->ev[2], c->ev[3]));
        CL_CUDA(cudaEventElapsedTime(&t03, c->ev[0], c->ev[3]));
        c->timings[0] = t01;
        c->timings[1] = t12;
        c->timings[2] = t23;
        c->timings[3] = t03;
        prof_collect(c);
        map_step_values(plan, step_values(plan, lay), h.data(), out);
    }
}

// cl_compute_states: the states' coefficients are uploaded one state at a time on a copy stream
// while the densities whose states have arrived are transformed.  Left densities are grouped by
// their higher state index; a group's pair densities and rounds wait only for its last state.
void compute_states_impl(cl_ctx* c, int n_states, int n_holes, int64_t n_atoms, int n_orb, const double* coeff,
                         const int64_t* cells, int64_t n_int, const int16_t* spec, double* out) {
    check_ctx(c);
    check_kernel(c);
    check_states_args(n_states, n_holes, n_atoms, n_orb, coeff, cells);
    if (n_int < 0 || (n_int && (!spec || !out))) cl::fail(CL_ERR_ARGUMENT, "invalid integral list");
    load_cells(c, n_atoms, cells);
    reserve_states(c, n_states, n_holes, n_atoms, n_orb);
    std::memset(c->timings, 0, sizeof c->timings);
    if (!c->copy_stream) CL_CUDA(cudaStreamCreateWithFlags(&c->copy_stream, cudaStreamNonBlocking));
    while ((int)c->state_ev.size() < n_states) {
        cudaEvent_t e;
        CL_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        c->state_ev.push_back(e);
    }
    if (n_int == 0) {
        for (int s = 0; s < n_states; ++s) upload_state_sorted(c, s, coeff, c->stream);
        CL_CUDA(cudaStreamSynchronize(c->stream));
        return;
    }
    // The integral list is checked (and planned) before any copy reads the caller's buffer.
    std::vector<std::array<int16_t, 4>> specs((size_t)n_int);
    for (int64_t i = 0; i < n_int; ++i)
        for (int k = 0; k < 4; ++k) specs[i][k] = spec[4 * i + k];
    const auto plan = cl::orient_steps(n_states, specs);
    // On every error path below, the copies already queued from the caller's buffer (and the
    // work waiting on them) finish before the call returns, so the buffer is free for reuse
    // once the call has returned, whatever its status.
    struct DrainOnError {
        cudaStream_t a, b;
        bool armed = true;
        ~DrainOnError() {
            if (!armed) return;
            cudaStreamSynchronize(a);
            cudaStreamSynchronize(b);
            cudaGetLastError();
        }
    } drain{c->copy_stream, c->stream};
    // Uploads, one state at a time on the copy stream.  From pinned memory they are all enqueued
    // now and overlap the planning below; from pageable memory a copy returns only once staged,
    // so they are interleaved with the groups that need them (the groups already enqueued run
    // meanwhile).
    CL_CUDA(cudaEventRecord(c->ev[0], c->stream));
    CL_CUDA(cudaStreamWaitEvent(c->copy_stream, c->ev[0], 0));
    int uploaded = 0;
    const auto upload_through = [&](int last) {
        for (; uploaded <= last && uploaded < n_states; ++uploaded) {
            upload_state_sorted(c, uploaded, coeff, c->copy_stream);
            CL_CUDA(cudaEventRecord(c->state_ev[uploaded], c->copy_stream));
        }
    };
    {
        cudaPointerAttributes attr{};
        if (cudaPointerGetAttributes(&attr, coeff) == cudaSuccess && attr.type == cudaMemoryTypeHost)
            upload_through(n_states - 1);
        cudaGetLastError();  // pageable memory is not an error
    }
    const DensityLayout lay = layout_densities(plan, n_states, symmetric_blocks(c));
    const std::vector<int>& columns = lay.columns;
    const std::vector<int2> rows = lay.states();
    const int nu = (int)lay.prods.size(), nl = lay.gram.nl, nr = lay.gram.nr;
    // groups of left densities: cut at a state boundary once a group holds nl/6 densities
    struct Group {
        int begin, end, last_state;
        PairSetup ps;
    };
    std::vector<std::unique_ptr<Group>> groups;
    const int min_group = std::max(1, nl / 6);
    for (int i = 0; i < nl;) {
        int j = i;
        int hi = rows[i].x;
        while (j < nl && (j - i < min_group || rows[j].x == hi)) {
            hi = std::max(hi, rows[j].x);
            ++j;
        }
        auto g = std::make_unique<Group>();
        g->begin = i;
        g->end = j;
        g->last_state = hi;
        groups.push_back(std::move(g));
        i = j;
    }
    auto pairs_of = [&](int b, int e) { return std::vector<int2>(rows.begin() + b, rows.begin() + e); };
    for (auto& g : groups) pair_setup(c, pairs_of(g->begin, g->end), g->ps);
    PairSetup ps_right;
    if (nu > nl) pair_setup(c, pairs_of(nl, nu), ps_right);
    const long long As = c->n_sorted;
    const bool v32 = v_fp32(c);
    DevBuf<int>& dr = c->req_rows;
    grow(dr, columns.size());
    CL_CUDA(cudaMemcpyAsync(dr.p, columns.data(), columns.size() * sizeof(int), cudaMemcpyHostToDevice, c->stream));
    DevBuf<cx<double>>& rho = c->req_rho;
    DevBuf<cx<double>>& V = c->req_V;
    grow(rho, (size_t)nu * As);
    grow(V, (size_t)nl * As);
    DevBuf<double>& o4 = c->req_o4;
    grow(o4, (size_t)4 * nl * nr + 1);
    tc_reserve(c, lay.gram, As, v_fp32(c), rho_bytes(c) == sizeof(cx<float>));
    CL_CUDA(cudaStreamSynchronize(c->stream));
    for (auto& g : groups) {
        upload_through(g->last_state);
        CL_CUDA(cudaStreamWaitEvent(c->stream, c->state_ev[g->last_state], 0));
        pair_launch(c, g->ps, rho_at(c, rho.p, (long long)g->begin * As));
        run_transforms(c, rho_at(c, rho.p, (long long)g->begin * As), As, g->end - g->begin,
                       v_at(V.p, (long long)g->begin * As, v32), As, v32);
    }
    upload_through(n_states - 1);
    CL_CUDA(cudaStreamWaitEvent(c->stream, c->state_ev[n_states - 1], 0));
    if (nu > nl) pair_launch(c, ps_right, rho_at(c, rho.p, (long long)nl * As));
    CL_CUDA(cudaEventRecord(c->ev[2], c->stream));
    gram(c, V.p, v32, As, rho.p, rho_bytes(c) == sizeof(cx<float>), As, dr.p, lay.gram, As, o4.p);
    CL_CUDA(cudaEventRecord(c->ev[3], c->stream));
    std::vector<double> h((size_t)4 * nl * nr + 1);
    CL_CUDA(cudaMemcpyAsync(h.data(), o4.p, h.size() * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    CL_CUDA(cudaStreamSynchronize(c->stream));  // after the wait on the last upload: all copies done
    drain.armed = false;
    check_gram_slot(h.back());
    float t02, t23, t03;
    CL_CUDA(cudaEventElapsedTime(&t02, c->ev[0], c->ev[2]));
    CL_CUDA(cudaEventElapsedTime(&t23, c->ev[2], c->ev[3]));
    CL_CUDA(cudaEventElapsedTime(&t03, c->ev[0], c->ev[3]));
    c->timings[0] = 0;  // pair densities are interleaved with the uploads and the rounds
    c->timings[1] = t02;
    c->timings[2] = t23;
    c->timings[3] = t03;
    prof_collect(c);
    map_step_values(plan, step_values(plan, lay), h.data(), out);
}
}  // namespace

extern "C" {

int cl_compute_states(cl_ctx* c, int n_states, int n_holes, int64_t n_atoms, int n_orb, const double* coeff,
                      const int64_t* cells, int64_t n_int, const int16_t* spec, double* out) {
    return cl::guarded(
        [&] { compute_states_impl(c, n_states, n_holes, n_atoms, n_orb, coeff, cells, n_int, spec, out); });
}

int cl_compute(cl_ctx* c, int64_t n_int, const int16_t* spec, double* out) {
    return cl::guarded([&] { compute_impl(c, n_int, spec, out, 0xFF); });
}

int cl_compute_rounds(cl_ctx* c, int64_t n_int, const int16_t* spec, int round_mask, double* out) {
    return cl::guarded([&] {
        if (round_mask < 0 || round_mask > 0xFF) cl::fail(CL_ERR_ARGUMENT, "round mask must be within 0..255");
        compute_impl(c, n_int, spec, out, round_mask);
    });
}

int cl_compute_shard(cl_ctx* c, int64_t n_int, const int16_t* spec, int shard, int n_shards, double* out) {
    return cl::guarded([&] { compute_impl(c, n_int, spec, out, 0xFF, shard, n_shards); });
}

int cl_set_profiling(cl_ctx* c, int enable) {
    return cl::guarded([&] {
        check_ctx(c);
        CL_CUDA(cudaStreamSynchronize(c->stream));
        prof_collect(c);
        c->profiling = enable != 0;
        if (c->profiling) {
            std::fill(std::begin(c->prof_ms), std::end(c->prof_ms), 0.0);
            std::fill(std::begin(c->prof_bytes), std::end(c->prof_bytes), 0.0);
            std::fill(std::begin(c->prof_launches), std::end(c->prof_launches), (int64_t)0);
        }
    });
}

int cl_kernel_profile(cl_ctx* c, double ms[CL_NUM_KCLASS], int64_t launches[CL_NUM_KCLASS],
                      double bytes[CL_NUM_KCLASS]) {
    return cl::guarded([&] {
        check_ctx(c);
        CL_CUDA(cudaStreamSynchronize(c->stream));
        prof_collect(c);
        for (int k = 0; k < CL_NUM_KCLASS; ++k) {
            if (ms) ms[k] = c->prof_ms[k];
            if (launches) launches[k] = c->prof_launches[k];
            if (bytes) bytes[k] = c->prof_bytes[k];
        }
    });
}

int cl_potentials(cl_ctx* c, double* out) {
    return cl::guarded([&] {
        check_ctx(c);
        check_kernel(c);
        if (c->n_states == 0) cl::fail(CL_ERR_STATE, "no states loaded (call cl_set_states)");
        if (!out) cl::fail(CL_ERR_ARGUMENT, "null output");
        const int n = c->n_states;
        const long long As = c->n_sorted;
        std::vector<int2> fl(n);
        for (int s = 0; s < n; ++s) fl[s] = make_int2(s, s);
        DevBuf<cx<double>>& rho = c->req_rho;
        DevBuf<cx<double>>& V = c->req_V;
        grow(rho, (size_t)n * As);
        grow(V, (size_t)n * As);
        grow(c->pot, (size_t)n * c->n_atoms);
        CL_CUDA(cudaEventRecord(c->ev[0], c->stream));
        pair_densities(c, fl, rho.p);
        CL_CUDA(cudaEventRecord(c->ev[1], c->stream));
        const bool v32 = c->sl.active && !fp64_form(c);  // as the inverse passes produce them
        run_transforms(c, rho.p, As, n, V.p, As, v32);
        CL_CUDA(cudaEventRecord(c->ev[2], c->stream));
        // the real parts in the caller's atom order: half the bytes over the host link
        const dim3 grid((unsigned)std::min<long long>((c->n_atoms + 255) / 256, 148LL * 8), n);
        if (v32)
            clk::k_potential_of_atoms<float><<<grid, 256, 0, c->stream>>>(reinterpret_cast<const cx<float>*>(V.p), As,
                                                                         c->slot_of_atom.p, c->n_atoms, c->pot.p);
        else
            clk::k_potential_of_atoms<double><<<grid, 256, 0, c->stream>>>(V.p, As, c->slot_of_atom.p, c->n_atoms,
                                                                          c->pot.p);
        CL_LAUNCHED();
        CL_CUDA(cudaMemcpyAsync(out, c->pot.p, sizeof(double) * (size_t)n * c->n_atoms, cudaMemcpyDeviceToHost, c->stream));
        CL_CUDA(cudaStreamSynchronize(c->stream));
        float t01, t12;
        CL_CUDA(cudaEventElapsedTime(&t01, c->ev[0], c->ev[1]));
        CL_CUDA(cudaEventElapsedTime(&t12, c->ev[1], c->ev[2]));
        prof_collect(c);
        c->timings[0] = t01;
        c->timings[1] = t12;
        c->timings[2] = 0;
        c->timings[3] = t01 + t12;
    });
}

}  // extern "C"

// ---------------------------------------------------------------------------------------
// Prepared requests and graph-captured batches
// ---------------------------------------------------------------------------------------
// What a request's launches depend on besides its own lists: a graph names the buffers, sizes and tables of its
// capture, and an eager run has sized them.
struct LaunchState {
    long long layout_version = -1, kernel_version = -1;
    unsigned long long moves = 0;
    bool operator==(const LaunchState& o) const {
        return layout_version == o.layout_version && kernel_version == o.kernel_version && moves == o.moves;
    }
};

struct cl_request {
    cl_ctx* ctx = nullptr;
    int device = 0;  // the context's: a request may be destroyed after its context
    int64_t n_int = 0;
    std::vector<cl::PlanStep> plan;
    DensityLayout lay;
    std::vector<StepValue> values;
    int nl = 0, nr = 0;
    PairSetup ps;
    DevBuf<int> rows;
    DevBuf<cx<double>> rho, V;
    DevBuf<double> o4;
    double* o4_host = nullptr;  // pinned
    LaunchState warm;  // at the last eager run
    int n_shards = 1;  // out entries of other shards' steps are zero
    int top_state = 0;              // the highest state that the request names, from 1
    long long layout_version = -1;  // the context's, at the last request_layout
    ~cl_request() {
        if (o4_host) cudaFreeHost(o4_host);
    }
};

struct cl_batch {
    int device = 0;
    std::vector<cl_request*> reqs;
    std::vector<LaunchState> captured;  // per request
    cudaStream_t master = nullptr;
    cudaEvent_t fork = nullptr, t0 = nullptr, t1 = nullptr;
    std::vector<cudaEvent_t> joins;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    double last_ms = 0;
    // per-launch event pairs captured into the graph for requests whose context profiles
    std::vector<std::vector<cl_ctx::ProfEntry>> prof;
    std::vector<cudaEvent_t> prof_events;
    void drop_graph() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        exec = nullptr;
        graph = nullptr;
        for (auto e : prof_events) cudaEventDestroy(e);
        prof_events.clear();
    }
    ~cl_batch() {
        drop_graph();
        for (auto e : joins) cudaEventDestroy(e);
        if (fork) cudaEventDestroy(fork);
        if (t0) cudaEventDestroy(t0);
        if (t1) cudaEventDestroy(t1);
        if (master) cudaStreamDestroy(master);
    }
};

namespace {

// Lists, launch shapes and buffers of a request for the states that its context holds now: made when the
// request is created, and again when cl_set_states or cl_compute_states has loaded other atoms, another number of
// states or of orbitals since (the stored shapes would read and write past the new buffers).
void request_layout(cl_request* r) {
    cl_ctx* c = r->ctx;
    if (r->nl == 0 || r->layout_version == c->layout_version) return;
    if (c->n_states < r->top_state)
        cl::fail(CL_ERR_STATE, "the request names state %d of %d loaded", r->top_state, c->n_states);
    const std::vector<int2> fl = r->lay.states();
    const long long As = c->n_sorted;
    r->ps.mma_ok = r->ps.tile_ok = false;
    pair_setup(c, fl, r->ps);
    grow(r->rho, fl.size() * As);
    grow(r->V, (size_t)r->nl * As);
    tc_reserve(c, r->lay.gram, As, v_fp32(c), rho_bytes(c) == sizeof(cx<float>));
    CL_CUDA(cudaStreamSynchronize(c->stream));
    r->layout_version = c->layout_version;
}

LaunchState launch_state(const cl_request* r) {
    const cl_ctx* c = r->ctx;
    return {c->layout_version, c->kernel_version, c->buffer_moves() + r->rho.moves + r->V.moves};
}

// Stream-ordered work of a prepared request: no allocation, no host synchronisation, no
// pageable copies -- it can be captured.
void request_enqueue(cl_request* r) {
    cl_ctx* c = r->ctx;
    if (r->nl == 0) return;  // a shard without densities
    const long long As = c->n_sorted;
    pair_launch(c, r->ps, r->rho.p);
    const bool v32 = v_fp32(c);
    run_transforms(c, r->rho.p, As, r->nl, r->V.p, As, v32);
    gram(c, r->V.p, v32, As, r->rho.p, rho_bytes(c) == sizeof(cx<float>), As, r->rows.p, r->lay.gram, As, r->o4.p);
    CL_CUDA(cudaMemcpyAsync(r->o4_host, r->o4.p, sizeof(double) * (4 * (size_t)r->nl * r->nr + 1),
                            cudaMemcpyDeviceToHost, c->stream));
}

void request_finish(cl_request* r, double* out) {
    if (r->n_shards > 1) std::memset(out, 0, sizeof(double) * 2 * (size_t)r->n_int);
    if (r->nl == 0) return;
    check_gram_slot(r->o4_host[4 * (size_t)r->nl * r->nr]);
    map_step_values(r->plan, r->values, r->o4_host, out);
}

}  // namespace

extern "C" {

int cl_request_create(cl_ctx* c, int64_t n_int, const int16_t* spec, cl_request** out) {
    return cl_request_create_shard(c, n_int, spec, 0, 1, out);
}

int cl_request_create_shard(cl_ctx* c, int64_t n_int, const int16_t* spec, int shard, int n_shards,
                            cl_request** out) {
    if (out) *out = nullptr;
    cl_request* r = nullptr;
    int st = cl::guarded([&] {
        check_ctx(c);
        check_kernel(c);
        if (!out) cl::fail(CL_ERR_ARGUMENT, "null output pointer");
        if (c->n_states == 0) cl::fail(CL_ERR_STATE, "no states loaded (call cl_set_states)");
        if (n_int <= 0 || !spec) cl::fail(CL_ERR_ARGUMENT, "invalid integral list");
        r = new cl_request();
        r->ctx = c;
        r->device = c->device;
        r->n_int = n_int;
        std::vector<std::array<int16_t, 4>> specs((size_t)n_int);
        for (int64_t i = 0; i < n_int; ++i)
            for (int k = 0; k < 4; ++k) specs[i][k] = spec[4 * i + k];
        r->plan = shard_steps(cl::orient_steps(c->n_states, specs), c->n_states, shard, n_shards);
        r->n_shards = n_shards;
        if (r->plan.empty()) {  // a shard without densities: runs produce zeros
            *out = r;
            return;
        }
        r->lay = layout_densities(r->plan, c->n_states, symmetric_blocks(c));
        r->nl = r->lay.gram.nl;
        r->nr = r->lay.gram.nr;
        r->values = step_values(r->plan, r->lay);
        for (const int2& p : r->lay.states()) r->top_state = std::max({r->top_state, p.x + 1, p.y + 1});
        const std::vector<int>& columns = r->lay.columns;
        r->rows.upload(columns.data(), columns.size(), c->stream);
        r->o4.alloc((size_t)4 * r->nl * r->nr + 1);
        CL_CUDA(cudaMallocHost(&r->o4_host, sizeof(double) * (4 * (size_t)r->nl * r->nr + 1)));
        request_layout(r);
        *out = r;
    });
    if (st != CL_OK) delete r;
    return st;
}

void cl_request_destroy(cl_request* r) {
    if (!r) return;
    cudaSetDevice(r->device);
    delete r;
}

int cl_request_run(cl_request* r, double* out) {
    return cl::guarded([&] {
        if (!r || !out) cl::fail(CL_ERR_ARGUMENT, "null argument");
        check_ctx(r->ctx);
        request_layout(r);
        request_enqueue(r);
        CL_CUDA(cudaStreamSynchronize(r->ctx->stream));
        prof_collect(r->ctx);
        r->warm = launch_state(r);
        request_finish(r, out);
    });
}

int cl_batch_create(cl_request** reqs, int n, cl_batch** out) {
    if (out) *out = nullptr;
    cl_batch* b = nullptr;
    int st = cl::guarded([&] {
        if (!reqs || n <= 0 || !out) cl::fail(CL_ERR_ARGUMENT, "invalid batch");
        const int dev = reqs[0]->ctx->device;
        for (int i = 0; i < n; ++i) {
            if (!reqs[i]) cl::fail(CL_ERR_ARGUMENT, "null request");
            if (reqs[i]->ctx->device != dev) cl::fail(CL_ERR_ARGUMENT, "all requests of a batch must share one device");
            for (int j = 0; j < i; ++j)
                if (reqs[j]->ctx == reqs[i]->ctx)
                    cl::fail(CL_ERR_ARGUMENT, "requests of one batch need distinct contexts (one stream each)");
        }
        CL_CUDA(cudaSetDevice(dev));
        b = new cl_batch();
        b->device = dev;
        b->reqs.assign(reqs, reqs + n);
        CL_CUDA(cudaStreamCreateWithFlags(&b->master, cudaStreamNonBlocking));
        CL_CUDA(cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming));
        CL_CUDA(cudaEventCreate(&b->t0));
        CL_CUDA(cudaEventCreate(&b->t1));
        b->joins.resize(n);
        for (auto& e : b->joins) CL_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        *out = b;
    });
    if (st != CL_OK) delete b;
    return st;
}

void cl_batch_destroy(cl_batch* b) {
    if (!b) return;
    cudaSetDevice(b->device);
    delete b;
}

int cl_batch_run(cl_batch* b, double** outs) {
    return cl::guarded([&] {
        if (!b || !outs) cl::fail(CL_ERR_ARGUMENT, "null argument");
        CL_CUDA(cudaSetDevice(b->device));
        for (cl_request* r : b->reqs) request_layout(r);
        // captured anew when a later call of one of the contexts has moved a buffer, loaded another layout or
        // set another kernel
        bool current = b->exec != nullptr;
        for (size_t i = 0; current && i < b->reqs.size(); ++i) current = b->captured[i] == launch_state(b->reqs[i]);
        if (!current) {
            b->drop_graph();
            b->captured.clear();
            // one eager run of every request sizes every buffer and sets every kernel
            // attribute; then the whole batch is captured once as parallel branches
            for (cl_request* r : b->reqs)
                if (!(r->warm == launch_state(r))) {
                    request_enqueue(r);
                    CL_CUDA(cudaStreamSynchronize(r->ctx->stream));
                    prof_collect(r->ctx);
                    r->warm = launch_state(r);
                }
            // contexts that profile record their launch events inside the graph
            b->prof.assign(b->reqs.size(), {});
            for (size_t i = 0; i < b->reqs.size(); ++i) {
                cl_ctx* c = b->reqs[i]->ctx;
                if (c->profiling) {
                    c->prof_sink = &b->prof[i];
                    c->prof_owned = &b->prof_events;
                }
            }
            CL_CUDA(cudaStreamBeginCapture(b->master, cudaStreamCaptureModeRelaxed));
            CL_CUDA(cudaEventRecord(b->fork, b->master));
            for (size_t i = 0; i < b->reqs.size(); ++i) {
                cl_request* r = b->reqs[i];
                CL_CUDA(cudaStreamWaitEvent(r->ctx->stream, b->fork, 0));
                request_enqueue(r);
                CL_CUDA(cudaEventRecord(b->joins[i], r->ctx->stream));
                CL_CUDA(cudaStreamWaitEvent(b->master, b->joins[i], 0));
            }
            CL_CUDA(cudaStreamEndCapture(b->master, &b->graph));
            for (cl_request* r : b->reqs) {
                r->ctx->prof_sink = nullptr;
                r->ctx->prof_owned = nullptr;
            }
            CL_CUDA(cudaGraphInstantiate(&b->exec, b->graph, 0));
            for (const cl_request* r : b->reqs) b->captured.push_back(launch_state(r));
        }
        CL_CUDA(cudaEventRecord(b->t0, b->master));
        CL_CUDA(cudaGraphLaunch(b->exec, b->master));
        CL_CUDA(cudaEventRecord(b->t1, b->master));
        CL_CUDA(cudaStreamSynchronize(b->master));
        float ms = 0;
        CL_CUDA(cudaEventElapsedTime(&ms, b->t0, b->t1));
        b->last_ms = ms;
        for (size_t i = 0; i < b->reqs.size(); ++i) {
            cl_ctx* c = b->reqs[i]->ctx;
            if (!c->profiling) continue;
            for (const auto& e : b->prof[i]) {
                float kms = 0;
                CL_CUDA(cudaEventElapsedTime(&kms, e.a, e.b));
                c->prof_ms[e.cls] += kms;
                c->prof_bytes[e.cls] += e.bytes;
                c->prof_launches[e.cls] += 1;
            }
        }
        for (size_t i = 0; i < b->reqs.size(); ++i) request_finish(b->reqs[i], outs[i]);
    });
}

int cl_batch_last_ms(cl_batch* b, double* ms) {
    return cl::guarded([&] {
        if (!b || !ms) cl::fail(CL_ERR_ARGUMENT, "null argument");
        *ms = b->last_ms;
    });
}

int cl_autotune_report(char* buf, int64_t len, int64_t* needed) {
    // precision and grid of a tuning key: "fp32" / "fp64" on the real grid, "fp32 sub-lattice" /
    // "fp64 sub-lattice" on the virtual grid of the sub-lattice forms
    const auto form_name = [](int f) {
        static const char* n[4] = {"fp64", "fp32", "fp64 sub-lattice", "fp32 sub-lattice"};
        return n[f & 3];
    };
    return cl::guarded([&] {
        static const char* names[clp::kNumPasses] = {"x_forward", "y_forward", "z_pass",   "y_inverse",
                                                     "x_inverse", "xy_forward", "xy_inverse"};
        std::string out;
        {
            std::lock_guard<std::mutex> g(g_tune_mu);
            for (const auto& kv : g_tune) {
                char line[256];
                const char* pn = names[kv.first.pass];
                if (kv.first.pass == clp::kXYFwd || kv.first.pass == clp::kXYInv) {
                    const char* ch = kv.second.v.split ? "fused plane pass" : "separate passes";
                    if (kv.second.candidates == 0)
                        std::snprintf(line, sizeof line, "%s %s %dx%dx%d: %s, from CL_TUNE_FILE\n", pn,
                                      form_name(kv.first.fp32), kv.first.nx, kv.first.ny, kv.first.nz, ch);
                    else
                        std::snprintf(line, sizeof line,
                                      "%s %s %dx%dx%d: %s, 2 candidates, fused %.4f ms, separate %.4f ms\n", pn,
                                      form_name(kv.first.fp32), kv.first.nx, kv.first.ny, kv.first.nz, ch,
                                      kv.second.ms, kv.second.ms_default);
                    out += line;
                    continue;
                }
                const char* pr = form_name(kv.first.fp32);
                const char* sp = kv.second.v.split ? "swapped" : "balanced";
                const char* ln = kv.second.v.half ? "half" : "default";
                const char* pd = kv.second.v.pad ? ", padded tile" : "";
                if (kv.second.candidates == 0)
                    std::snprintf(line, sizeof line, "%s %s %dx%dx%d: split %s, lines %s%s, from CL_TUNE_FILE\n", pn,
                                  pr, kv.first.nx, kv.first.ny, kv.first.nz, sp, ln, pd);
                else
                    std::snprintf(line, sizeof line,
                                  "%s %s %dx%dx%d: split %s, lines %s%s, %d candidates, %.4f ms (default %.4f ms)\n",
                                  pn, pr, kv.first.nx, kv.first.ny, kv.first.nz, sp, ln, pd, kv.second.candidates,
                                  kv.second.ms, kv.second.ms_default);
                out += line;
            }
        }
        if (needed) *needed = (int64_t)out.size() + 1;
        if (buf && len > 0) {
            const size_t n = std::min<size_t>(out.size(), (size_t)len - 1);
            std::memcpy(buf, out.data(), n);
            buf[n] = 0;
        }
    });
}

int cl_form_info(cl_ctx* c, int info[8]) {
    return cl::guarded([&] {
        check_ctx(c);
        if (!info) cl::fail(CL_ERR_ARGUMENT, "null output");
        const Sublattice& sl = c->sl;
        info[0] = sl.active ? 1 : 0;
        info[1] = sl.active ? sl.m : 0;
        info[2] = sl.active ? sl.S : 0;
        info[3] = sl.active && sl.zb ? 1 : 0;
        for (int d = 0; d < 3; ++d) info[4 + d] = sl.active ? sl.pad[d] : 0;
        info[7] = sl.active ? sl.table.nh : 0;
    });
}

int cl_last_timings(cl_ctx* c, double t[4]) {
    return cl::guarded([&] {
        if (!c || !t) cl::fail(CL_ERR_ARGUMENT, "null argument");
        for (int i = 0; i < 4; ++i) t[i] = c->timings[i];
    });
}

int cl_fft3d(int nx, int ny, int nz, int batch, int sign, int fp32, double* data) {
    return cl::guarded([&] {
        if (nx <= 0 || ny <= 0 || nz <= 0 || batch <= 0 || !data || (sign != -1 && sign != 1))
            cl::fail(CL_ERR_ARGUMENT, "invalid FFT arguments");
        cl_ctx* raw = nullptr;
        if (cl_create(&raw, nx, ny, nz, 1, 1, 1, fp32 ? CL_MODE_FP32_ROUNDS : CL_MODE_FP64_PLAIN) != CL_OK)
            cl::fail(CL_ERR_ARGUMENT, "%s", cl_last_error());
        std::unique_ptr<cl_ctx> c(raw);
        const long long M = c->M;
        const size_t n = (size_t)M * batch;
        DevBuf<cx<double>> d64;
        d64.upload(reinterpret_cast<const cx<double>*>(data), n, c->stream);
        auto run = [&](auto tag) {
            using T = decltype(tag);
            DevBuf<cx<T>> dT;
            cx<T>* buf;
            if constexpr (sizeof(T) == 4) {
                dT.alloc(n);
                clk::k_narrow<float><<<grid_for((long long)n), 256, 0, c->stream>>>(d64.p, dT.p, (long long)n);
                CL_LAUNCHED();
                buf = dT.p;
            } else {
                buf = d64.p;
            }
            const Axis& X = c->ax[0];
            const Axis& Y = c->ax[1];
            const Axis& Z = c->ax[2];
            const cx<T>* twx = sizeof(T) == 4 ? (const cx<T>*)X.tw32.p : (const cx<T>*)X.tw64.p;
            const cx<T>* twy = sizeof(T) == 4 ? (const cx<T>*)Y.tw32.p : (const cx<T>*)Y.tw64.p;
            const cx<T>* twz = sizeof(T) == 4 ? (const cx<T>*)Z.tw32.p : (const cx<T>*)Z.tw64.p;
            const int nrows = ny * nz;
            const XTile xt = x_tile<T>(nx, nrows);
            const LTile yt = l_tile<T>(ny, false);
            const LTile zt = l_tile<T>(nz, false);
            const int xblocks = (nrows + xt.rows - 1) / xt.rows;
            const int ychunks = (nx + yt.W - 1) / yt.W;
            const long long nxy = (long long)nx * ny;
            const long long zblocks = (nxy + zt.W - 1) / zt.W;
            // the x and y passes take the grid index from blockIdx.y (at most 65535): slices of grids
            for (int b0 = 0; b0 < batch; b0 += 65535) {
                const int nb = std::min(65535, batch - b0);
                cx<T>* slice = buf + (long long)b0 * M;
                if (sign < 0) {
                    ensure_smem(clk::k_xpass<-1, T>, xt.smem);
                    ensure_smem(clk::k_ypass<-1, T>, yt.smem);
                    clk::k_xpass<-1, T><<<dim3(xblocks, nb), 256, xt.smem, c->stream>>>(slice, M, X.plan, twx, nx,
                                                                                       nrows, xt.rows, xt.ld);
                    CL_LAUNCHED();
                    clk::k_ypass<-1, T><<<dim3(ychunks * nz, nb), 256, yt.smem, c->stream>>>(slice, M, Y.plan, twy,
                                                                                            nx, ny, yt.W, ychunks);
                    CL_LAUNCHED();
                } else {
                    ensure_smem(clk::k_xpass<+1, T>, xt.smem);
                    ensure_smem(clk::k_ypass<+1, T>, yt.smem);
                    clk::k_xpass<+1, T><<<dim3(xblocks, nb), 256, xt.smem, c->stream>>>(slice, M, X.plan, twx, nx,
                                                                                       nrows, xt.rows, xt.ld);
                    CL_LAUNCHED();
                    clk::k_ypass<+1, T><<<dim3(ychunks * nz, nb), 256, yt.smem, c->stream>>>(slice, M, Y.plan, twy,
                                                                                            nx, ny, yt.W, ychunks);
                    CL_LAUNCHED();
                }
            }
            ensure_smem(clk::k_zpass<T>, zt.smem);
            clk::k_zpass<T><<<(unsigned)zblocks, 256, zt.smem, c->stream>>>(buf, M, Z.plan, twz, nullptr, nxy, nz,
                                                                             zt.W, batch, sign, 0u, 0LL);
            CL_LAUNCHED();
            if constexpr (sizeof(T) == 4) {
                clk::k_widen<float><<<grid_for((long long)n), 256, 0, c->stream>>>(dT.p, d64.p, (long long)n);
                CL_LAUNCHED();
            }
            CL_CUDA(cudaMemcpyAsync(data, d64.p, n * sizeof(cx<double>), cudaMemcpyDeviceToHost, c->stream));
            CL_CUDA(cudaStreamSynchronize(c->stream));
        };
        if (fp32)
            run(float{});
        else
            run(double{});
    });
}

}  // extern "C"
