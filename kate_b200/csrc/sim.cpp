// Device simulator. See sim.hpp.
#include "sim.hpp"

#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <random>

#include "devcache.hpp"
#include "jit.hpp"
#include "launch.hpp"

namespace kate {

namespace {
constexpr double kPi = 3.1415926535897932384626433;
constexpr double kSqrt2 = 1.4142135623730951;

std::string cuda_err(const char* what, cudaError_t e) {
    return std::string(what) + ": " + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")";
}
#define KCHECK(call)                                              \
    do {                                                          \
        cudaError_t e_ = (call);                                  \
        if (e_ != cudaSuccess) return cuda_err(#call, e_);        \
    } while (0)
}  // namespace

struct SimImpl {
    int device = 0;
    int n = 0;
    int precision = 0;
    Program prog;
    Plan plan;
    PlanOptions opt;
    void* d_state = nullptr;
    char* d_ws = nullptr;      // the workspace the pointers below lie in
    DevOp* d_ops = nullptr;
    DevOp* d_sops = nullptr;   // shared-memory ops of register-staged programs
    void* d_pool = nullptr;
    void* d_part = nullptr;
    void* d_bimg = nullptr;   // complex64 block operand images
    int* d_err = nullptr;     // set by kernels whose bounded waits gave up
    // Measurement results: the error flag, then (at +16 bytes) the bit sums,
    // or samples. Pinned host memory that kernels write directly, or, when
    // none is left, device memory copied to `host_out` after the kernel.
    char* pinned = nullptr;
    char* d_res = nullptr;
    std::vector<char> host_out;
    char* d_samp = nullptr;   // sampling workspace, kept once used
    size_t samp_bytes = 0;
    void* d_norm = nullptr;   // complex64: renormalisation scratch and result
    bool renormed = false;    // a complex64 run has been renormalised
    std::vector<DevPass> hpasses;
    cudaStream_t stream = nullptr;
    std::vector<int> phys;  // current layout: logical -> physical
    bool has_state = false;
    int grid = 0;
    int tile_grid = 0;
    int nbuf = 1;  // tile kernel buffering (1: two CTAs per SM, 2: one CTA, prefetching)
    int ws_grid = 0;
    std::vector<char> ws_ok;  // pass i runs on the warp-specialised complex128 tile kernel
    std::vector<void*> jit_fn;  // pass i runs on its pass-specialised kernel (complex128)
    std::vector<std::vector<double2>> jit_mats;  // its matrices (kernel parameter)
    // Shared-memory ops of pass i's program.
    const DevOp* sops_of(size_t i) const { return plan.smem_ops.data() + plan.passes[i].prog->sop0; }
    void* jit_fn0 = nullptr;    // pass 0 generating its input |0...0> (no initialisation pass)
    bool zero_start = false;    // the run being enqueued starts with jit_fn0
    bool basis0 = false;        // the run being enqueued starts from |0...0>
    void* jit_fnP = nullptr;    // pass 0 computing a product-state input (no initialisation pass)
    bool prod_start = false;    // the run being enqueued starts with jit_fnP and prod_tab
    ProdTab prod_tab{};
    int jit_grid_n = 0;
    // States of fewer than 12 qubits: every pass's program, run by one CTA in
    // one launch (BatchProg headers, then the programs).
    bool small = false;
    char* d_small = nullptr;
    int small_start = 1;  // the run being enqueued: 1 from |0...0>, 2 from small_prod
    ProductInit small_prod{};

    cudaError_t launch_small_range(int p0, int p1, int init, bool sums, cudaStream_t st) {
        return launch_small(d_state, precision, n, small_reg_bits(n), (const BatchProg*)d_small, p0, p1, d_small, d_sops, d_pool,
                            !plan.smem_ops.empty(), init, small_prod, sums ? res_sums() : nullptr, st);
    }
    // The headers and programs as one blob.
    std::vector<char> small_blob() const {
        std::vector<char> blob(plan.passes.size() * sizeof(BatchProg));
        auto put = [&](const void* p, size_t bytes) {
            blob.resize((blob.size() + 15) & ~size_t(15));
            const size_t at = blob.size();
            blob.insert(blob.end(), (const char*)p, (const char*)p + bytes);
            return (uint64_t)at;
        };
        for (size_t i = 0; i < plan.passes.size(); i++) {
            const PassProg& P = *plan.passes[i].sprog;
            BatchProg b{};
            b.m = P.m;
            b.nops = P.nops;
            b.nmats = P.nmats;
            b.nstages = P.nstages;
            b.sop0 = P.sop0;
            b.ops_off = put(P.ops, sizeof(SOp) * (size_t)P.nops);
            b.mats_off = put(P.mats, 16 * (size_t)P.nmats);
            b.stab_off = put(P.stab, sizeof(P.stab[0]) * (size_t)P.nstages);
            std::memcpy(blob.data() + i * sizeof(BatchProg), &b, sizeof b);
        }
        blob.resize(((blob.size() + 15) & ~size_t(15)) + 16);
        return blob;
    }

    // Launches pass i of the plan on stream st.
    cudaError_t launch_pass(size_t i, cudaStream_t st) {
        if (small) return launch_small_range((int)i, (int)i + 1, 0, false, st);
        const PlannedPass& p = plan.passes[i];
        // Only the cosets that are not zero (a first pass that generates
        // |0...0> writes them all). A 30-qubit layered circuit reaches its
        // last qubits in the fourth of 20 passes, an SU(4) brickwork in
        // complex64 in its ninth of 26: 200.8 -> 182.4 and 94.4 -> 73.5 ms a
        // run; 23 qubits in three passes 396 -> 263 us.
        const int idle = basis0 && !(i == 0 && zero_start) ? p.idle : 0;
        if (p.bprog) {
            BlockProg b = *p.bprog;
            b.ncb -= idle;
            return launch_block_c64(d_state, b, d_bimg, i == 0 && zero_start, d_err, block_c64_grid(n - idle, device),
                                    sum_norm && i + 1 == plan.passes.size() ? d_norm : nullptr, st);
        }
        if (i == 0 && zero_start && jit_fn0) return jit_launch(jit_fn0, d_state, jit_mats[0], nullptr, jit_grid_n, st);
        if (i == 0 && prod_start && jit_fnP) return jit_launch(jit_fnP, d_state, jit_mats[0], &prod_tab, jit_grid_n, st);
        if (p.prog && i < jit_fn.size() && jit_fn[i])
            return jit_launch(jit_fn[i], d_state, jit_mats[i], nullptr, jit_grid_n >> idle, st);
        if (p.prog && i < ws_ok.size() && ws_ok[i]) return launch_tile_ws(d_state, *p.prog, d_err, ws_grid, st);
        if (p.prog && idle) {
            PassProg q = *p.prog;
            q.ncb -= idle;
            return launch_tile(d_state, precision, q, d_sops, d_pool, std::min(tile_grid, 1 << q.ncb), nbuf, st);
        }
        if (p.prog) return launch_tile(d_state, precision, *p.prog, d_sops, d_pool, tile_grid, nbuf, st);
        return launch_pass_generic(d_state, precision, hpasses[i], d_ops, d_pool, grid, st);
    }
    bool sum_norm = false;  // the pass being enqueued, if it is the last, leaves ||psi||^2 in d_norm
    // Whether the last pass can: it is one of tensor-core blocks.
    bool last_sums_norm() const { return !small && !plan.passes.empty() && plan.passes.back().bprog; }
    // Whether the first pass generates |0...0> itself.
    bool starts_from_zero() const { return jit_fn0 || (!plan.passes.empty() && plan.passes[0].bprog); }

    uint64_t dim() const { return 1ull << n; }
    size_t amp_bytes() const { return precision == 0 ? 16 : 8; }

    // Target layout for readback: label x at physical bit x.
    std::vector<int> label_layout() const {
        std::vector<int> t(n);
        for (int x = 0; x < n; x++) t[plan.label_to_logical[x]] = x;
        return t;
    }
    // Physical bit of program label x.
    int phys_of_label(int x) const { return phys[plan.label_to_logical[x]]; }

    std::string run_relayout(const std::vector<int>& target) {
        if (phys == target) return "";
        std::vector<PlannedPass> pp = plan_relayout(n, phys, target, opt);
        for (auto& p : pp) {
            DevPass d = to_devpass(n, p, 0);
            int grid_r = generic_pass_grid(n, d.m, device);
            KCHECK(launch_pass_generic(d_state, precision, d, d_ops, d_pool, grid_r, stream));
        }
        phys = target;
        return "";
    }

    // Where a measurement's kernels write (flag first) and its bytes.
    size_t res_bytes() const { return 16 + std::max<size_t>(25, 1 + 2 * (size_t)n) * sizeof(double2); }
    char* res() const { return pinned ? pinned : d_res; }
    void* res_sums() const { return res() + 16; }
    int* res_flag() const { return (int*)res(); }

    // Waits for the bit sums queued on the simulator's stream and the work
    // before them; *out points at the sums on the host. `check`: the flag was
    // written with them and is looked at.
    std::string fetch(const char** out, bool check) {
        if (!pinned) {
            host_out.resize(res_bytes());
            KCHECK(cudaMemcpyAsync(host_out.data(), d_res, host_out.size(), cudaMemcpyDeviceToHost, stream));
        }
        KCHECK(cudaStreamSynchronize(stream));
        const char* r = pinned ? pinned : host_out.data();
        int flag = 0;
        if (check) std::memcpy(&flag, r, sizeof flag);
        if (flag) return timed_out();
        *out = r + 16;
        return "";
    }
    std::string timed_out() {
        cudaMemset(d_err, 0, sizeof(int));
        return "timed out: a bounded device wait gave up (tensor-core completion not observed)";
    }

    // Sums over amplitudes (kind 0, two doubles per value) or probabilities
    // (kind 1, one): *sums holds the total, then the sums with physical bit b
    // 0 and 1 at values 1 + 2b and 2 + 2b.
    std::string bit_sums(int kind, const double** sums) {
        KCHECK(launch_bitsums(d_state, precision, n, kind, d_part, res_sums(), nullptr, nullptr, stream));
        const char* r = nullptr;
        std::string e = fetch(&r, false);
        *sums = (const double*)r;
        return e;
    }

    // The reference's measurement from the amplitude sums
    // (HIPcode/simulator.hpp:519-535 with its Complex division, norm and
    // angle, backendagnosticcode/basic_host_types.hpp:28-57).
    void proba_from_sums(const double* sums, double* out) const {
        const double p = std::pow(kSqrt2, (double)n);
        auto cdiv = [](double ar, double ai, double br, double bi, double& rr, double& ri) {
            double d = br * br + bi * bi;
            rr = (ar * br + ai * bi) / d;
            ri = (br * ai - ar * bi) / d;
        };
        for (int x = 0; x < n; x++) {
            const int b = phys_of_label(x);
            const double *s0 = sums + 2 * (1 + 2 * b), *s1 = s0 + 2;
            double v0r, v0i, v1r, v1i;
            cdiv(s0[0], s0[1], p, 0.0, v0r, v0i);
            cdiv(s1[0], s1[1], p, 0.0, v1r, v1i);
            double n0 = std::sqrt(v0r * v0r + v0i * v0i), n1 = std::sqrt(v1r * v1r + v1i * v1i);
            double teta, phi;
            if (n0 < 0.0000000000001) {
                teta = 1;
                phi = 0;
            } else if (n1 < 0.00000000000001) {
                teta = 0;
                phi = 0;
            } else {
                teta = std::atan(n1 / n0) / (kPi / 2);
                double qr, qi;
                cdiv(v1r, v1i, v0r, v0i, qr, qi);
                phi = std::atan(qi / qr);
            }
            const int o = plan.final_inverse_permutation.empty() ? x : plan.final_inverse_permutation[x];
            out[2 * o] = teta;
            out[2 * o + 1] = phi;
        }
    }
};

std::string Simulator::create(const Program& prog_in, int precision, int device, Simulator** out) {
    if (precision != 0 && precision != 1) return "unknown precision";
    if (prog_in.nqbits < 1 || prog_in.nqbits > 34) return "the device simulator supports 1 to 34 qubits";
    auto* impl = new SimImpl();
    auto fail = [&](const std::string& e) {
        auto* s = new Simulator();
        s->d_ = impl;
        delete s;
        return e;
    };
    impl->device = device;
    impl->n = prog_in.nqbits;
    impl->precision = precision;
    impl->prog = prog_in;
    if (impl->prog.instructions.empty()) {
        std::string e = pass_compile_default(impl->prog, 0, impl->prog.nqbits);
        if (!e.empty()) return fail(e);
    }
    impl->opt = simulator_plan_options(impl->n, precision);
    std::string e = build_plan(impl->prog, impl->opt, &impl->plan);
    if (!e.empty()) return fail(e);

    cudaError_t ce = cudaSetDevice(device);
    if (ce != cudaSuccess) return fail(cuda_err("cudaSetDevice", ce));
    ce = stream_take(&impl->stream, device);
    if (ce != cudaSuccess) return fail(cuda_err("cudaStreamCreate", ce));
    // One workspace holds what the kernels read (uploaded in one copy) and
    // the measurement's partials.
    std::vector<char> up;
    auto put = [&](const void* p, size_t bytes) {
        const size_t at = (up.size() + 255) & ~size_t(255);
        up.resize(at + std::max<size_t>(bytes, 16));
        if (p && bytes) std::memcpy(up.data() + at, p, bytes);
        return at;
    };
    std::vector<DevOp> ops;
    for (auto& p : impl->plan.passes) {
        impl->hpasses.push_back(to_devpass(impl->n, p, (int)ops.size()));
        ops.insert(ops.end(), p.ops.begin(), p.ops.end());
    }
    const size_t o_err = put(nullptr, sizeof(int));
    const size_t o_norm = precision == 1 ? put(nullptr, renorm_scratch_bytes()) : 0;
    const size_t o_ops = put(ops.data(), ops.size() * sizeof(DevOp));
    const size_t o_sops = put(impl->plan.smem_ops.data(), impl->plan.smem_ops.size() * sizeof(DevOp));
    const size_t o_pool = put(impl->plan.pool.data(), impl->plan.pool.size() * sizeof(Cx));
    const size_t o_bimg = put(impl->plan.bimg.data(), impl->plan.bimg.size());
    impl->small = impl->n < KATE_TILE_BITS;
    for (const auto& p : impl->plan.passes) impl->small = impl->small && p.sprog;
    for (const auto& p : impl->plan.passes)
        if (!p.prog && !p.bprog && !impl->small && p.ops.size() != p.gates.size())
            return fail("internal: a pass has neither a program nor its device ops");
    size_t o_small = 0;
    if (impl->small) {
        const std::vector<char> blob = impl->small_blob();
        o_small = put(blob.data(), blob.size());
    }
    const BitSumShape sh = bitsum_shape(impl->n);
    const size_t o_part = (up.size() + 255) & ~size_t(255);
    const size_t part_bytes = sh.grid > 1 ? (size_t)sh.grid * sh.nout * 2 * sizeof(double) : 16;
    ce = cached_malloc((void**)&impl->d_ws, o_part + part_bytes, device);
    if (ce != cudaSuccess) return fail(cuda_err("cudaMalloc(workspace)", ce));
    // On the simulator's stream and waited for: a run may be queued on any stream.
    ce = cudaMemcpyAsync(impl->d_ws, up.data(), up.size(), cudaMemcpyHostToDevice, impl->stream);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(impl->stream);
    if (ce != cudaSuccess) return fail(cuda_err("upload", ce));
    impl->d_err = (int*)(impl->d_ws + o_err);
    impl->d_norm = precision == 1 ? impl->d_ws + o_norm : nullptr;
    impl->d_ops = (DevOp*)(impl->d_ws + o_ops);
    impl->d_sops = (DevOp*)(impl->d_ws + o_sops);
    impl->d_pool = impl->d_ws + o_pool;
    impl->d_bimg = impl->d_ws + o_bimg;
    impl->d_small = impl->d_ws + o_small;
    impl->d_part = impl->d_ws + o_part;
    if (impl->small) {
        ce = small_prepare(device);
        if (ce != cudaSuccess) return fail(cuda_err("one-CTA kernel", ce));
    }
    impl->pinned = (char*)pinned_take();
    if (!impl->pinned) {
        ce = cudaMalloc(&impl->d_res, impl->res_bytes());
        if (ce != cudaSuccess) return fail(cuda_err("cudaMalloc(results)", ce));
    }
    ce = cached_malloc(&impl->d_state, impl->dim() * impl->amp_bytes(), device);
    if (ce != cudaSuccess) return fail(cuda_err("cudaMalloc(state)", ce));
    impl->grid = generic_pass_grid(impl->n, std::min(impl->opt.max_tile, impl->n), device);
    if (const char* e = std::getenv("KATE_TILE_NBUF")) {
        const int v = std::atoi(e);
        impl->nbuf = v == 2 ? 2 : v == 3 ? 3 : 1;
    }
    if (impl->n >= KATE_TILE_BITS) {
        impl->tile_grid = tile_pass_grid(impl->n, device, impl->nbuf, precision);
        const char* jv = std::getenv("KATE_JIT");
        if (precision == 0 && !(jv && std::atoi(jv) == 0)) {
            // Pass-specialised kernels for every register-staged pass whose
            // program the generator takes; the others keep the interpreter.
            // Two CTAs per SM (at most 128 registers). KATE_JIT_OCC=3 asks
            // for three (at most 80 registers; a kernel that would spill
            // stays at two): measured slower on the layered workload (54.6
            // against 56.8 layers/s), kept as a tuning option.
            const char* oe = std::getenv("KATE_JIT_OCC");
            const int occ_force = oe ? std::atoi(oe) : 0;
            const int occ_first = occ_force == 3 ? 3 : 2;
            // Kernels per (pass, form): form 0 loads its input, form 1 (pass
            // 0) generates |0...0>, form 2 (pass 0) computes a product state.
            // Kernels compiled before for the same pass shape are found by
            // key; only the others get their source generated.
            std::vector<size_t> idx;
            std::vector<int> forms;
            std::vector<std::string> todo;
            std::vector<void*> fns;
            std::vector<std::string> keys;
            std::vector<size_t> miss;
            auto want = [&](size_t i, int form, int occ) {
                std::string key = jit_pass_key(*impl->plan.passes[i].prog, impl->sops_of(i), form, occ);
                void* f = jit_find(device, key);
                idx.push_back(i);
                forms.push_back(form);
                if (!f) {
                    miss.push_back(fns.size());
                    todo.push_back(jit_pass_source(*impl->plan.passes[i].prog, impl->sops_of(i), nullptr, form, occ));
                }
                fns.push_back(f);
                keys.push_back(std::move(key));
            };
            for (size_t i = 0; i < impl->plan.passes.size(); i++) {
                const PlannedPass& p = impl->plan.passes[i];
                if (!p.prog || p.bprog) continue;
                want(i, 0, occ_first);
            }
            if (!idx.empty() && idx[0] == 0) {
                want(0, 1, occ_first);
                want(0, 2, occ_first);
            }
            auto compile_missing = [&]() -> std::string {
                // Sources the generator declined stay null: those passes keep the interpreter.
                std::vector<std::string> srcs;
                std::vector<size_t> at;
                for (size_t m = 0; m < miss.size(); m++)
                    if (!todo[m].empty()) {
                        srcs.push_back(std::move(todo[m]));
                        at.push_back(miss[m]);
                    }
                std::vector<void*> got;
                std::string je = jit_compile(device, srcs, &got);
                if (!je.empty()) return je;
                for (size_t m = 0; m < at.size(); m++) {
                    fns[at[m]] = got[m];
                    jit_remember(device, keys[at[m]], got[m]);
                }
                miss.clear();
                todo.clear();
                return "";
            };
            std::string je = compile_missing();
            if (!je.empty()) return fail("pass kernel compilation: " + je);
            if (occ_first == 3) {
                // A kernel that spills at three CTAs per SM goes back to two.
                for (size_t k = 0; k < fns.size(); k++)
                    if (fns[k] && jit_local_bytes(fns[k]) != 0) {
                        std::string key = jit_pass_key(*impl->plan.passes[idx[k]].prog, impl->sops_of(idx[k]), forms[k], 2);
                        void* f = jit_find(device, key);
                        if (!f) {
                            miss.push_back(k);
                            todo.push_back(jit_pass_source(*impl->plan.passes[idx[k]].prog, impl->sops_of(idx[k]), nullptr,
                                                           forms[k], 2));
                        }
                        fns[k] = f;
                        keys[k] = std::move(key);
                    }
                je = compile_missing();
                if (!je.empty()) return fail("pass kernel compilation: " + je);
            }
            impl->jit_fn.assign(impl->plan.passes.size(), nullptr);
            impl->jit_mats.resize(impl->plan.passes.size());
            for (size_t k = 0; k < idx.size(); k++) {
                if (!fns[k]) continue;
                if (forms[k] == 0) {
                    impl->jit_fn[idx[k]] = fns[k];
                    impl->jit_mats[idx[k]] = jit_pass_mats(*impl->plan.passes[idx[k]].prog, impl->sops_of(idx[k]),
                                                           impl->plan.pool.data());
                }
                else if (forms[k] == 1) impl->jit_fn0 = fns[k];
                else impl->jit_fnP = fns[k];
            }
            // The start forms only serve when pass 0 itself has a kernel.
            if (impl->jit_fn.empty() || !impl->jit_fn[0]) impl->jit_fn0 = impl->jit_fnP = nullptr;
            impl->jit_grid_n = jit_grid(impl->n - KATE_TILE_BITS, device);
        }
        const char* ws = std::getenv("KATE_TILE_WS");
        if (precision == 0 && ws && std::atoi(ws) == 1) {
            impl->ws_grid = tile_ws_grid(impl->n, device);
            impl->ws_ok.assign(impl->plan.passes.size(), 0);
            for (size_t i = 0; i < impl->plan.passes.size(); i++) {
                const PlannedPass& p = impl->plan.passes[i];
                impl->ws_ok[i] = p.prog && !p.bprog && tile_ws_applies(*p.prog);
            }
        }
        if (precision == 1) block_c64_grid(impl->n, device);  // sets the kernel's shared memory limit
    }
    impl->phys.resize(impl->n);
    std::iota(impl->phys.begin(), impl->phys.end(), 0);
    auto* s = new Simulator();
    s->d_ = impl;
    *out = s;
    return "";
}

Simulator::~Simulator() {
    if (!d_) return;
    cudaSetDevice(d_->device);
    // Nothing of this simulator is in use once the device is idle.
    const bool idle = device_idle();
    cached_free(d_->d_state, d_->device, idle);
    cached_free(d_->d_ws, d_->device, idle);
    pinned_give(d_->pinned);
    cudaFree(d_->d_res);
    cudaFree(d_->d_samp);
    if (idle) stream_give(d_->stream, d_->device);
    else if (d_->stream) cudaStreamDestroy(d_->stream);
    delete d_;
}

int Simulator::nqbits() const { return d_->n; }
int Simulator::precision() const { return d_->precision; }
const Plan& Simulator::plan() const { return d_->plan; }

std::string Simulator::run_async(void* stream_in, const double* tp) {
    SimImpl& S = *d_;
    KCHECK(cudaSetDevice(S.device));
    cudaStream_t st = stream_in ? (cudaStream_t)stream_in : S.stream;
    std::string e = enqueue_init(st, tp);
    if (!e.empty()) return e;
    e = enqueue_passes(st);
    if (!e.empty()) return e;
    if (st != S.stream) {
        // Order later library work on the simulator's stream after the caller's.
        cudaEvent_t ev;
        KCHECK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        KCHECK(cudaEventRecord(ev, st));
        KCHECK(cudaStreamWaitEvent(S.stream, ev, 0));
        cudaEventDestroy(ev);
    }
    return "";
}

std::string Simulator::enqueue_init(void* stream, const double* tp) {
    SimImpl& S = *d_;
    cudaStream_t st = (cudaStream_t)stream;
    S.basis0 = !tp;
    if (tp) {
        // execute(proba_state&): product state, qubit i placed at label
        // initial_permutation[i] (CPUcode/simulator.hpp:139-162).
        ProductInit P{};
        P.n = S.n;
        for (int i = 0; i < S.n; i++) {
            double c0 = std::cos(tp[2 * i] * kPi / 2), s0 = std::sin(tp[2 * i] * kPi / 2);
            double er = std::cos(tp[2 * i + 1]), ei = std::sin(tp[2 * i + 1]);
            int lab = S.plan.initial_permutation.empty() ? i : S.plan.initial_permutation[i];
            P.v[0][lab][0] = c0;
            P.v[0][lab][1] = 0.0;
            P.v[1][lab][0] = er * s0;
            P.v[1][lab][1] = ei * s0;
        }
        S.prod_start = false;
        if (S.small) {
            S.small_prod = P;
            S.small_start = 2;
            return "";
        }
        if (S.jit_fnP && !S.hpasses.empty()) {
            // The first pass computes the product state itself (no
            // initialisation pass, and the state is not read).
            for (int b = 0; b < 2; b++)
                for (int p = 0; p < S.n; p++) S.prod_tab.v[b][p] = make_double2(P.v[b][p][0], P.v[b][p][1]);
            S.prod_start = true;
            S.zero_start = false;
            return "";
        }
        KCHECK(launch_init_product(S.d_state, S.n, P, S.precision, st));
    } else if (S.small) {
        S.small_start = 1;
        return "";
    } else if (S.starts_from_zero()) {
        // The first pass writes the whole state from |0...0> itself.
        S.zero_start = true;
        S.prod_start = false;
        return "";
    } else {
        KCHECK(launch_set_basis0(S.d_state, S.dim(), S.precision, st));
    }
    S.zero_start = false;
    S.prod_start = false;
    return "";
}

std::string Simulator::execute(const double* tp_in, double* tp_out) {
    SimImpl& S = *d_;
    KCHECK(cudaSetDevice(S.device));
    std::string e = enqueue_init(S.stream, tp_in);
    if (e.empty()) e = enqueue_passes(S.stream, tp_out != nullptr);
    if (!e.empty()) return e;
    if (!tp_out) return synchronize();
    const char* r = nullptr;
    e = S.fetch(&r, !S.small);
    if (e.empty()) S.proba_from_sums((const double*)r, tp_out);
    return e;
}

std::string Simulator::enqueue_passes(void* stream, bool sums) {
    SimImpl& S = *d_;
    cudaStream_t st = (cudaStream_t)stream;
    const bool zs = S.zero_start, ps = S.prod_start;
    S.zero_start = S.prod_start = false;
    const bool b0 = S.basis0;
    S.basis0 = false;
    if (S.small) KCHECK(S.launch_small_range(0, (int)S.hpasses.size(), S.small_start, sums && S.precision == 0, st));
    if (zs && S.hpasses.empty()) KCHECK(launch_set_basis0(S.d_state, S.dim(), S.precision, st));
    for (size_t i = 0; i < S.hpasses.size() && !S.small; i++) {
        S.zero_start = zs && i == 0;
        S.prod_start = ps && i == 0;
        S.basis0 = b0;
        S.sum_norm = S.last_sums_norm();
        const cudaError_t ce = S.launch_pass(i, st);
        S.zero_start = S.prod_start = S.sum_norm = S.basis0 = false;
        KCHECK(ce);
    }
    if (S.precision == 1) {
        // Complex64: ||psi|| in FP64, then the state rescaled to norm 1.
        const bool summed = S.last_sums_norm();
        if (sums)
            KCHECK(launch_renorm_bitsums_c64(S.d_state, S.n, S.d_norm, summed, S.d_part, S.res_sums(), S.d_err, S.res_flag(), st));
        else
            KCHECK(launch_renorm_c64(S.d_state, S.n, S.d_norm, summed, st));
        S.renormed = true;
    } else if (sums && !S.small) {
        KCHECK(launch_bitsums(S.d_state, 0, S.n, 0, S.d_part, S.res_sums(), S.d_err, S.res_flag(), st));
    }
    S.phys = S.plan.final_phys;
    S.has_state = true;
    return "";
}

namespace {
struct EventSet {
    cudaEvent_t e[3] = {nullptr, nullptr, nullptr};
    ~EventSet() {
        for (auto x : e)
            if (x) cudaEventDestroy(x);
    }
};
}  // namespace

std::string Simulator::execute_timed(const double* tp_in, double* tp_out, double* ms) {
    SimImpl& S = *d_;
    KCHECK(cudaSetDevice(S.device));
    EventSet ev;
    for (auto& x : ev.e) KCHECK(cudaEventCreate(&x));
    KCHECK(cudaEventRecord(ev.e[0], S.stream));
    std::string e = enqueue_init(S.stream, tp_in);
    if (!e.empty()) return e;
    KCHECK(cudaEventRecord(ev.e[1], S.stream));
    e = enqueue_passes(S.stream);
    if (!e.empty()) return e;
    KCHECK(cudaEventRecord(ev.e[2], S.stream));
    e = synchronize();
    if (!e.empty()) return e;
    float a = 0, b = 0;
    KCHECK(cudaEventElapsedTime(&a, ev.e[0], ev.e[1]));
    KCHECK(cudaEventElapsedTime(&b, ev.e[1], ev.e[2]));
    const auto t0 = std::chrono::steady_clock::now();
    if (tp_out) {
        e = proba_state(tp_out);
        if (!e.empty()) return e;
    }
    const auto t1 = std::chrono::steady_clock::now();
    if (ms) {
        ms[0] = a;
        ms[1] = b;
        ms[2] = std::chrono::duration<double, std::milli>(t1 - t0).count();
        ms[3] = (double)S.hpasses.size();
    }
    return "";
}

std::string Simulator::synchronize() {
    KCHECK(cudaSetDevice(d_->device));
    KCHECK(cudaStreamSynchronize(d_->stream));
    int flag = 0;
    KCHECK(cudaMemcpy(&flag, d_->d_err, sizeof(int), cudaMemcpyDeviceToHost));
    return flag ? d_->timed_out() : "";
}

std::string Simulator::proba_state(double* out) {
    SimImpl& S = *d_;
    if (!S.has_state) return "no state: execute the simulator first";
    KCHECK(cudaSetDevice(S.device));
    const double* sums = nullptr;
    std::string e = S.bit_sums(0, &sums);
    if (e.empty()) S.proba_from_sums(sums, out);
    return e;
}

std::string Simulator::expect_z(double* out) {
    SimImpl& S = *d_;
    if (!S.has_state) return "no state: execute the simulator first";
    KCHECK(cudaSetDevice(S.device));
    const double* sums = nullptr;
    std::string e = S.bit_sums(1, &sums);
    if (!e.empty()) return e;
    for (int x = 0; x < S.n; x++) {
        const double* s0 = sums + 1 + 2 * S.phys_of_label(x);
        out[x] = s0[0] - s0[1];
    }
    return "";
}

std::string Simulator::get_state(double* out) {
    SimImpl& S = *d_;
    if (!S.has_state) return "no state: execute the simulator first";
    KCHECK(cudaSetDevice(S.device));
    std::string e = S.run_relayout(S.label_layout());
    if (!e.empty()) return e;
    if (S.precision == 0) {
        KCHECK(cudaMemcpyAsync(out, S.d_state, S.dim() * 16, cudaMemcpyDeviceToHost, S.stream));
        KCHECK(cudaStreamSynchronize(S.stream));
        return "";
    }
    // complex64: copy as floats, widen in place from the end of the buffer.
    float* f = reinterpret_cast<float*>(out);
    KCHECK(cudaMemcpyAsync(f, S.d_state, S.dim() * 8, cudaMemcpyDeviceToHost, S.stream));
    KCHECK(cudaStreamSynchronize(S.stream));
    for (uint64_t i = 2 * S.dim(); i-- > 0;) out[i] = (double)f[i];
    return "";
}

std::string Simulator::set_state(const double* in) {
    SimImpl& S = *d_;
    KCHECK(cudaSetDevice(S.device));
    if (S.precision == 0) {
        KCHECK(cudaMemcpyAsync(S.d_state, in, S.dim() * 16, cudaMemcpyHostToDevice, S.stream));
        KCHECK(cudaStreamSynchronize(S.stream));
    } else {
        std::vector<float> f(2 * S.dim());
        for (size_t i = 0; i < f.size(); i++) f[i] = (float)in[i];
        KCHECK(cudaMemcpyAsync(S.d_state, f.data(), f.size() * sizeof(float), cudaMemcpyHostToDevice, S.stream));
        KCHECK(cudaStreamSynchronize(S.stream));
    }
    S.phys = S.label_layout();
    S.has_state = true;
    return "";
}

std::string Simulator::probabilities(double* out) {
    SimImpl& S = *d_;
    if (!S.has_state) return "no state: execute the simulator first";
    if (S.n > 30) return "probabilities are limited to 30 qubits";
    KCHECK(cudaSetDevice(S.device));
    std::string e = S.run_relayout(S.label_layout());
    if (!e.empty()) return e;
    double* d = nullptr;
    KCHECK(cudaMallocAsync((void**)&d, S.dim() * sizeof(double), S.stream));
    cudaError_t ce = launch_probs(S.d_state, S.precision, S.dim(), d, S.stream);
    if (ce == cudaSuccess)
        ce = cudaMemcpyAsync(out, d, S.dim() * sizeof(double), cudaMemcpyDeviceToHost, S.stream);
    cudaFreeAsync(d, S.stream);
    if (ce != cudaSuccess) return cuda_err("probabilities", ce);
    KCHECK(cudaStreamSynchronize(S.stream));
    return "";
}

std::string Simulator::sample(int shots, uint64_t seed, uint64_t* out) {
    SimImpl& S = *d_;
    if (shots < 0) return "shots must be >= 0";
    if (!S.has_state) return "no state: execute the simulator first";
    if (shots == 0) return "";
    KCHECK(cudaSetDevice(S.device));
    // Samples go straight to pinned memory when they fit, else to the end of
    // the workspace and from there in one copy.
    const size_t out_bytes = (size_t)shots * sizeof(uint64_t);
    const bool direct = S.pinned && out_bytes <= kPinnedSlotBytes;
    const size_t scr = sample_scratch_doubles(S.n) * sizeof(double);
    const size_t need = scr + (direct ? 0 : out_bytes);
    if (S.samp_bytes < need) {
        KCHECK(cudaStreamSynchronize(S.stream));
        cudaFree(S.d_samp);
        S.d_samp = nullptr;
        S.samp_bytes = 0;
        KCHECK(cudaMalloc(&S.d_samp, need));
        S.samp_bytes = need;
    }
    SampleLabels L{};
    for (int x = 0; x < S.n; x++) L.phys[x] = (uint8_t)S.phys_of_label(x);
    uint64_t* dst = (uint64_t*)(direct ? S.pinned : S.d_samp + scr);
    KCHECK(launch_sample(S.d_state, S.precision, S.n, seed, shots, L, (double*)S.d_samp, dst, S.stream));
    if (!direct) KCHECK(cudaMemcpyAsync(out, dst, out_bytes, cudaMemcpyDeviceToHost, S.stream));
    KCHECK(cudaStreamSynchronize(S.stream));
    if (direct) std::memcpy(out, S.pinned, out_bytes);
    return "";
}

std::string Simulator::profile_passes(float* ms, float* init_ms) {
    SimImpl& S = *d_;
    KCHECK(cudaSetDevice(S.device));
    std::vector<cudaEvent_t> ev(S.hpasses.size() + 2);
    for (auto& e : ev) KCHECK(cudaEventCreate(&e));
    KCHECK(cudaEventRecord(ev[0], S.stream));
    KCHECK(launch_set_basis0(S.d_state, S.dim(), S.precision, S.stream));
    KCHECK(cudaEventRecord(ev[1], S.stream));
    for (size_t i = 0; i < S.hpasses.size(); i++) {
        KCHECK(S.launch_pass(i, S.stream));
        KCHECK(cudaEventRecord(ev[i + 2], S.stream));
    }
    KCHECK(cudaEventSynchronize(ev.back()));
    if (init_ms) KCHECK(cudaEventElapsedTime(init_ms, ev[0], ev[1]));
    for (size_t i = 0; i < S.hpasses.size(); i++) KCHECK(cudaEventElapsedTime(&ms[i], ev[i + 1], ev[i + 2]));
    for (auto& e : ev) cudaEventDestroy(e);
    S.phys = S.plan.final_phys;
    S.has_state = true;
    return "";
}

int Simulator::launches_per_run() const {
    if (d_->small) return 1 + (d_->precision == 1 ? 2 : 0);
    return (d_->starts_from_zero() ? 0 : 1) + (int)d_->hpasses.size() +
           (d_->precision == 1 ? d_->last_sums_norm() ? 1 : 2 : 0);
}

std::string Simulator::norm2_before_renorm(double* out) {
    SimImpl& S = *d_;
    if (S.precision != 1) return "only complex64 simulators are renormalised";
    if (!S.renormed) return "no run has been renormalised yet";
    KCHECK(cudaSetDevice(S.device));
    KCHECK(cudaStreamSynchronize(S.stream));
    KCHECK(cudaMemcpy(out, (const char*)S.d_norm + renorm_result_offset(), sizeof(double), cudaMemcpyDeviceToHost));
    return "";
}

int Simulator::pass_kernel(int i) const {
    const SimImpl& S = *d_;
    if (i < 0 || i >= (int)S.plan.passes.size()) return -1;
    const PlannedPass& p = S.plan.passes[i];
    if (p.bprog) return 3;
    if (S.small) return 1;
    if (p.prog && (size_t)i < S.jit_fn.size() && S.jit_fn[i]) return 2;
    if (p.prog) return 1;
    return 0;
}

bool Simulator::pass_work(int i, double out[3]) const {
    if (pass_kernel(i) != 2) return false;
    out[0] = 2.0 * 16.0;
    return jit_pass_work(*d_->plan.passes[i].prog, d_->sops_of((size_t)i), &out[1], &out[2]);
}

std::string Simulator::state_device(void** dptr, int* phys) {
    *dptr = d_->d_state;
    for (int x = 0; x < d_->n; x++) phys[x] = d_->phys_of_label(x);
    return "";
}

}  // namespace kate
