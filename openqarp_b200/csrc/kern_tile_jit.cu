// kern_tile_jit.cu — register-tile passes compiled for their own plan (executor 3).
//
// The register-tile kernel (kern_tile_rt.cu) interprets a pass's steps: every step reads its
// descriptor, dispatches on its kind and slot mask, and recomputes layout-dependent indices;
// on a 28-qubit brickwork pass only 40 % of its instructions are FP64 work, the rest are
// register moves at the joins of the step loop and index arithmetic.  Here each pass's plan
// (the same planner, plan_rt) becomes straight-line CUDA C: the 16 amplitudes a thread holds
// are named variables, every layout and register-slot pattern is a compile-time constant (a
// sign flip on register slots costs nothing; a transpose is 16 stores and 16 loads at constant
// offsets from one per-thread base), and the op coefficients are kernel parameters, read from
// the constant bank as FMA operands.  The source depends only on the circuit's structure
// (gate kinds, qubits, tile layouts) and the register width, so one compiled module serves every
// parameter set of a circuit; modules are compiled once with NVRTC, kept per device for the
// process and cached on disk by a hash of their source (QSV_JIT_CACHE, default
// ~/.cache/openqarp_b200/jit).
//
// NVRTC and the CUDA driver API are opened with dlopen on first use, so the library loads
// (and every other executor runs) where they are absent.
#include <dlfcn.h>
#include <sys/stat.h>
#include <unistd.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <map>
#include <memory>
#include <mutex>
#include <sstream>
#include <thread>
#include <atomic>
#include <stdexcept>
#include <string>
#include <vector>

#include <cuda.h>
#include <nvrtc.h>

#include "../../include/qsv.h"
#include "kernels.h"
#include "tile.h"

namespace qsv {

namespace {

// ---------------------------------------------------------------- dlopen'ed entry points

struct Nvrtc {
    decltype(&nvrtcCreateProgram) create = nullptr;
    decltype(&nvrtcCompileProgram) compile = nullptr;
    decltype(&nvrtcGetProgramLogSize) log_size = nullptr;
    decltype(&nvrtcGetProgramLog) log = nullptr;
    decltype(&nvrtcGetCUBINSize) cubin_size = nullptr;
    decltype(&nvrtcGetCUBIN) cubin = nullptr;
    decltype(&nvrtcDestroyProgram) destroy = nullptr;
    decltype(&nvrtcGetErrorString) error = nullptr;
};

struct Driver {
    decltype(&cuModuleLoadData) load = nullptr;
    decltype(&cuModuleGetFunction) get_function = nullptr;
    decltype(&cuFuncSetAttribute) set_attribute = nullptr;
    decltype(&cuLaunchKernel) launch = nullptr;
    decltype(&cuGetErrorString) error = nullptr;
    decltype(&cuCtxGetCurrent) current = nullptr;
};

template <typename F>
void bind(void* lib, const char* name, F* out) {
    void* p = dlsym(lib, name);
    if (!p) throw std::runtime_error(std::string("JIT tiles: symbol ") + name + " not found");
    *out = reinterpret_cast<F>(p);
}

const Nvrtc& nvrtc() {
    static std::once_flag once;
    static Nvrtc api;
    static std::string err;
    std::call_once(once, [] {
        void* lib = dlopen("libnvrtc.so.12", RTLD_NOW | RTLD_LOCAL);
        if (!lib) lib = dlopen("libnvrtc.so", RTLD_NOW | RTLD_LOCAL);
        if (!lib) { err = "JIT tiles: libnvrtc.so.12 not found"; return; }
        try {
            bind(lib, "nvrtcCreateProgram", &api.create);
            bind(lib, "nvrtcCompileProgram", &api.compile);
            bind(lib, "nvrtcGetProgramLogSize", &api.log_size);
            bind(lib, "nvrtcGetProgramLog", &api.log);
            bind(lib, "nvrtcGetCUBINSize", &api.cubin_size);
            bind(lib, "nvrtcGetCUBIN", &api.cubin);
            bind(lib, "nvrtcDestroyProgram", &api.destroy);
            bind(lib, "nvrtcGetErrorString", &api.error);
        } catch (const std::exception& e) {
            err = e.what();
        }
    });
    if (!err.empty()) throw std::runtime_error(err);
    return api;
}

const Driver& driver() {
    static std::once_flag once;
    static Driver api;
    static std::string err;
    std::call_once(once, [] {
        void* lib = dlopen("libcuda.so.1", RTLD_NOW | RTLD_LOCAL);
        if (!lib) { err = "JIT tiles: libcuda.so.1 not found"; return; }
        try {
            bind(lib, "cuModuleLoadData", &api.load);
            bind(lib, "cuModuleGetFunction", &api.get_function);
            bind(lib, "cuFuncSetAttribute", &api.set_attribute);
            bind(lib, "cuLaunchKernel", &api.launch);
            bind(lib, "cuGetErrorString", &api.error);
            bind(lib, "cuCtxGetCurrent", &api.current);
        } catch (const std::exception& e) {
            err = e.what();
        }
    });
    if (!err.empty()) throw std::runtime_error(err);
    return api;
}

void check_cu(CUresult r, const char* what) {
    if (r == CUDA_SUCCESS) return;
    const char* s = nullptr;
    driver().error(r, &s);
    throw cuda_error(std::string(what) + ": " + (s ? s : "CUDA driver error"));
}

// ---------------------------------------------------------------- code generation

constexpr int kJitAmps = 1 << kRtRegBits;                 // 16 amplitudes per thread
constexpr int kJitThreads = 1 << (kRtLaneBits + kRtWarpBits);
constexpr size_t kJitMaxCoefDoubles = 3400;               // kernel parameters stay under 28 KiB
constexpr int kJitCtasPerSm = 2;                          // complex128: 64 KiB of shared memory, <= 128 registers
constexpr int kJitCtasPerSmF32 = 3;                       // complex64: 32 KiB, <= 85 registers
int jit_ctas(bool f32) { return f32 ? kJitCtasPerSmF32 : kJitCtasPerSm; }
size_t jit_smem(bool f32) { return (size_t{1} << kRtQubits) * (f32 ? 8 : 16); }
// Pair passes (the adjoint's reverse sweep, complex128): psi and phi tiles and a column of accumulators
// per thread; one CTA per SM, whose threads hold both tiles' 16 amplitudes (128 of 255 registers).  A
// 24-qubit pass of some 21 inner products takes 0.35 ms, 3.1 TB/s: reading the tiles, the steps and the
// stores of its one CTA follow one another.  The interpreter it replaces (1.6 ms) read and wrote both
// tiles in shared memory at every step, with a barrier between.
constexpr int kPairMaxAcc = 48;
size_t pair_smem(int n_acc) { return 2 * jit_smem(false) + static_cast<size_t>(n_acc) * kJitThreads * sizeof(double); }

uint32_t swz(uint32_t i) { return i ^ ((i >> 3 ^ i >> 6 ^ i >> 9) & 7u); }

std::string hex64(uint64_t v) {
    char b[32];
    std::snprintf(b, sizeof b, "0x%llxull", static_cast<unsigned long long>(v));
    return b;
}

// Local index of register r in layout L (the register-slot bits only).
uint32_t reg_local(const RtLayout& L, int r) {
    uint32_t i = 0;
    for (int p = 0; p < kRtRegBits; ++p)
        if ((r >> p) & 1) i |= 1u << L.reg[p];
    return i;
}

// One-qubit unitary as U = D1 R D2: D1 = diag(d1[0], d1[1]) and D2 = diag(d2[0], d2[1]) unit
// phases, R = [[c, -s], [s, c]] real with c, s >= 0.  From the entries of D1 R D2 —
// c d1_0 d2_0, -s d1_0 d2_1, s d1_1 d2_0, c d1_1 d2_1 — with one phase fixed to 1 per factor
// (the larger of c, s keeps its entries' phases exact).
struct Factor1q {
    c128 d1[2], d2[2];
    double c = 1, s = 0;
};

c128 unit_phase(c128 v) {
    const double a = std::abs(v);
    return a > 0 ? v / a : c128(1.0, 0.0);
}

// Whether v is a phase: products of a few thousand gates' phases stay well inside.
bool is_phase(c128 v) { return std::abs(std::norm(v) - 1.0) <= 1e-10; }

// False where u is not unitary (to 1e-12 an entry).
bool factor_unitary(const std::vector<c128>& u, Factor1q* out) {
    Factor1q f;
    double c = std::abs(u[0]), s = std::abs(u[2]);
    const double r = std::sqrt(c * c + s * s);
    if (r > 0) { c /= r; s /= r; }
    f.c = c;
    f.s = s;
    if (c >= s) {
        const c128 P = unit_phase(u[0]);
        const c128 T = s > 0 ? unit_phase(-u[1]) / P : c128(1.0, 0.0);
        f.d1[0] = P; f.d1[1] = unit_phase(u[3]) / T;
        f.d2[0] = c128(1.0, 0.0); f.d2[1] = T;
    } else {
        const c128 P = unit_phase(-u[1]);
        const c128 R = c > 0 ? unit_phase(u[0]) / P : c128(1.0, 0.0);
        f.d1[0] = P; f.d1[1] = unit_phase(u[2]) / R;
        f.d2[0] = R; f.d2[1] = c128(1.0, 0.0);
    }
    const c128 m[4] = {c * f.d1[0] * f.d2[0], -s * f.d1[0] * f.d2[1], s * f.d1[1] * f.d2[0], c * f.d1[1] * f.d2[1]};
    for (int e = 0; e < 4; ++e)
        if (std::abs(m[e] - u[e]) > 1e-12 * std::max(1.0, std::abs(u[e]))) return false;
    *out = f;
    return true;
}

// the factors must reproduce the gate: a planner or rounding surprise becomes a host error
Factor1q factor_1q(const std::vector<c128>& u) {
    Factor1q f;
    if (!factor_unitary(u, &f))
        throw std::logic_error("JIT tiles: one-qubit factorisation does not reproduce the gate");
    return f;
}

// A deferred one-qubit phase pair on global qubit q: amplitudes with the bit 0 / 1 owe p[0/1].
struct QubitPhase {
    int q = 0;
    c128 p[2];
};

// What one compiled pass hands to the next of its chain instead of applying it: the deferred
// phases of the qubits it touched (and those it carried through untouched), and the tile
// constant with its table count.  Every amplitude of the register owes the same factors, so
// the next pass can fold them into its own tables.
struct Carry {
    std::vector<QubitPhase> phases;   // ascending q, at most one entry per qubit
    c128 cglob{1.0, 0.0};
    int normalised = 0;
};

// Code generator of one pass.  With emit off it only walks the plan, collecting the
// coefficients and the structural signature (everything the source depends on), so a pass
// whose kernel is already compiled costs no source generation.
struct Gen {
    bool emit = true;
    std::ostringstream o;
    std::vector<double> coef;
    std::vector<uint64_t> sig;
    int local_of[64];
    // deferred one-qubit phases per local bit: amplitudes with the bit 0 / 1 owe pend[b][0/1]
    c128 pend[kRtQubits][2];
    bool has[kRtQubits] = {};
    // a factor owed by every amplitude of the tile: the bit-0 phases of normalised tables
    c128 cglob{1.0, 0.0};
    // Bit-flip frame: the amplitude stored at local index i belongs to index i ^ (the bits with
    // turned[b]).  A rotation by more than a quarter turn leaves its bit turned instead of moving
    // data (gate_batch); every other op is rewritten for the stored index on the host, and the
    // pass's store puts the amplitudes back (an XOR on the address).  Which bits are turned depends
    // on the matrices, the source never does.
    bool turned[kRtQubits] = {};
    // deferred phases of qubits outside the tile (constants of the tile's base index)
    std::vector<QubitPhase> outside;
    int normalised = 0;   // normalised tables since cglob was last applied
    double flops = 0;   // FP64 operations per thread per tile (FMA = 2, MUL = 1)

    size_t push(c128 v) {
        coef.push_back(v.real());
        coef.push_back(v.imag());
        return coef.size() - 2;
    }
    // A real coefficient.  Complex128: a pair with a 0, or the complex entries after it straddle 16 bytes,
    // are read in halves, and ptxas spills amplitudes (28-qubit brickwork: 2680 bytes of spill stores over
    // its 15 passes against 1150, 48.7 against 47.1 ms; 656 as it is now).  Complex64 takes single ones
    // and 64-bit tile numbers: the 30-qubit Heisenberg step 17.87 ms, 18.04 to 18.24 in the other forms.
    size_t real(double v) {
        if (!f32) return push(v);
        coef.push_back(v);
        return coef.size() - 1;
    }
    static std::string cr(size_t at) { return "P.c[" + std::to_string(at) + "]"; }
    static std::string ci(size_t at) { return "P.c[" + std::to_string(at + 1) + "]"; }
    // `pair`: a pass of the adjoint's reverse sweep, every op on the registers of psi ("a") and of phi
    // ("b"); the register names below are those of `set`
    bool pair = false;
    char set = 'a';
    std::string ar(int r) const { return set + std::to_string(r) + "r"; }
    std::string ai(int r) const { return set + std::to_string(r) + "i"; }
    template <typename F>
    void each_set(F&& f) {
        f();
        if (!pair) return;
        set = 'b';
        f();
        set = 'a';
    }
    void mark(uint64_t a, uint64_t b = 0) { sig.push_back(a); sig.push_back(b); }
    void mark_layout(const RtLayout& L) {
        uint64_t x = 0, y = 0;
        std::memcpy(&x, &L, 8);
        std::memcpy(&y, reinterpret_cast<const uint8_t*>(&L) + 8, sizeof(RtLayout) - 8);
        mark(x, y);
    }

    // per-thread local index bits of layout L (lane and warp bits), as an expression
    static std::string lfix_expr(const RtLayout& L) {
        std::string e = "0u";
        for (int k = 0; k < kRtLaneBits; ++k)
            e += " | (((lane >> " + std::to_string(k) + ") & 1u) << " + std::to_string(L.lane[k]) + ")";
        for (int k = 0; k < kRtWarpBits; ++k)
            e += " | (((warp >> " + std::to_string(k) + ") & 1u) << " + std::to_string(L.warp[k]) + ")";
        return e;
    }

    // where local bit b lives in layout L: 'r' slot p, 'l' lane bit k, 'w' warp bit k
    static char place(const RtLayout& L, int b, int* k) {
        for (int p = 0; p < kRtRegBits; ++p) if (L.reg[p] == b) { *k = p; return 'r'; }
        for (int j = 0; j < kRtLaneBits; ++j) if (L.lane[j] == b) { *k = j; return 'l'; }
        for (int j = 0; j < kRtWarpBits; ++j) if (L.warp[j] == b) { *k = j; return 'w'; }
        throw std::logic_error("JIT tiles: local bit outside the layout");
    }

    // Runtime part of "all of these local bits are 1" (lane and warp bits); the register-slot
    // part is returned as a slot pattern.
    static std::string thread_cond(const RtLayout& L, uint32_t lm, uint32_t* slot_pattern) {
        uint32_t rm = 0;
        std::string c;
        for (int b = 0; b < kRtQubits; ++b) {
            if (!((lm >> b) & 1)) continue;
            int k = 0;
            const char w = place(L, b, &k);
            if (w == 'r') rm |= 1u << k;
            else c += (c.empty() ? "" : " && ") + std::string(w == 'l' ? "((lane >> " : "((warp >> ") +
                      std::to_string(k) + ") & 1u)";
        }
        *slot_pattern = rm;
        return c;
    }

    uint32_t split(uint64_t gm, uint64_t* outside) const {
        uint32_t lm = 0;
        uint64_t out = 0;
        for (int q = 0; q < 64; ++q)
            if ((gm >> q) & 1) {
                if (local_of[q] >= 0) lm |= 1u << local_of[q];
                else out |= 1ull << q;
            }
        *outside = out;
        return lm;
    }

    std::string full_cond(const RtLayout& L, uint64_t gmask, uint32_t* rm) {
        uint64_t outside = 0;
        const uint32_t lm = split(gmask, &outside);
        std::string c = thread_cond(L, lm, rm);
        mark(lm, outside);
        if (outside) c = "((base & " + hex64(outside) + ") == " + hex64(outside) + ")" + (c.empty() ? "" : " && " + c);
        return c;
    }

    void cmul_into(int r, const std::string& pr, const std::string& pi) {
        o << "    { const R xr = " << ar(r) << ", xi = " << ai(r) << "; "
          << ar(r) << " = " << pr << " * xr - " << pi << " * xi; "
          << ai(r) << " = " << pr << " * xi + " << pi << " * xr; }\n";
    }

    // apply the deferred phases of the local bits now in register slots: one table over those
    // slots, one complex multiply per amplitude.  The table is normalised: each bit's phase
    // pair pend[b] = (p0, p1) becomes (1, p1 / p0) with p0 joining the tile constant cglob, so
    // the amplitudes whose slot bits are all 0 need no multiply.  A full table (every entry
    // times cglob, every amplitude multiplied) ends the pass and, every 16 tables, keeps the
    // deferred rotation scales (each >= 1/sqrt(2)) from growing the amplitudes past 2^32.
    void flush_slots(const RtLayout& L, bool full = false) {
        int slots[kRtRegBits], m = 0;
        for (int p = 0; p < kRtRegBits; ++p)
            if (has[L.reg[p]]) slots[m++] = p;
        if (m > 0 && !full && ++normalised >= 16) full = true;
        uint32_t smask = 0;
        for (int j = 0; j < m; ++j) smask |= 1u << slots[j];
        mark(full ? 0xF3u : 0xF1u, smask);
        if (m == 0 && !full) return;
        const size_t at = coef.size();
        if (full) {
            for (int idx = 0; idx < (1 << m); ++idx) {
                c128 t = cglob;
                for (int j = 0; j < m; ++j) t *= pend[L.reg[slots[j]]][(idx >> j) & 1];
                push(t);
            }
            cglob = c128(1.0, 0.0);
            normalised = 0;
            flops += 6.0 * kJitAmps;
        } else {
            c128 ratio[kRtRegBits];
            for (int j = 0; j < m; ++j) {
                const c128* pb = pend[L.reg[slots[j]]];
                cglob *= pb[0];
                ratio[j] = pb[1] / pb[0];
            }
            for (int idx = 1; idx < (1 << m); ++idx) {
                c128 t(1.0, 0.0);
                for (int j = 0; j < m; ++j)
                    if ((idx >> j) & 1) t *= ratio[j];
                push(t);
            }
            flops += 6.0 * (kJitAmps - (kJitAmps >> m));
        }
        for (int j = 0; j < m; ++j) has[L.reg[slots[j]]] = false;
        if (!emit) return;
        each_set([&] {
            for (int r = 0; r < kJitAmps; ++r) {
                int idx = 0;
                for (int j = 0; j < m; ++j) idx |= ((r >> slots[j]) & 1) << j;
                if (!full && idx == 0) continue;
                const size_t e = at + 2 * static_cast<size_t>(full ? idx : idx - 1);
                cmul_into(r, cr(e), ci(e));
            }
        });
    }

    // end of a chain of passes: the deferred phases of lane and warp bits, and those carried
    // in on qubits outside the tile (constants of the tile's base index), as one factor per
    // thread (starting from the tile constant), after the slot table; without lane, warp or
    // outside phases the slot table is the full one
    void flush_all(const RtLayout& L) {
        uint64_t m = 0, om = 0;
        for (int b = 0; b < kRtQubits; ++b) {
            if (!has[b]) continue;
            int k = 0;
            const char w = place(L, b, &k);
            if (w == 'r') continue;
            m |= 1ull << ((w == 'l' ? 0 : 16) + k);
        }
        for (const QubitPhase& x : outside) om |= 1ull << x.q;
        mark(0xF2u, m);
        mark(0xF4u, om);
        if (m == 0 && om == 0) {
            flush_slots(L, true);
            return;
        }
        flush_slots(L);
        const size_t c0 = push(cglob);
        cglob = c128(1.0, 0.0);
        normalised = 0;
        std::vector<std::pair<int, size_t>> bits;   // (place code, coefficient offset)
        for (int b = 0; b < kRtQubits; ++b) {
            if (!has[b]) continue;
            int k = 0;
            const char w = place(L, b, &k);
            bits.push_back({(w == 'l' ? 0 : 16) + k, push(pend[b][0])});
            push(pend[b][1]);
            has[b] = false;
        }
        for (const QubitPhase& x : outside) {
            bits.push_back({64 + x.q, push(x.p[0])});
            push(x.p[1]);
        }
        flops += 6.0 * kJitAmps + 6.0 * static_cast<double>(bits.size());
        if (!emit) return;
        o << "  { R fr = " << cr(c0) << ", fi = " << ci(c0) << ";\n";
        for (const auto& [code, at] : bits) {
            const std::string on = code >= 64 ? "((base >> " + std::to_string(code - 64) + ") & 1ull)"
                                   : code < 16 ? "((lane >> " + std::to_string(code) + ") & 1u)"
                                               : "((warp >> " + std::to_string(code - 16) + ") & 1u)";
            o << "    { const bool on = " << on << "; const R pr = on ? " << cr(at + 2) << " : " << cr(at)
              << ", pi = on ? " << ci(at + 2) << " : " << ci(at) << "; const R nr = fr * pr - fi * pi;"
              << " fi = fr * pi + fi * pr; fr = nr; }\n";
        }
        each_set([&] {
            for (int r = 0; r < kJitAmps; ++r) cmul_into(r, "fr", "fi");
        });
        o << "  }\n";
    }

    // the deferred pair of qubit q (a tile bit's in the stored index), created as 1, 1
    c128* owed(int q) {
        const int b = local_of[q];
        if (b >= 0) {
            if (!has[b]) pend[b][0] = pend[b][1] = c128(1.0, 0.0);
            has[b] = true;
            return pend[b];
        }
        for (QubitPhase& x : outside)
            if (x.q == q) return x.p;
        QubitPhase x;
        x.q = q;
        x.p[0] = x.p[1] = c128(1.0, 0.0);
        outside.push_back(x);
        return outside.back().p;
    }
    bool turned_q(int q) const { return local_of[q] >= 0 && turned[local_of[q]]; }

    // consecutive one-qubit gates on distinct register slots: their D2 factors join the
    // deferred phases, one table applies them, then the real rotations; D1 is deferred.
    // A rotation is divided by its larger entry, so each output component is one FMA:
    //   c >= s:  R = c [[1, -t], [t, 1]],  t = s / c
    //   s >  c:  R = s [[u, -1], [1, u]],  u = c / s, which is [[1, u], [-u, 1]] (the first form with
    //            t = -u) whose outputs come exchanged, the second with its sign changed: the bit is
    //            left turned and the sign joins D1
    // the scale (c or s, the same for both basis states) joins the deferred phases.  One form serves
    // every matrix, so a structure is compiled once and has no branch at a gate.  28-qubit brickwork
    // with new matrices each call, whole call: 48.3 ms in complex128 and 33.1 ms in complex64;
    // 52.8 and 38.0 ms with a uniform branch on the form at every gate.
    void gate_batch(const std::vector<const RtStep*>& gates, const RtLayout& L, int local_bit_of_slot[]) {
        std::vector<Factor1q> f;
        uint32_t smask = 0;
        for (const RtStep* st : gates) {
            const int p = st->slot_of[0];
            const int b = local_bit_of_slot[p];
            const std::vector<c128>& m = st->op->m;
            f.push_back(factor_1q(turned[b] ? std::vector<c128>{m[3], m[2], m[1], m[0]} : m));
            const Factor1q& z = f.back();
            for (int v = 0; v < 2; ++v) pend[b][v] = (has[b] ? pend[b][v] : c128(1.0, 0.0)) * z.d2[v];
            has[b] = true;
            smask |= 1u << p;
        }
        mark(0xB0u, smask);
        flush_slots(L);
        for (size_t i = 0; i < gates.size(); ++i) {
            const int p = gates[i]->slot_of[0];
            const int b = local_bit_of_slot[p];
            rotate(p, b, f[i].c, f[i].s, f[i].d1[0], f[i].d1[1]);
        }
    }

    // diag(d0, d1) [[c, -s], [s, c]] on slot p holding local bit b, as above.  In a pair pass the scale
    // joins the tile constant, so the deferred pairs stay unit phases and cancel in inner products.
    void rotate(int p, int b, double c, double s, c128 d0, c128 d1) {
        const bool cos_form = std::abs(c) >= std::abs(s);
        double scale = cos_form ? c : s;
        const size_t at = real(cos_form ? s / c : -(c / s));
        if (pair) {
            cglob *= scale;
            scale = 1.0;
        }
        pend[b][0] = (cos_form ? d0 : d1) * scale;
        pend[b][1] = (cos_form ? d1 : -d0) * scale;
        has[b] = true;
        turned[b] ^= !cos_form;
        mark(0xB1u, static_cast<uint64_t>(p));
        flops += 8.0 * (kJitAmps / 2) * (pair ? 2 : 1);
        if (!emit) return;
        const int B = 1 << p;
        o << "  { const R t = " << cr(at) << ";\n";
        each_set([&] {
            // complex64: each amplitude is one float2, and a rotation updates both of its
            // components with one packed FMA (__ffma2_rn, rounding as fmaf per component)
            if (f32) o << "    const R2 t2 = make_float2(t, t), nt2 = make_float2(-t, -t);\n";
            for (int g = 0; g < kJitAmps; ++g) {
                if (g & B) continue;
                const int h = g | B;
                if (f32) {
                    const std::string x0 = "a" + std::to_string(g), x1 = "a" + std::to_string(h);
                    o << "    { const R2 y0 = " << x0 << "; " << x0 << " = __ffma2_rn(nt2, " << x1 << ", y0); "
                      << x1 << " = __ffma2_rn(t2, y0, " << x1 << "); }\n";
                    continue;
                }
                const std::string x0r = ar(g), x0i = ai(g), x1r = ar(h), x1i = ai(h);
                o << "    { const R y0r = " << x0r << ", y0i = " << x0i << "; "
                  << x0r << " = FMA(-t, " << x1r << ", y0r); " << x0i << " = FMA(-t, " << x1i << ", y0i); "
                  << x1r << " = FMA(t, y0r, " << x1r << "); " << x1i << " = FMA(t, y0i, " << x1i << "); }\n";
            }
        });
        o << "  }\n";
    }

    // Puts slot p's bit back where it is turned (a uniform branch on a coefficient): before ops whose
    // form the host cannot rewrite.
    void unturn_slot(const RtLayout& L, int p) {
        const int b = L.reg[p];
        const size_t at = real(turned[b] ? 1.0 : 0.0);
        if (turned[b]) std::swap(pend[b][0], pend[b][1]);
        turned[b] = false;
        mark(0xF7u, static_cast<uint64_t>(p));
        if (!emit) return;
        o << "  if (" << cr(at) << " != 0) {\n";
        each_set([&] {
            for (int g = 0; g < kJitAmps; ++g)
                if (!(g & (1 << p))) swap_regs(g, g | (1 << p));
        });
        o << "  }\n";
    }
    void swap_regs(int g, int h) {
        o << "    { const R xr = " << ar(g) << ", xi = " << ai(g) << "; " << ar(g) << " = " << ar(h) << "; " << ai(g) << " = "
          << ai(h) << "; " << ar(h) << " = xr; " << ai(h) << " = xi; }\n";
    }

    void dense(const Op& op, const std::vector<int>& slot_of) {
        const int k = op.k, D = 1 << k;
        const size_t at = coef.size();
        int tm = 0;      // turned bits: rows and columns exchanged
        for (int b = 0; b < k; ++b)
            if (turned_q(static_cast<int>(op.qubits[b]))) tm |= 1 << b;
        for (int y = 0; y < D; ++y)
            for (int x = 0; x < D; ++x) push(op.m[static_cast<size_t>((y ^ tm) * D + (x ^ tm))]);
        uint32_t slots = 0;
        uint64_t so = 0;
        for (int b = 0; b < k; ++b) {
            slots |= 1u << slot_of[b];
            so |= static_cast<uint64_t>(slot_of[b]) << (4 * b);
        }
        mark(0xD0u + static_cast<uint64_t>(k), so);
        flops += static_cast<double>(kJitAmps / D) * D * D * 8.0;
        if (!emit) return;
        each_set([&] {
        for (int g = 0; g < kJitAmps; ++g) {
            if (g & static_cast<int>(slots)) continue;
            std::vector<int> reg(D);
            for (int x = 0; x < D; ++x) {
                int r = g;
                for (int b = 0; b < k; ++b)
                    if ((x >> b) & 1) r |= 1 << slot_of[b];
                reg[x] = r;
            }
            o << "  {\n";
            for (int y = 0; y < D; ++y) {
                o << "    const R o" << y << "r = ";
                for (int x = 0; x < D; ++x) {
                    const size_t e = at + 2 * static_cast<size_t>(y * D + x);
                    o << (x ? " + " : "") << cr(e) << " * " << ar(reg[x]) << " - " << ci(e) << " * " << ai(reg[x]);
                }
                o << ";\n    const R o" << y << "i = ";
                for (int x = 0; x < D; ++x) {
                    const size_t e = at + 2 * static_cast<size_t>(y * D + x);
                    o << (x ? " + " : "") << cr(e) << " * " << ai(reg[x]) << " + " << ci(e) << " * " << ar(reg[x]);
                }
                o << ";\n";
            }
            for (int y = 0; y < D; ++y) o << "    " << ar(reg[y]) << " = o" << y << "r; " << ai(reg[y]) << " = o" << y << "i;\n";
            o << "  }\n";
        }
        });
    }

    // m0 on the amplitudes whose bits of op.mask are all 1.  One bit: deferred.  Two bits: with turned
    // bits f and s = 1 - 2 f, (f1 + s1 b1)(f2 + s2 b2) is the phase of the stored bits, so the turned
    // bits leave one-qubit phases and the pair's sign.  More: the turned bits are put back or flip
    // their part of the condition.
    void phase(const Op& op, const RtLayout& L) {
        const int width = __builtin_popcountll(op.mask);
        c128 m0 = op.m[0];
        const bool sign = m0 == c128(-1.0, 0.0);
        if (width == 1) {
            const int q = __builtin_ctzll(op.mask);
            const bool t = turned_q(q);
            owed(q)[t ? 0 : 1] *= m0;
            mark(0xA3u, op.mask);
            return;
        }
        if (width == 2) {
            const int q1 = __builtin_ctzll(op.mask), q2 = 63 - __builtin_clzll(op.mask);
            const bool f1 = turned_q(q1), f2 = turned_q(q2);
            auto power = [&](int e) { return e == 0 ? c128(1.0, 0.0) : e > 0 ? m0 : 1.0 / m0; };
            const int s1 = f1 ? -1 : 1, s2 = f2 ? -1 : 1;
            // both pairs are touched whatever is turned: the structure does not depend on the matrices
            owed(q1)[1] *= power(f2 ? s1 : 0);
            owed(q2)[1] *= power(f1 ? s2 : 0);
            if (f1 && f2) cglob *= m0;
            m0 = sign ? m0 : power(s1 * s2);
        }
        uint32_t rm = 0;
        const std::string c = width == 2 ? full_cond(L, op.mask, &rm) : turned_cond(L, op.mask, &rm);
        mark(sign ? 0xA1u : 0xA2u, rm);
        if (sign && c.empty()) {
            if (emit) each_set([&] {
                for (int r = 0; r < kJitAmps; ++r)
                    if ((static_cast<uint32_t>(r) & rm) == rm) o << "  " << ar(r) << " = -" << ar(r) << "; " << ai(r) << " = -" << ai(r) << ";\n";
            });
            return;
        }
        if (sign) {
            // a sign flip under a runtime condition: XOR of the sign bits (integer pipe)
            if (!emit) return;
            o << "  { const int sm = (" << c << ") ? (int)0x80000000 : 0;\n";
            each_set([&] {
                for (int r = 0; r < kJitAmps; ++r)
                    if ((static_cast<uint32_t>(r) & rm) == rm)
                        o << "    " << ar(r) << " = flip(" << ar(r) << ", sm); " << ai(r) << " = flip(" << ai(r) << ", sm);\n";
            });
            o << "  }\n";
            return;
        }
        const size_t at = push(m0);
        flops += 6.0 * static_cast<double>(kJitAmps >> __builtin_popcount(rm));
        if (!emit) return;
        o << "  if (" << (c.empty() ? "true" : c) << ") {\n";
        each_set([&] {
            for (int r = 0; r < kJitAmps; ++r)
                if ((static_cast<uint32_t>(r) & rm) == rm) cmul_into(r, cr(at), ci(at));
        });
        o << "  }\n";
    }

    // full_cond for ops that take the bits as they are: slot bits are put back, turned lane and warp
    // bits compare with a coefficient
    std::string turned_cond(const RtLayout& L, uint64_t gmask, uint32_t* rm) {
        uint64_t out = 0;
        const uint32_t lm = split(gmask, &out);
        for (int b = 0; b < kRtQubits; ++b) {
            int k = 0;
            if (((lm >> b) & 1) && place(L, b, &k) == 'r') unturn_slot(L, k);
        }
        *rm = 0;
        std::string c;
        mark(lm, out);
        if (out) c = "((base & " + hex64(out) + ") == " + hex64(out) + ")";
        for (int b = 0; b < kRtQubits; ++b) {
            if (!((lm >> b) & 1)) continue;
            int k = 0;
            const char w = place(L, b, &k);
            if (w == 'r') {
                *rm |= 1u << k;
                continue;
            }
            const size_t at = real(turned[b] ? 1.0 : 0.0);
            c += (c.empty() ? "" : " && ") + std::string(w == 'l' ? "((((lane >> " : "((((warp >> ") + std::to_string(k) +
                 ") & 1u) != 0u) != (" + cr(at) + " != 0))";
        }
        return c;
    }

    // A controlled X from one control moves data without arithmetic: a rename where the control is a
    // slot bit, selects elsewhere.  A turned control applies X to the other half: the same exchange
    // with the target left turned.
    bool exchange(const Op& op, const RtLayout& L, uint8_t slots) {
        const bool x = op.m[0] == c128(0.0, 0.0) && op.m[3] == c128(0.0, 0.0) && op.m[1] == c128(1.0, 0.0) &&
                       op.m[2] == c128(1.0, 0.0);
        if (!x || __builtin_popcountll(op.mask) != 1) return false;
        uint32_t rm = 0;
        const std::string c = full_cond(L, op.mask, &rm);
        mark(0xC2u, slots);
        if (turned_q(__builtin_ctzll(op.mask))) {
            const int t = local_of[op.target];
            turned[t] = !turned[t];
            std::swap(pend[t][0], pend[t][1]);
        }
        if (!emit) return true;
        const int tb = slots;
        if (!c.empty()) o << "  { const bool on = " << c << ";\n";
        each_set([&] {
            for (int g = 0; g < kJitAmps; ++g) {
                if ((g & tb) || (static_cast<uint32_t>(g) & rm) != rm) continue;
                const int h = g | tb;
                if (c.empty()) {
                    swap_regs(g, h);
                    continue;
                }
                o << "    { const R xr = " << ar(g) << ", xi = " << ai(g) << ", yr = " << ar(h) << ", yi = " << ai(h) << "; "
                  << ar(g) << " = on ? yr : xr; " << ai(g) << " = on ? yi : xi; " << ar(h) << " = on ? xr : yr; " << ai(h)
                  << " = on ? xi : yi; }\n";
            }
        });
        if (!c.empty()) o << "  }\n";
        return true;
    }

    void ctrl1(const Op& op, const RtLayout& L, uint8_t slots) {
        if (exchange(op, L, slots)) return;
        uint32_t rm = 0;
        const std::string c = turned_cond(L, op.mask, &rm);
        const size_t at = coef.size();
        const bool t = turned_q(op.target);
        for (int e = 0; e < 4; ++e) push(op.m[t ? 3 - e : e]);
        mark(0xC1u, slots);
        flops += 16.0 * (kJitAmps / 2);
        if (!emit) return;
        const int tb = slots;
        o << "  if (" << (c.empty() ? "true" : c) << ") {\n";
        each_set([&] {
        for (int g = 0; g < kJitAmps; ++g) {
            if ((g & tb) || (static_cast<uint32_t>(g) & rm) != rm) continue;
            const int h = g | tb;
            o << "    { const R x0r = " << ar(g) << ", x0i = " << ai(g) << ", x1r = " << ar(h) << ", x1i = " << ai(h) << ";\n"
              << "      " << ar(g) << " = " << cr(at) << " * x0r - " << ci(at) << " * x0i + " << cr(at + 2) << " * x1r - " << ci(at + 2) << " * x1i;\n"
              << "      " << ai(g) << " = " << cr(at) << " * x0i + " << ci(at) << " * x0r + " << cr(at + 2) << " * x1i + " << ci(at + 2) << " * x1r;\n"
              << "      " << ar(h) << " = " << cr(at + 4) << " * x0r - " << ci(at + 4) << " * x0i + " << cr(at + 6) << " * x1r - " << ci(at + 6) << " * x1i;\n"
              << "      " << ai(h) << " = " << cr(at + 4) << " * x0i + " << ci(at + 4) << " * x0r + " << cr(at + 6) << " * x1i + " << ci(at + 6) << " * x1r; }\n";
        }
        });
        o << "  }\n";
    }

    void diag(const Op& op, const RtLayout& L) {
        uint32_t tm = 0;
        for (int b = 0; b < op.k; ++b)
            if (turned_q(static_cast<int>(op.qubits[b]))) tm |= 1u << b;
        // a one-qubit diagonal of phases is owed; any other (a projector, say) keeps its table: tables of
        // owed pairs divide by the first entry and count on moduli near 1
        if (op.k == 1 && is_phase(op.m[0]) && is_phase(op.m[1])) {
            const int q = static_cast<int>(op.qubits[0]);
            c128* p = owed(q);
            for (uint32_t v = 0; v < 2; ++v) p[v] *= op.m[v ^ tm];
            mark(0xEFu, static_cast<uint64_t>(q));
            return;
        }
        const size_t at = coef.size();
        for (uint32_t v = 0; v < op.m.size(); ++v) push(op.m[v ^ tm]);
        // table index bit b <- qubit op.qubits[b]: slot bits are constants per register; lane,
        // warp and outside bits form a per-thread base index
        std::string thr = "0u";
        std::vector<int> slot_bit(op.k, -1);
        uint64_t so = 0;
        for (int b = 0; b < op.k; ++b) {
            const int q = static_cast<int>(op.qubits[b]);
            so = so * 131 + static_cast<uint64_t>(q);
            const int lb = local_of[q];
            if (lb < 0) {
                thr += " | ((unsigned)((base >> " + std::to_string(q) + ") & 1ull) << " + std::to_string(b) + ")";
                continue;
            }
            int k = 0;
            const char w = place(L, lb, &k);
            if (w == 'r') slot_bit[b] = k;
            else thr += std::string(" | (((") + (w == 'l' ? "lane" : "warp") + " >> " + std::to_string(k) + ") & 1u) << " +
                        std::to_string(b) + ")";
        }
        mark(0xE0u + static_cast<uint64_t>(op.k), so);
        flops += 6.0 * kJitAmps;
        if (!emit) return;
        o << "  { const unsigned di = " << thr << ";\n";
        each_set([&] {
        for (int r = 0; r < kJitAmps; ++r) {
            uint32_t cst = 0;
            for (int b = 0; b < op.k; ++b)
                if (slot_bit[b] >= 0 && ((r >> slot_bit[b]) & 1)) cst |= 1u << b;
            o << "    { const unsigned e = " << at << "u + 2u * (di | " << cst << "u); const R pr = P.c[e], pi = P.c[e + 1];"
              << " const R xr = " << ar(r) << ", xi = " << ai(r) << "; "
              << ar(r) << " = pr * xr - pi * xi; " << ai(r) << " = pr * xi + pi * xr; }\n";
        }
        });
        o << "  }\n";
    }

    // exp(-i theta/2 P): P's X/Y bits are register slots (pairs g, g ^ xm); its Z parity splits
    // into a per-register constant, a per-thread part (lane and warp bits) and a per-tile part
    // (qubits outside the tile).  new_g = c a_g + s i^(nY+3) (-1)^parity(h & z) a_h, h = g ^ xm.
    void pauli(const Op& op, const RtLayout& L) {
        uint64_t outx = 0, outz = 0;
        const uint32_t lx = split(op.mask, &outx), lz = split(op.zmask, &outz);
        if (outx) throw std::logic_error("JIT tiles: Pauli rotation with an X bit outside the tile");
        uint32_t xm = 0, zm = 0;
        std::string tz = "0u";
        for (int b = 0; b < kRtQubits; ++b) {
            int k = 0;
            if ((lx >> b) & 1) {
                if (place(L, b, &k) != 'r') throw std::logic_error("JIT tiles: Pauli X bit outside the register slots");
                xm |= 1u << k;
            }
            if ((lz >> b) & 1) {
                const char w = place(L, b, &k);
                if (w == 'r') zm |= 1u << k;
                else tz += std::string(" ^ ((") + (w == 'l' ? "lane" : "warp") + " >> " + std::to_string(k) + ") & 1u)";
            }
        }
        if (outz) tz += " ^ ((unsigned)__popcll(base & " + hex64(outz) + ") & 1u)";
        const int e = (__builtin_popcountll(op.mask & op.zmask) + 3) & 3;
        bool odd = false;     // turned qubits under a Z or Y change the sign of s
        for (int q = 0; q < 64; ++q)
            if ((op.zmask >> q) & 1) odd ^= turned_q(q);
        const size_t at = push(odd ? std::conj(op.m[0]) : op.m[0]);
        mark(0x9Au, xm | (zm << 8) | (static_cast<uint64_t>(e) << 16));
        mark(outz, static_cast<uint64_t>(lz));
        flops += 6.0 * kJitAmps;
        if (!emit) return;
        const int pivot = static_cast<int>(xm & (~xm + 1));
        auto term = [&](int src, std::string* tr, std::string* ti) {
            // (-1)^{parity(src slots & z)} * i^e * a_src, as expressions of the saved values
            const bool neg = __builtin_popcount(static_cast<uint32_t>(src) & zm) & 1;
            const std::string xr = "v" + std::to_string(src) + "r", xi = "v" + std::to_string(src) + "i";
            std::string r, i;
            switch (e) {
                case 0: r = xr; i = xi; break;
                case 1: r = "(-" + xi + ")"; i = xr; break;
                case 2: r = "(-" + xr + ")"; i = "(-" + xi + ")"; break;
                default: r = xi; i = "(-" + xr + ")"; break;
            }
            *tr = neg ? "(-" + r + ")" : r;
            *ti = neg ? "(-" + i + ")" : i;
        };
        o << "  { const unsigned tp = (" << tz << ") & 1u; const R c = " << cr(at) << ", sp = tp ? -" << ci(at)
          << " : " << ci(at) << ";\n";
        each_set([&] {
        for (int g = 0; g < kJitAmps; ++g) {
            if (g & pivot) continue;
            const int h = g ^ static_cast<int>(xm);
            std::string hr, hi, gr, gi;
            term(h, &hr, &hi);
            term(g, &gr, &gi);
            o << "    { const R v" << g << "r = " << ar(g) << ", v" << g << "i = " << ai(g) << ", v" << h << "r = "
              << ar(h) << ", v" << h << "i = " << ai(h) << ";\n"
              << "      " << ar(g) << " = c * v" << g << "r + sp * " << hr << "; " << ai(g) << " = c * v" << g << "i + sp * " << hi << ";\n"
              << "      " << ar(h) << " = c * v" << h << "r + sp * " << gr << "; " << ai(h) << " = c * v" << h << "i + sp * " << gi << "; }\n";
        }
        });
        o << "  }\n";
    }

    void scale(const Op& op) {
        const size_t at = push(op.m[0]);
        mark(0x5Cu);
        flops += 6.0 * kJitAmps;
        if (!emit) return;
        each_set([&] {
            for (int r = 0; r < kJitAmps; ++r) cmul_into(r, cr(at), ci(at));
        });
    }

    // ---- adjoint steps (pair passes).  A step's result is Im <phi|G|psi> (every generator's prefactor is
    // imaginary), as a weighted sum of the pass's accumulators; with the deferred factors of the other
    // qubits unit phases, the stored registers lack only |cglob|^2 of it.
    struct AdjOut {
        int slot;
        std::vector<std::pair<int, double>> acc;   // (accumulator, weight)
    };
    std::vector<AdjOut> outs;
    int n_acc = 0;

    // Emits acc[a] += sum over (f, x, imag, sign) of sign * (Im or Re of conj(phi_f) psi_x), in four
    // running sums so that neighbouring FMAs do not wait for one another.
    struct Product {
        int f, x;
        bool imag, neg;
    };
    int accumulate(const std::vector<Product>& ps) {
        const int a = n_acc++;
        mark(0xAD1u, static_cast<uint64_t>(ps.size()));
        for (const Product& q : ps) mark(static_cast<uint64_t>(q.f) | static_cast<uint64_t>(q.x) << 8, (q.imag ? 1u : 0u) | (q.neg ? 2u : 0u));
        flops += 4.0 * static_cast<double>(ps.size());
        if (!emit) return a;
        o << "  { R v0 = 0, v1 = 0, v2 = 0, v3 = 0;\n";
        for (size_t i = 0; i < ps.size(); ++i) {
            const Product& q = ps[i];
            const std::string fr = "b" + std::to_string(q.f) + "r", fi = "b" + std::to_string(q.f) + "i";
            const std::string xr = "a" + std::to_string(q.x) + "r", xi = "a" + std::to_string(q.x) + "i";
            const std::string v = "v" + std::to_string(i & 3);
            const std::string p = q.neg ? "-" : "", m = q.neg ? "" : "-";
            if (q.imag) o << "    " << v << " = FMA(" << p << fr << ", " << xi << ", " << v << "); " << v << " = FMA(" << m << fi << ", " << xr << ", " << v << ");\n";
            else o << "    " << v << " = FMA(" << p << fr << ", " << xr << ", " << v << "); " << v << " = FMA(" << p << fi << ", " << xi << ", " << v << ");\n";
        }
        o << "    acc[" << a * kJitThreads << "u + tid] += (v0 + v1) + (v2 + v3); }\n";
        return a;
    }

    enum AdjKind { ADJ_NONE, ADJ_DIAG, ADJ_X, ADJ_Y, ADJ_GENERAL };
    static AdjKind adj_kind(const Op& op) {
        if (op.k != 1) return ADJ_GENERAL;
        const std::vector<c128>& G = op.g;
        const bool off0 = G[1] == 0.0 && G[2] == 0.0;
        if (off0 && G[0].imag() == 0 && G[3].imag() == 0 && op.m[1] == 0.0 && op.m[2] == 0.0) return ADJ_DIAG;
        if (G[0] != 0.0 || G[3] != 0.0) return ADJ_NONE;
        if (G[1] == G[2] && G[1].imag() == 0) return ADJ_X;
        if (G[1] == -G[2] && G[1].real() == 0) return ADJ_Y;
        return ADJ_NONE;
    }
    // diagonal generator and dagger: no data moves, the dagger is deferred
    void adj_diag(const RtStep& st, const RtLayout& L) {
        const Op& op = *st.op;
        const int p = st.slot_of[0], b = L.reg[p], B = 1 << p;
        const double w = std::norm(cglob);
        const double z0 = op.g[turned[b] ? 3 : 0].real(), z1 = op.g[turned[b] ? 0 : 3].real();
        AdjOut out{op.slot, {}};
        std::vector<Product> half[2];
        for (int r = 0; r < kJitAmps; ++r) half[(r & B) ? 1 : 0].push_back({r, r, true, false});
        mark(0xAD2u, static_cast<uint64_t>(p));
        if (op.g[0] == -op.g[3]) {
            for (Product& q : half[1]) q.neg = true;
            half[0].insert(half[0].end(), half[1].begin(), half[1].end());
            out.acc.push_back({accumulate(half[0]), w * z0});
        } else {
            out.acc.push_back({accumulate(half[0]), w * z0});
            out.acc.push_back({accumulate(half[1]), w * z1});
        }
        outs.push_back(std::move(out));
        c128* o2 = owed(static_cast<int>(op.qubits[0]));
        o2[0] *= op.m[turned[b] ? 3 : 0];
        o2[1] *= op.m[turned[b] ? 0 : 3];
    }
    // off-diagonal generator: the inner product only (slot phases flushed); the dagger follows
    void adj_off(const RtStep& st, const RtLayout& L, AdjKind kind) {
        const Op& op = *st.op;
        const int p = st.slot_of[0], b = L.reg[p], B = 1 << p;
        // X: Im conj(phi0) psi1 + Im conj(phi1) psi0 times g; Y: Re conj(phi1) psi0 - Re conj(phi0) psi1
        // times Im g10.  On a turned bit Y changes sign.
        double w = std::norm(cglob) * (kind == ADJ_X ? op.g[2].real() : op.g[2].imag());
        if (kind == ADJ_Y && turned[b]) w = -w;
        std::vector<Product> ps;
        for (int g = 0; g < kJitAmps; ++g) {
            if (g & B) continue;
            ps.push_back({g, g | B, kind == ADJ_X, kind == ADJ_Y});
            ps.push_back({g | B, g, kind == ADJ_X, false});
        }
        mark(0xAD3u, static_cast<uint64_t>(p) | static_cast<uint64_t>(kind) << 8);
        outs.push_back({op.slot, {{accumulate(ps), w}}});
    }
    // two-qubit (or global phase) generator with entries 0, +-1, +-i, then its dagger
    bool adj_general(const RtStep& st, const RtLayout& L) {
        const Op& op = *st.op;
        flush_slots(L);
        for (int b = 0; b < op.k; ++b) unturn_slot(L, st.slot_of[b]);
        uint32_t slots = 0;
        for (int b = 0; b < op.k; ++b) slots |= 1u << st.slot_of[b];
        const int D = 1 << op.k;
        std::vector<Product> ps;
        for (int g = 0; g < kJitAmps; ++g) {
            if (g & static_cast<int>(slots)) continue;
            auto reg = [&](int x) {
                int r = g;
                for (int b = 0; b < op.k; ++b)
                    if ((x >> b) & 1) r |= 1 << st.slot_of[b];
                return r;
            };
            for (int y = 0; y < D; ++y)
                for (int x = 0; x < D; ++x) {
                    const c128 e = op.g[static_cast<size_t>(y * D + x)];
                    if (e == 0.0) continue;
                    if (std::abs(e.real()) == 1.0 && e.imag() == 0) ps.push_back({reg(y), reg(x), true, e.real() < 0});
                    else if (std::abs(e.imag()) == 1.0 && e.real() == 0) ps.push_back({reg(y), reg(x), false, e.imag() < 0});
                    else return false;
                }
        }
        mark(0xAD4u, slots);
        const double w = std::norm(cglob);
        outs.push_back({op.slot, {{accumulate(ps), w}}});
        if (op.k == 0) cglob *= op.m[0];
        else dense(op, st.slot_of);
        return true;
    }
    // One-qubit steps between layout changes act on distinct slots or in order on one: per round, every
    // slot's leading diagonal steps (no data moves), then one rotation per slot behind one phase table.
    bool one_qubit_run(const std::vector<const RtStep*>& run, const RtLayout& L) {
        std::vector<const RtStep*> queue[kRtRegBits];
        for (const RtStep* st : run) queue[st->slot_of[0]].push_back(st);
        size_t at[kRtRegBits] = {};
        for (;;) {
            std::vector<const RtStep*> heads;
            for (int p = 0; p < kRtRegBits; ++p) {
                while (at[p] < queue[p].size() && queue[p][at[p]]->kind == RT_ADJ && adj_kind(*queue[p][at[p]]->op) == ADJ_DIAG)
                    adj_diag(*queue[p][at[p]++], L);
                if (at[p] < queue[p].size()) heads.push_back(queue[p][at[p]++]);
            }
            if (heads.empty()) return true;
            flush_slots(L);
            std::vector<const RtStep*> complex_gates;
            int bit_of_slot[kRtRegBits];
            for (int p = 0; p < kRtRegBits; ++p) bit_of_slot[p] = L.reg[p];
            for (const RtStep* st : heads) {
                const std::vector<c128>& m = st->op->m;
                // by the gate's kind, not its entries: an X rotation by 0 has real ones too, and a structure
                // is compiled once for all angles
                bool real_rotation = st->op->y_turn;
                if (st->kind == RT_ADJ) {
                    const AdjKind kind = adj_kind(*st->op);
                    if (kind != ADJ_X && kind != ADJ_Y) return false;
                    adj_off(*st, L, kind);
                    real_rotation = kind == ADJ_Y;
                }
                mark(0xAD5u, real_rotation ? 1u : 0u);
                if (!real_rotation) {
                    // a matrix given to fewer digits than these passes factor by: the interpreted sweep's
                    Factor1q f;
                    if (!factor_unitary(m, &f)) return false;
                    complex_gates.push_back(st);
                    continue;
                }
                // [[c, -s], [s, c]] needs no phases before it (on a turned bit s changes sign)
                const int p = st->slot_of[0], b = L.reg[p];
                rotate(p, b, m[0].real(), turned[b] ? -m[2].real() : m[2].real(), 1.0, 1.0);
            }
            if (!complex_gates.empty()) gate_batch(complex_gates, L, bit_of_slot);
        }
    }

    // shared-memory slot of register r in layout L: complex128 amplitudes take one 16-byte slot
    // each (index swz(local)); complex64 amplitudes are the halves of 16-byte chunks (chunk
    // swz(local >> 1), half local & 1)
    static std::string slot_setup(const RtLayout& L, bool f32) {
        if (!f32) return "const unsigned sf = swz(" + lfix_expr(L) + ");";
        return "const unsigned lf = " + lfix_expr(L) + "; const unsigned sf = swz(lf >> 1), e0 = lf & 1u;";
    }
    static std::string slot_of(const RtLayout& L, int r, bool f32, char set = 'a') {
        const uint32_t lr = reg_local(L, r);
        if (!f32) return std::string(set == 'a' ? "xb" : "yb") + "[sf ^ " + std::to_string(swz(lr)) + "u]";
        return "xf[2u * (sf ^ " + std::to_string(swz(lr >> 1)) + "u) + (e0 ^ " + std::to_string(lr & 1u) + "u)]";
    }

    bool f32 = false;

    void move_to(const RtLayout& from, const RtLayout& to, bool first) {
        mark(0x7Au);
        mark_layout(to);
        if (!emit) return;
        if (!first) o << "  __syncthreads();\n";
        o << "  { " << slot_setup(from, f32) << "\n";
        each_set([&] {
            for (int r = 0; r < kJitAmps; ++r)
                o << "    " << slot_of(from, r, f32, set) << " = MK(" << ar(r) << ", " << ai(r) << ");\n";
        });
        o << "  }\n  __syncthreads();\n  { " << slot_setup(to, f32) << "\n";
        each_set([&] {
            for (int r = 0; r < kJitAmps; ++r)
                o << "    { const R2 x = " << slot_of(to, r, f32, set) << "; " << ar(r) << " = x.x; " << ai(r) << " = x.y; }\n";
        });
        o << "  }\n";
    }
};

// Is every op of the pass one the generator handles?
bool jit_capable(const RtPlan& plan) {
    for (const RtStep& s : plan.steps)
        if (s.kind != RT_XPOSE && s.kind != RT_RELABEL && s.kind != RT_DENSE && s.kind != RT_PHASE &&
            s.kind != RT_CTRL1 && s.kind != RT_DIAG && s.kind != RT_SCALE && s.kind != RT_PAULI && s.kind != RT_ADJ)
            return false;
    return true;
}

const char* kPrelude = R"(
typedef unsigned long long u64;
__device__ __forceinline__ unsigned swz(unsigned i) { return i ^ ((i >> 3 ^ i >> 6 ^ i >> 9) & 7u); }
__device__ __forceinline__ double flip(double a, int m) {
    return __hiloint2double(__double2hiint(a) ^ m, __double2loint(a));
}
__device__ __forceinline__ float flip(float a, int m) { return __int_as_float(__float_as_int(a) ^ m); }
// the bits of i placed at the set bits of m, lowest first
template <typename U>
__device__ __forceinline__ U spread(U i, U m) {
    U r = 0;
    for (; i && m; i >>= 1, m &= m - 1)
        if (i & 1) r |= m & (0 - m);
    return r;
}
__device__ __forceinline__ void cp16(void* dst, const void* src) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(src) : "memory");
}
)";
#ifdef QSV_DEBUG_BOUNDS
// debug build: every global index of a compiled pass is checked against the register; a miss
// is counted in dbg[0] (first index in dbg[1]) and the access goes to amplitude 0 instead
const char* kPreludeDebug = R"(
__device__ __forceinline__ u64 dbg_idx(u64 i, u64 dim, unsigned long long* dbg) {
    if (i < dim) return i;
    if (atomicAdd(dbg, 1ull) == 0ull) dbg[1] = i;
    return 0ull;
}
)";
constexpr bool kJitDebug = true;
#else
const char* kPreludeDebug = "";
constexpr bool kJitDebug = false;
#endif
// Complex128 stores walk a pointer by JitStore::step; complex64 ones, and the debug build's checked ones,
// take an index each (pass_source).
bool jit_walks(bool f32) { return !kJitDebug && !f32; }
static_assert(kRtRegBits == 4, "JitStore::step and the kernels' d0..d3");

// Walk one pass's plan: coefficients, structural signature and (with emit) the steps' source.
// Returns false when the pass needs an op the generator does not handle or too many
// coefficients.
// A pass of a chain starts from the carry of the pass before (cin: phases on its tile qubits
// become its own deferred phases, the others pass through) and, unless it ends the chain,
// hands its deferred phases on (cout) instead of applying them.  *turned: the qubits whose bits the
// pass's store turns back.
bool walk_pass(const TilePass& pass, const RtPlan& plan, int n, Gen* g, RtLayout* last, const Carry* cin,
               bool final, Carry* cout, uint64_t* turned) {
    if (!jit_capable(plan)) return false;
    for (int q = 0; q < 64; ++q) g->local_of[q] = -1;
    for (int j = 0; j < kRtQubits; ++j) g->local_of[pass.tile_qubits[j]] = j;
    g->mark(static_cast<uint64_t>(n), 0x715Eu);
    for (int j = 0; j < kRtQubits; ++j) g->mark(pass.tile_qubits[j]);
    g->mark_layout(plan.load);
    if (cin) {
        uint64_t in_mask = 0;
        for (const QubitPhase& x : cin->phases) {
            const int b = g->local_of[x.q];
            if (b >= 0) {
                g->pend[b][0] = x.p[0];
                g->pend[b][1] = x.p[1];
                g->has[b] = true;
            } else {
                g->outside.push_back(x);
            }
            in_mask |= 1ull << x.q;
        }
        g->cglob = cin->cglob;
        g->normalised = cin->normalised;
        g->mark(0xCA11u, in_mask);
        g->mark(static_cast<uint64_t>(cin->normalised), final ? 1u : 0u);
    }
    RtLayout L = plan.load;
    bool first_move = true;
    const size_t ns = plan.steps.size();
    for (size_t i = 0; i < ns; ++i) {
        const RtStep& st = plan.steps[i];
        switch (st.kind) {
            case RT_XPOSE:
                g->move_to(L, st.layout, first_move);
                first_move = false;
                L = st.layout;
                break;
            case RT_RELABEL: {
                // a SWAP renames two local bits; their deferred phases follow the data
                const int a = g->local_of[st.op->qubits[0]], b = g->local_of[st.op->qubits[1]];
                std::swap(g->pend[a][0], g->pend[b][0]);
                std::swap(g->pend[a][1], g->pend[b][1]);
                std::swap(g->has[a], g->has[b]);
                std::swap(g->turned[a], g->turned[b]);
                g->mark(0x7Bu);
                g->mark_layout(st.layout);
                L = st.layout;
                break;
            }
            case RT_ADJ:
            case RT_DENSE:
                if (g->pair && st.op->k == 1) {
                    std::vector<const RtStep*> run;
                    size_t j = i;
                    for (; j < ns && (plan.steps[j].kind == RT_DENSE || plan.steps[j].kind == RT_ADJ) && plan.steps[j].op->k == 1; ++j)
                        run.push_back(&plan.steps[j]);
                    if (!g->one_qubit_run(run, L)) return false;
                    i = j - 1;
                } else if (st.kind == RT_ADJ) {
                    if (!g->adj_general(st, L)) return false;
                } else if (st.op->k == 1) {
                    std::vector<const RtStep*> batch;
                    uint32_t used = 0;
                    size_t j = i;
                    for (; j < ns && plan.steps[j].kind == RT_DENSE && plan.steps[j].op->k == 1 &&
                           !((used >> plan.steps[j].slot_of[0]) & 1u); ++j) {
                        batch.push_back(&plan.steps[j]);
                        used |= 1u << plan.steps[j].slot_of[0];
                    }
                    int bit_of_slot[kRtRegBits];
                    for (int p = 0; p < kRtRegBits; ++p) bit_of_slot[p] = L.reg[p];
                    g->gate_batch(batch, L, bit_of_slot);
                    i = j - 1;
                } else {
                    g->flush_slots(L);
                    g->dense(*st.op, st.slot_of);
                }
                break;
            case RT_PHASE: g->phase(*st.op, L); break;
            case RT_CTRL1:
                g->flush_slots(L);
                g->ctrl1(*st.op, L, st.slots);
                break;
            case RT_DIAG: g->diag(*st.op, L); break;
            case RT_SCALE: g->scale(*st.op); break;
            case RT_PAULI:
                g->flush_slots(L);
                g->pauli(*st.op, L);
                break;
            default: return false;
        }
    }
    *turned = 0;
    for (int b = 0; b < kRtQubits; ++b)
        if (g->turned[b]) *turned |= 1ull << pass.tile_qubits[b];
    if (final || !cout) {
        g->flush_all(L);
    } else {
        cout->phases = g->outside;
        for (int b = 0; b < kRtQubits; ++b)
            if (g->has[b]) {
                QubitPhase x;
                x.q = static_cast<int>(pass.tile_qubits[b]);
                // the store puts turned bits back
                x.p[0] = g->pend[b][g->turned[b] ? 1 : 0];
                x.p[1] = g->pend[b][g->turned[b] ? 0 : 1];
                cout->phases.push_back(x);
            }
        std::sort(cout->phases.begin(), cout->phases.end(),
                  [](const QubitPhase& a, const QubitPhase& b) { return a.q < b.q; });
        cout->cglob = g->cglob;
        cout->normalised = g->normalised;
        g->mark(0xCA12u);
    }
    *last = L;
    return g->coef.size() <= kJitMaxCoefDoubles;
}

// Source of one pass kernel (qsv_jit_<idx>) from a walk with emit on.  Complex128: 16-byte
// amplitudes, 16 staged copies of one amplitude per thread, 64 KiB of shared memory, two CTAs
// per SM.  Complex64: 8-byte amplitudes held as float2 (packed FMAs), 8 staged copies of two
// amplitudes per thread, 32 KiB, three CTAs per SM (85 registers; 31.6 ms against 34.4 ms with
// two on the 28-qubit brickwork, and four no faster).
std::string pass_source(const TilePass& pass, const RtPlan& plan, int n, int idx, const std::string& steps,
                        size_t n_coef, const RtLayout& F, bool f32, bool pair, int n_acc) {
    const std::string sets = pair ? "ab" : "a";
    auto re = [](char set, int r) { return set + std::to_string(r) + "r"; };
    auto im = [](char set, int r) { return set + std::to_string(r) + "i"; };
    const size_t nc = std::max<size_t>(n_coef, 1);
    // tile base: the bits of t deposited into the non-tile qubit positions, ascending
    std::vector<int> outside;
    uint32_t in_tile[64] = {};
    for (int j = 0; j < kRtQubits; ++j) in_tile[pass.tile_qubits[j]] = 1;
    for (int q = 0; q < n; ++q)
        if (!in_tile[q]) outside.push_back(q);
    auto deposit = [&](const char* var) {
        std::string base = "0ull";
        for (size_t j = 0; j < outside.size();) {
            size_t e = j;
            while (e + 1 < outside.size() &&
                   outside[e + 1] - static_cast<int>(e + 1) == outside[j] - static_cast<int>(j)) ++e;
            const uint32_t mask = ((1u << (e - j + 1)) - 1u) << j;
            base += std::string(" | ((u64)(") + var + " & " + std::to_string(mask) + "u) << " + std::to_string(outside[j] - static_cast<int>(j)) + ")";
            j = e + 1;
        }
        return base;
    };
    const uint32_t* tq = pass.tile_qubits.data();
    // staging: 16-byte chunk c = tid + 256 j holds local amplitude c (complex128) or the pair
    // 2c, 2c + 1 (complex64); local bit b of the chunk's first amplitude sits at qubit tq[b]
    const int low = f32 ? 1 : 0;                 // local bits below the chunk index
    const int chunks = (1 << kRtQubits) >> low;
    std::string gtid = "0ull";
    for (int b = 0; b < 8; ++b)
        gtid += " | ((u64)((tid >> " + std::to_string(b) + ") & 1u) << " + std::to_string(tq[b + low]) + ")";
    // store: the last layout's lanes are local bits 0..4
    std::string gfin = "0ull";
    for (int k = 0; k < kRtLaneBits; ++k)
        gfin += " | ((u64)((lane >> " + std::to_string(k) + ") & 1u) << " + std::to_string(tq[F.lane[k]]) + ")";
    for (int k = 0; k < kRtWarpBits; ++k)
        gfin += " | ((u64)((warp >> " + std::to_string(k) + ") & 1u) << " + std::to_string(tq[F.warp[k]]) + ")";
    // a global amplitude index: checked against the register in the debug build
    const std::string dim = hex64(1ull << n);
    auto at = [&](const std::string& e) {
        return kJitDebug ? "dbg_idx(" + e + ", " + dim + ", dbg)" : "(" + e + ")";
    };
    auto issue = [&](const std::string& b) {
        std::ostringstream x;
        for (int j = 0; j < chunks / kJitThreads; ++j) {
            uint64_t gj = 0;
            for (int b2 = 0; b2 < 4 && 8 + low + b2 < kRtQubits; ++b2)
                if ((j >> b2) & 1) gj |= 1ull << tq[8 + low + b2];
            for (char set : sets)
                x << "    cp16(" << (set == 'a' ? "xb" : "yb") << " + (stid ^ " << swz(static_cast<uint32_t>(j) * kJitThreads)
                  << "u), " << (set == 'a' ? "s" : "s2") << " + " << at("(" + b + ") | gtid | " + hex64(gj)) << ");\n";
        }
        return x.str();
    };
    // pair passes, which have registers to spare, form the store's strides themselves (24 qubits, 8 layers:
    // 10.94 ms, 11.10 with parameters)
    std::string strides;
    for (int p = 0; p < kRtRegBits && pair && jit_walks(f32); ++p) {
        const std::string q = std::to_string(tq[F.reg[p]]);
        strides += "  const long long d" + std::to_string(p) + " = (turned >> " + q + ") & 1 ? -(1ll << " + q + ") : 1ll << " + q + ";\n";
    }
    const std::string ix = f32 ? "u64" : "unsigned";      // tile numbers
    std::ostringstream s;
    if (f32) {
        s << "typedef float R; typedef float2 R2;\n#define FMA fmaf\n#define MK make_float2\n";
        for (int r = 0; r < kJitAmps; ++r) s << "#define a" << r << "r a" << r << ".x\n#define a" << r << "i a" << r << ".y\n";
    } else {
        s << "typedef double R; typedef double2 R2;\n#define FMA fma\n#define MK make_double2\n";
    }
    s << "struct __align__(8) C" << idx << " { R c[" << nc << "]; };\n"
      << "extern \"C\" __global__ void __launch_bounds__(" << kJitThreads << ", " << (pair ? 1 : jit_ctas(f32))
      << ") qsv_jit_" << idx << "(R2* __restrict__ s, " << ix << " n_tiles, " << ix << " tmask, " << ix << " tstep, u64 turned, "
      << (jit_walks(f32) && !pair ? "long long d0, long long d1, long long d2, long long d3, " : "")
      << (pair ? "R2* __restrict__ s2, double2* __restrict__ partials, " : "") << "const __grid_constant__ C" << idx << " P"
      << (kJitDebug ? ", unsigned long long* __restrict__ dbg" : "") << ") {\n"
      << "  extern __shared__ __align__(16) unsigned char smem[];\n"
      << "  double2* xb = reinterpret_cast<double2*>(smem);\n"
      << "  R2* xf = reinterpret_cast<R2*>(smem);\n";
    if (pair)
        s << "  double2* yb = xb + " << (1 << kRtQubits) << ";\n  double* acc = reinterpret_cast<double*>(yb + "
          << (1 << kRtQubits) << ");\n  for (unsigned k = 0; k < " << n_acc << "u; ++k) acc[k * " << kJitThreads
          << "u + threadIdx.x] = 0;\n";
    s << "  const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;\n"
      << "  const u64 gtid = " << gtid << ";\n"
      << "  const unsigned stid = swz(tid);\n"
      << "  const u64 gfin = " << gfin << ";\n"
      // the i-th tile is the i-th subset of tmask; tstep = spread(gridDim.x, tmask), added with the
      // carries running through the other bits
      << "  " << ix << " i = blockIdx.x, t = spread(i, tmask);\n"
      << strides
      << "  if (i < n_tiles) {\n    const u64 b0 = " << deposit("t") << ";\n" << issue("b0") << "  }\n"
      << "  asm volatile(\"cp.async.commit_group;\\n\" ::: \"memory\");\n"
      << "  for (; i < n_tiles; i += gridDim.x, t = ((t | ~tmask) + tstep) & tmask) {\n"
      << "  const u64 base = " << deposit("t") << ";\n"
      << "  asm volatile(\"cp.async.wait_group 0;\\n\" ::: \"memory\");\n"
      << "  __syncthreads();\n"
      << "  ";
    if (f32) {
        // complex64 amplitudes are float2 pairs (packed FMAs); aNr / aNi name their halves
        s << "R2 ";
        for (int r = 0; r < kJitAmps; ++r) s << (r ? ", a" : "a") << r;
    } else {
        s << "R ";
        for (char set : sets)
            for (int r = 0; r < kJitAmps; ++r) s << (r || set == 'b' ? ", " : "") << re(set, r) << ", " << im(set, r);
    }
    s << ";\n  { " << Gen::slot_setup(plan.load, f32) << "\n";
    for (char set : sets)
        for (int r = 0; r < kJitAmps; ++r)
            s << "    { const R2 x = " << Gen::slot_of(plan.load, r, f32, set) << "; " << re(set, r) << " = x.x; "
              << im(set, r) << " = x.y; }\n";
    // one buffer serves the tile's loads and its transposes: the next tile's copies start once
    // the last transpose has been read, and run under this tile's stores (and the other CTAs
    // on the SM compute meanwhile)
    s << "  }\n  __syncthreads();\n"
      << steps
      << "  __syncthreads();\n"
      << "  if (i + gridDim.x < n_tiles) {\n    const " << ix << " tn = ((t | ~tmask) + tstep) & tmask;\n    const u64 b1 = " << deposit("tn")
      << ";\n" << issue("b1") << "  }\n"
      << "  asm volatile(\"cp.async.commit_group;\\n\" ::: \"memory\");\n";
    s << "  const u64 to = (base | gfin) ^ turned;\n";
    for (int r = 0; r < kJitAmps && !jit_walks(f32); ++r) {
        uint64_t gc = 0;
        for (int p = 0; p < kRtRegBits; ++p)
            if ((r >> p) & 1) gc |= 1ull << tq[F.reg[p]];
        for (char set : sets)
            s << "  __stcs(" << (set == 'a' ? "s" : "s2") << " + " << at("to ^ " + hex64(gc)) << ", MK(" << re(set, r) << ", "
              << im(set, r) << "));\n";
    }
    // The slots in Gray order, a pointer stepping by a slot bit's stride, negative where the bit is turned.
    // The strides are kernel parameters and tile numbers 32-bit: formed in the kernel and 64-bit they
    // took the registers that the amplitudes need (28 qubits, depth 20, complex128: 47.1 -> 46.3 ms
    // applied again and again; an XOR and a scaled address per store 47.3).
    if (jit_walks(f32)) {
        for (char set : sets) s << "  R2* w" << set << " = " << (set == 'a' ? "s" : "s2") << " + to;\n";
        for (int k = 0, r = 0; k < kJitAmps; ++k) {
            for (char set : sets) s << "  __stcs(w" << set << ", MK(" << re(set, r) << ", " << im(set, r) << "));\n";
            if (k + 1 == kJitAmps) break;
            const int p = __builtin_ctz(static_cast<unsigned>(k + 1));
            for (char set : sets) s << "  w" << set << ((r >> p) & 1 ? " -= d" : " += d") << p << ";\n";
            r ^= 1 << p;
        }
    }
    s << "  }\n  asm volatile(\"cp.async.wait_group 0;\\n\" ::: \"memory\");\n";
    if (pair)
        s << "  __syncthreads();\n  for (unsigned k = warp; k < " << n_acc << "u; k += " << kJitThreads / 32 << "u) {\n"
          << "    double v = 0;\n    for (unsigned j = lane; j < " << kJitThreads << "u; j += 32u) v += acc[k * " << kJitThreads
          << "u + j];\n    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);\n"
          << "    if (lane == 0) partials[(u64)k * gridDim.x + blockIdx.x] = make_double2(v, 0);\n  }\n";
    s << "}\n";
    return s.str();
}

// Source (with emit) or only the signature and coefficients (without) of one pass; `pair`: a pass of the
// reverse sweep, with its adjoint steps' results in `outs`.
bool gen_pass(const TilePass& pass, const RtPlan& plan, int n, int idx, bool emit, bool f32, bool pair, std::string* src,
              std::vector<double>* coef, uint64_t* sig_hash, JitStore* store, double* flops_per_amp = nullptr,
              const Carry* cin = nullptr, bool final = true, Carry* cout = nullptr, std::vector<Gen::AdjOut>* outs = nullptr,
              int* n_acc = nullptr) {
    Gen g;
    g.emit = emit;
    g.f32 = f32;
    g.pair = pair;
    g.mark(pair ? 0xFADu : f32 ? 0xF32u : 0xF64u);
    RtLayout last{};
    if (!walk_pass(pass, plan, n, &g, &last, cin, final, cout, &store->turned)) return false;
    for (int p = 0; p < kRtRegBits; ++p) {
        const uint32_t q = pass.tile_qubits[last.reg[p]];
        store->step[p] = (store->turned >> q) & 1 ? -(1ll << q) : 1ll << q;
    }
    if (g.n_acc > kPairMaxAcc) return false;
    uint64_t h = 1469598103934665603ull;
    for (uint64_t v : g.sig)
        for (int b = 0; b < 8; ++b) {
            h ^= (v >> (8 * b)) & 0xffu;
            h *= 1099511628211ull;
        }
    *sig_hash = h;
    if (flops_per_amp) *flops_per_amp = g.flops / kJitAmps;
    if (emit) *src = pass_source(pass, plan, n, idx, g.o.str(), g.coef.size(), last, f32, pair, g.n_acc);
    if (outs) outs->swap(g.outs);
    if (n_acc) *n_acc = g.n_acc;
    coef->swap(g.coef);
    if (coef->empty()) coef->push_back(0.0);
    return true;
}

uint64_t fnv1a(const std::string& s) {
    uint64_t h = 1469598103934665603ull;
    for (unsigned char c : s) {
        h ^= c;
        h *= 1099511628211ull;
    }
    return h;
}

std::string cache_dir() {
    if (const char* e = std::getenv("QSV_JIT_CACHE")) return e;
    const char* home = std::getenv("HOME");
    return std::string(home ? home : "/tmp") + "/.cache/openqarp_b200/jit";
}

std::vector<char> read_file(const std::string& path) {
    std::ifstream f(path, std::ios::binary);
    if (!f) return {};
    return std::vector<char>((std::istreambuf_iterator<char>(f)), std::istreambuf_iterator<char>());
}

void write_file(const std::string& path, const std::vector<char>& data) {
    const std::string dir = cache_dir();
    // create the directory chain (mkdir -p) without a shell
    for (size_t i = 1; i <= dir.size(); ++i)
        if (i == dir.size() || dir[i] == '/') {
            const std::string part = dir.substr(0, i);
            mkdir(part.c_str(), 0755);
        }
    const std::string tmp = path + ".tmp" + std::to_string(getpid());
    {
        std::ofstream f(tmp, std::ios::binary);
        if (!f) return;
        f.write(data.data(), static_cast<std::streamsize>(data.size()));
    }
    std::rename(tmp.c_str(), path.c_str());
}

std::vector<char> compile_cubin(const std::string& src, int cc_major, int cc_minor) {
    const Nvrtc& api = nvrtc();
    nvrtcProgram prog = nullptr;
    if (api.create(&prog, src.c_str(), "qsv_jit_tiles.cu", 0, nullptr, nullptr) != NVRTC_SUCCESS)
        throw std::runtime_error("JIT tiles: nvrtcCreateProgram failed");
    const std::string arch = "-arch=sm_" + std::to_string(cc_major) + std::to_string(cc_minor) +
                             (cc_major >= 9 ? "a" : "");
    const char* opts[] = {arch.c_str(), "-std=c++17", "-default-device", "-lineinfo"};
    const nvrtcResult rc = api.compile(prog, 4, opts);
    if (rc != NVRTC_SUCCESS) {
        size_t ls = 0;
        api.log_size(prog, &ls);
        std::string log(ls, '\0');
        if (ls) api.log(prog, &log[0]);
        api.destroy(&prog);
        throw std::runtime_error("JIT tiles: NVRTC compile failed: " + log.substr(0, 2000));
    }
    size_t cs = 0;
    api.cubin_size(prog, &cs);
    std::vector<char> cubin(cs);
    api.cubin(prog, cubin.data());
    api.destroy(&prog);
    return cubin;
}

// Walk every pass of a plan without emitting source.  Consecutive compiled passes form a
// chain: each hands its deferred phases to the next (one fewer full-register multiply per
// pass, and the next pass's first table absorbs them), and the chain's last pass applies
// everything owed.  A pass that breaks a chain (not compiled, or a stream pass) ends it.  If a
// pass fails only with carried phases (too many coefficients), the plan is walked without
// carrying.
struct PassWalk {
    bool ok = false;
    uint64_t sig = 0;
    std::vector<double> coef;
    double flops_per_amp = 0;
    bool has_cin = false;
    Carry cin;
    bool final = true;
    JitStore store;
    std::vector<Gen::AdjOut> outs;
    int n_acc = 0;
};

std::vector<PassWalk> walk_all(const std::vector<const TilePass*>& passes, std::vector<RtPlan>& plans, int n,
                               bool f32, bool pair = false) {
    const size_t np = passes.size();
    plans.assign(np, RtPlan{});
    std::vector<PassWalk> alone(np);
    for (size_t i = 0; i < np; ++i) {
        if (passes[i]->tile_qubits.empty()) continue;
        if (!plan_rt(*passes[i], &plans[i], f32 ? 8 : 16)) continue;
        std::string unused;
        PassWalk& w = alone[i];
        w.ok = gen_pass(*passes[i], plans[i], n, 0, false, f32, pair, &unused, &w.coef, &w.sig, &w.store,
                        &w.flops_per_amp, nullptr, true, nullptr, &w.outs, &w.n_acc);
    }
    std::vector<PassWalk> chained(np);
    Carry cur;
    bool in_chain = false;
    for (size_t i = 0; i < np; ++i) {
        if (!alone[i].ok) {
            in_chain = false;
            continue;
        }
        PassWalk& w = chained[i];
        w.final = !(i + 1 < np && alone[i + 1].ok);
        w.has_cin = in_chain;
        if (in_chain) w.cin = cur;
        Carry next;
        std::string unused;
        w.ok = gen_pass(*passes[i], plans[i], n, 0, false, f32, pair, &unused, &w.coef, &w.sig, &w.store,
                        &w.flops_per_amp, w.has_cin ? &w.cin : nullptr, w.final, w.final ? nullptr : &next, &w.outs, &w.n_acc);
        if (!w.ok) return alone;
        cur = std::move(next);
        in_chain = !w.final;
    }
    return chained;
}

std::mutex g_jit_mu;

#ifdef QSV_DEBUG_BOUNDS
// the compiled passes' fault words (count, first index), one per device, polled with the other
// translation units' records after every entry point
std::mutex g_dbg_mu;
std::map<int, unsigned long long*> g_dbg_words;

unsigned long long* jit_fault_word(int device) {
    std::lock_guard<std::mutex> lock(g_dbg_mu);
    unsigned long long*& w = g_dbg_words[device];
    if (!w) {
        check_cuda(dev_malloc(&w, 2 * sizeof(unsigned long long)), "JIT debug word");
        check_cuda(cudaMemset(w, 0, 2 * sizeof(unsigned long long)), "JIT debug word");
    }
    return w;
}

void jit_dbg_sync(const ::qsv::dbg::Ranges&) {}

void jit_dbg_poll(::qsv::dbg::Fault* out) {
    *out = ::qsv::dbg::Fault{};
    int device = 0;
    cudaGetDevice(&device);
    unsigned long long* w = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_dbg_mu);
        auto it = g_dbg_words.find(device);
        if (it == g_dbg_words.end()) return;
        w = it->second;
    }
    unsigned long long h[2] = {0, 0};
    cudaMemcpy(h, w, sizeof h, cudaMemcpyDeviceToHost);
    if (!h[0]) return;
    out->count = h[0];
    out->addr = h[1];   // an amplitude index, not an address
    out->line = 0;
    out->bytes = 0;
    cudaMemset(w, 0, sizeof h);
}

[[maybe_unused]] const bool g_jit_dbg_registered =
    ::qsv::dbg::register_unit("compiled tile pass (index)", &jit_dbg_sync, &jit_dbg_poll);
#endif
// compiled pass kernels, by (source hash, context); modules stay loaded until exit
std::map<std::pair<uint64_t, CUcontext>, CUfunction> g_kernels;

}  // namespace

// ---------------------------------------------------------------- public

JitPlan jit_prepare(const std::vector<const TilePass*>& passes, int n, int device, bool f32, bool pair) {
    JitPlan out;
    out.f32 = f32;
    out.pair = pair;
    out.idx.assign(passes.size(), -1);
    int major = 0, minor = 0;
    check_cuda(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device), "compute capability");
    check_cuda(cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device), "compute capability");
    const std::string tag = "// sm_" + std::to_string(major) + std::to_string(minor) + "\n";
    const Driver& drv = driver();
    CUcontext ctx = nullptr;
    check_cu(drv.current(&ctx), "cuCtxGetCurrent");
    // walk every pass without emitting source: its signature finds a compiled kernel
    std::vector<size_t> pass_of;
    std::vector<uint64_t> sigs;
    std::vector<RtPlan> plans;
    std::vector<PassWalk> walks = walk_all(passes, plans, n, f32, pair);
    for (size_t i = 0; i < passes.size(); ++i) {
        PassWalk& w = walks[i];
        if (!w.ok && pair && !passes[i]->tile_qubits.empty()) return JitPlan{};   // all of a sweep, or none
        if (!w.ok) continue;
        out.flops_per_amp.push_back(w.flops_per_amp);
        out.store.push_back(w.store);
        out.n_acc.push_back(w.n_acc);
        for (Gen::AdjOut& a : w.outs) {
            for (auto& [acc, weight] : a.acc) acc += out.total_acc;
            out.adj.push_back({a.slot, std::move(a.acc)});
        }
        out.acc0.push_back(out.total_acc);
        out.total_acc += w.n_acc;
        const uint64_t sig = w.sig ^ (static_cast<uint64_t>(major) << 56) ^ (static_cast<uint64_t>(minor) << 48);
        out.idx[i] = static_cast<int>(sigs.size());
        sigs.push_back(sig);
        pass_of.push_back(i);
        // kernel parameters in the storage type's precision
        std::vector<uint8_t> arg;
        if (f32) {
            std::vector<float> c(w.coef.begin(), w.coef.end());
            arg.assign(reinterpret_cast<const uint8_t*>(c.data()), reinterpret_cast<const uint8_t*>(c.data() + c.size()));
        } else {
            arg.assign(reinterpret_cast<const uint8_t*>(w.coef.data()),
                       reinterpret_cast<const uint8_t*>(w.coef.data() + w.coef.size()));
        }
        out.coef.push_back(std::move(arg));
    }
    if (sigs.empty()) return out;
    std::lock_guard<std::mutex> lock(g_jit_mu);
    std::vector<size_t> missing;
    for (size_t k = 0; k < sigs.size(); ++k)
        if (!g_kernels.count({sigs[k], ctx})) missing.push_back(k);
    if (!missing.empty()) {
        // sources of the missing passes; their cubins from the disk cache or compiled on the
        // host cores in parallel
        std::vector<std::string> srcs(missing.size());
        std::vector<std::string> files(missing.size());
        std::vector<std::vector<char>> cubins(missing.size());
        std::vector<size_t> todo;
        for (size_t j = 0; j < missing.size(); ++j) {
            const size_t i = pass_of[missing[j]];
            const PassWalk& w = walks[i];
            std::vector<double> coef;
            uint64_t sig = 0;
            JitStore store;
            Carry next;
            gen_pass(*passes[i], plans[i], n, 0, true, f32, pair, &srcs[j], &coef, &sig, &store, nullptr,
                     w.has_cin ? &w.cin : nullptr, w.final, w.final ? nullptr : &next);
            srcs[j] = std::string(kPrelude) + kPreludeDebug + srcs[j] + tag;
            char name[40];
            std::snprintf(name, sizeof name, "%016llx.cubin", static_cast<unsigned long long>(fnv1a(srcs[j])));
            files[j] = cache_dir() + "/" + name;
            cubins[j] = read_file(files[j]);
            if (cubins[j].empty()) todo.push_back(j);
        }
        if (!todo.empty()) {
            const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
            std::vector<std::thread> pool;
            std::vector<std::string> errors(todo.size());
            std::atomic<size_t> next{0};
            for (unsigned w = 0; w < std::min<size_t>(hw, todo.size()); ++w)
                pool.emplace_back([&] {
                    for (size_t t = next++; t < todo.size(); t = next++) {
                        try {
                            cubins[todo[t]] = compile_cubin(srcs[todo[t]], major, minor);
                        } catch (const std::exception& e) {
                            errors[t] = e.what();
                        }
                    }
                });
            for (std::thread& t : pool) t.join();
            for (const std::string& e : errors)
                if (!e.empty()) throw std::runtime_error(e);
            for (size_t j : todo) write_file(files[j], cubins[j]);
        }
        for (size_t j = 0; j < missing.size(); ++j) {
            CUmodule mod = nullptr;
            check_cu(drv.load(&mod, cubins[j].data()), "cuModuleLoadData (JIT tiles)");
            CUfunction f = nullptr;
            check_cu(drv.get_function(&f, mod, "qsv_jit_0"), "cuModuleGetFunction (JIT tiles)");
            check_cu(drv.set_attribute(f, CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES,
                                       static_cast<int>(pair ? pair_smem(kPairMaxAcc) : jit_smem(f32))),
                     "cuFuncSetAttribute (JIT tiles)");
            g_kernels[{sigs[missing[j]], ctx}] = f;
        }
    }
    for (size_t k = 0; k < sigs.size(); ++k) out.fns.push_back(g_kernels[{sigs[k], ctx}]);
    return out;
}

namespace {
void launch_pass(const JitPlan& plan, int pass, void* s, void* s2, double2* partials, int n, uint64_t tiles,
                 cudaStream_t st) {
    const int k = plan.idx.at(pass);
    if (k < 0) throw std::logic_error("JIT tiles: pass was not compiled");
    int sms = 0, device = 0;
    check_cuda(cudaGetDevice(&device), "device");
    check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "sm count");
    // tile numbers take n - 12 bits
    static_assert(QSV_MAX_QUBITS - kRtQubits < 32, "tile numbers are 32-bit in the kernels");
    unsigned long long tmask = tiles & ((1ull << (n - kRtQubits)) - 1);    // a 32-bit parameter takes the low half
    unsigned long long n_tiles = 1ull << __builtin_popcountll(tmask);
    // a pair pass writes its partials by block: the grid its caller sized them for
    const unsigned grid = plan.pair ? adjoint_tile_grid(n, kRtQubits)
                                    : static_cast<unsigned>(std::min<uint64_t>(
                                          n_tiles, static_cast<uint64_t>(jit_ctas(plan.f32)) * static_cast<uint64_t>(sms)));
    const std::vector<uint8_t>& c = plan.coef[static_cast<size_t>(k)];
    JitStore store = plan.store[static_cast<size_t>(k)];
    unsigned long long tstep = 0;      // spread(grid, tmask)
    for (unsigned long long i = grid, m = tmask; i && m; i >>= 1, m &= m - 1)
        if (i & 1) tstep |= m & (0 - m);
    double2* part = partials ? partials + static_cast<size_t>(plan.acc0[static_cast<size_t>(k)]) * grid : nullptr;
    std::vector<void*> args{&s, &n_tiles, &tmask, &tstep, &store.turned};
    if (jit_walks(plan.f32) && !plan.pair)
        for (long long& d : store.step) args.push_back(&d);
    if (plan.pair) args.insert(args.end(), {static_cast<void*>(&s2), static_cast<void*>(&part)});
    args.push_back(const_cast<uint8_t*>(c.data()));
#ifdef QSV_DEBUG_BOUNDS
    unsigned long long* dbg = jit_fault_word(device);
    args.push_back(&dbg);
#endif
    const size_t smem = plan.pair ? pair_smem(plan.n_acc[static_cast<size_t>(k)]) : jit_smem(plan.f32);
    check_cu(driver().launch(static_cast<CUfunction>(plan.fns[static_cast<size_t>(k)]), grid, 1, 1, kJitThreads, 1, 1,
                             static_cast<unsigned>(smem), reinterpret_cast<CUstream>(st), args.data(), nullptr),
             "cuLaunchKernel (JIT tiles)");
}
}  // namespace

void jit_launch(const JitPlan& plan, int pass, void* s, int n, uint64_t tmask, cudaStream_t st) {
    launch_pass(plan, pass, s, nullptr, nullptr, n, tmask, st);
}

void jit_launch_pair(const JitPlan& plan, int pass, void* psi, void* phi, double2* partials, int n, cudaStream_t st) {
    launch_pass(plan, pass, psi, phi, partials, n, ~0ull, st);
}

bool run_adjoint_compiled(const std::vector<Op>& ops, double2* psi, double2* phi, int n, double2* partials, unsigned nb,
                          cudaStream_t st, const std::function<void()>& settle,
                          const std::function<void(const Op&)>& stream_op, uint64_t* launches, int* n_acc,
                          std::vector<JitPlan::Adj>* steps) {
    if (ops.empty()) return true;
    if (nb != adjoint_tile_grid(n, kRtQubits)) throw std::logic_error("adjoint partials sized for another grid");
    // a pass ends where its accumulators or its parameters would overflow (at most 32 doubles of phase
    // table and ratio a step, or the step's matrix)
    std::vector<TilePass> passes;
    // Seeded plans save a pass now and then and take the host 0.2 ms more for 400 steps: a pass takes that
    // long from 24 qubits on (14 qubits, 3 layers: 601 -> 568 us without; 22 qubits, 8 layers 4.35 -> 4.14 ms).
    for (TilePass& p : plan_tiles(ops, n, kRtQubits, coalesced_low_qubits(16), n < 24 ? 0 : kJitPlanSeeds)) {
        if (p.tile_qubits.empty()) {
            for (const Op& o : p.ops)
                if (o.kind == OP_ADJ) return false;
            passes.push_back(std::move(p));
            continue;
        }
        TilePass cur;
        int acc = 0;
        size_t words = 0;
        auto close = [&] {
            if (cur.ops.empty()) return;
            cur.tile_qubits = p.tile_qubits;
            cur.low = p.low;
            passes.push_back(std::move(cur));
            cur = TilePass{};
            acc = 0;
            words = 0;
        };
        for (Op& o : p.ops) {
            const int a = o.kind != OP_ADJ ? 0 : o.k == 1 ? 2 : 1;
            const size_t w = 34 + 2 * o.m.size();
            if (acc + a > kPairMaxAcc || words + w > kJitMaxCoefDoubles - 400) close();
            acc += a;
            words += w;
            cur.ops.push_back(std::move(o));
        }
        close();
    }
    std::vector<const TilePass*> ptrs;
    for (const TilePass& p : passes) ptrs.push_back(&p);
    int device = 0;
    check_cuda(cudaGetDevice(&device), "device");
    JitPlan plan = jit_prepare(ptrs, n, device, false, true);
    if (plan.idx.empty()) return false;
    settle();
    for (size_t i = 0; i < passes.size(); ++i) {
        if (passes[i].tile_qubits.empty()) {
            for (const Op& o : passes[i].ops) stream_op(o);
            continue;
        }
        jit_launch_pair(plan, static_cast<int>(i), psi, phi, partials + static_cast<size_t>(*n_acc) * nb, n, st);
        ++*launches;
    }
    for (JitPlan::Adj& a : plan.adj) {
        for (auto& [acc, weight] : a.acc) acc += *n_acc;
        steps->push_back(std::move(a));
    }
    *n_acc += plan.total_acc;
    return true;
}

std::string jit_source_for_test(const std::vector<const TilePass*>& passes, int n, bool f32, size_t* n_kernels) {
    std::string src = std::string(kPrelude) + kPreludeDebug;
    int next = 0;
    std::vector<RtPlan> plans;
    const std::vector<PassWalk> walks = walk_all(passes, plans, n, f32);
    for (size_t i = 0; i < passes.size(); ++i) {
        const PassWalk& w = walks[i];
        if (!w.ok) continue;
        std::string ps;
        std::vector<double> coef;
        uint64_t sig = 0;
        JitStore store;
        Carry out;
        if (!gen_pass(*passes[i], plans[i], n, next, true, f32, false, &ps, &coef, &sig, &store, nullptr,
                      w.has_cin ? &w.cin : nullptr, w.final, w.final ? nullptr : &out))
            continue;
        if (next > 0) {
            // one program holds every pass: the type definitions come once, with the first
            const size_t cut = ps.find("struct __align__");
            ps = ps.substr(cut);
        }
        src += ps;
        ++next;
    }
    *n_kernels = static_cast<size_t>(next);
    return src;
}

std::vector<char> jit_compile_for_test(const std::string& src, int cc_major, int cc_minor) {
    return compile_cubin(src, cc_major, cc_minor);
}

}  // namespace qsv
