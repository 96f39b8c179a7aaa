// kern_qaoa.cu — batched QAOA MaxCut: many instances of uneven width in one persistent launch.
//
// The reference evaluates such sweeps one circuit at a time (QarpEngine._sweep,
// src/qarp/engines/_qarp_engine.py:450-503; QarpSimulator::batch_expectation,
// qarp_simulator.cpp:971-984), each a full statevector + expectation (+ adjoint) on the CPU.
// Here one CTA per SM pulls instances from a work queue (heaviest first) and runs the whole
// instance — forward circuit, <C>, and the adjoint gradient of every gamma and beta — with
// its half register in shared memory and registers (n <= 13) or streamed through tiles of 2^11
// amplitudes (2^12 above 22 qubits) from an HBM buffer.
//
// Circuit (the same commands circuits.qaoa_maxcut emits): H on every qubit, then for each
// round r: RZZ(2 gamma_r) on every edge — together the diagonal phase exp(-i gamma_r D(z)),
// D(z) = sum_e s_u s_v = E - 2 cut(z) — and RX(2 beta_r) on every qubit.
// Cost: C(z) = sum_e (1 - s_u s_v) / 2 = cut(z).
// Adjoint (run_gradient_core, qarp_simulator.cpp:1519-1605, applied per commuting layer):
// phi = C psi; for r = p-1..0: dE/dbeta_r = 2 Im <phi| sum_q X_q |psi>, un-apply the mixer;
// dE/dgamma_r = 2 Im <phi| D |psi>, un-apply the phase.  (RX and RZZ generators are -i/2 P
// with d angle / d param = 2, so each term is 2 * 2 Re(-i/2 <phi|P|psi>) = 2 Im <phi|P|psi>.)
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <numeric>
#include <stdexcept>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/qsv.h"
#include "kernels.h"

namespace qsv {

namespace {

constexpr int kQThreads = 512;
constexpr int kQMaxEdges = 96;
constexpr int kQMaxQubits = 24;
constexpr int kQMaxDepth = 64;
constexpr int kQMaxLayers = 7;           // adjacency bit planes: an edge may be listed up to 96 times
constexpr int kQSmallBits = 12;          // half registers of up to 2^12 amplitudes stay on chip
constexpr int kQTile = 1 << kQSmallBits;

// The half register.  Every state of the circuit is symmetric under flipping all qubits (the
// uniform start is, the cost is, the mixer commutes with the flip), so psi(z) = psi(~z) and only
// the 2^m amplitudes, m = n - 1, with qubit n-1 at 0 are kept: half the memory, traffic and
// arithmetic of the full register, each sum over it counting twice.  RX on a qubit below n-1
// pairs z with z ^ bit; RX on qubit n-1 pairs z with its m-bit complement.
// RX(2b) = c - i s X is applied as (1 - i t X), t = s / c, two FMAs per amplitude; where |s| > |c|
// the factor -iX is pulled out first (s + i c X; X on every qubit is 1 on symmetric states and the
// phase cancels between psi and phi), so |t| <= 1.  The left-out scales c^n join the next phase table.
//
// What bounds it: shared-memory traffic of the layout changes (about 1.4x the FP64 time) and,
// above 12 half-register bits, HBM streaming.  A thread holds 8 amplitudes of psi and of phi in
// registers (512 threads x 128 registers), so three qubits are mixed per shared-memory round
// trip; 16 amplitudes a thread would save a round trip in four but leave 8 warps an SM.  One pass over the
// register finishes one layer's mixer on its qubits, applies the next phase and starts the next
// mixer on the same qubits: 2p + 1 passes for energy and gradient of p layers.
// 1024 instances of 10..20 qubits, p 1..4, with gradients: 14.0 ms; one full-register shared-memory
// pass per qubit and separate passes for phases and overlaps took 89.8 ms.  The busiest SM runs its
// shared-memory pipe at 67 %.
struct QaoaInst {
    int32_t n, p, n_edges, edge_off;
    int32_t param_off, layers;   // layers: adjacency bit planes (1 unless an edge repeats)
    int64_t state_off;       // psi at pool + state_off, phi right after it; -1: the CTA's own slot
};

__device__ __forceinline__ double2 cmul2(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// block-wide sum of two doubles; every thread gets the result
__device__ __forceinline__ double2 qblock_sum(double2 v, double2* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double2 t = make_double2(0, 0);
    for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) {
        t.x += red[w].x;
        t.y += red[w].y;
    }
    __syncthreads();
    return t;
}

// A mixer angle as (1 - i t X) times a scale.  The scale is taken from the rounded t, 1 / (1 + t^2) for
// both directions of one gate, and not from the cosine: undoing a mixer then multiplies by exactly 1
// to the precision of the pair (s2, s2l), and no error builds up over the n p gates.
struct Mix {
    double t, s2, s2l;      // scale^2 and its rounding error
    double scn;             // scale^n
};
// scale^(2 k) with the rounding error of the running product beside it
struct Power {
    double hi = 1.0, lo = 0.0;
    __device__ __forceinline__ void times(const Mix& m) {
        const double p = hi * m.s2;
        lo = fma(lo, m.s2, fma(hi, m.s2l, fma(hi, m.s2, -p)));
        hi = p;
    }
    __device__ __forceinline__ double value() const { return hi + lo; }
};
__device__ __forceinline__ Mix mix_of(double beta, int n) {
    double sn, cs;
    sincos(beta, &sn, &cs);
    const bool turn = fabs(sn) > fabs(cs);
    Mix m;
    m.t = turn ? -cs / sn : sn / cs;
    const double q = m.t * m.t, one = 1.0 + q;
    const double rest = (1.0 - one) + q + fma(m.t, m.t, -q);
    m.s2 = 1.0 / one;
    m.s2l = m.s2 * (fma(-m.s2, one, 1.0) - m.s2 * rest);
    Power s;
    for (int k = 0; k < n; ++k) s.times(m);
    m.scn = sqrt(s.value());
    return m;
}

// ---------------------------------------------------------------- 8 amplitudes in registers
// A tile of 2^TB amplitudes belongs to 2^(TB-3) threads.  In the layout with shift `sh` a thread's
// slot bits are the tile's index bits sh..sh+2 and its other index bits are the thread number's.
// swz spreads 16-byte accesses: index bits fold three at a time into the 128-byte bank line, so the
// eight lanes of a shared-memory phase hit eight bank groups in every layout.
__device__ __forceinline__ uint32_t swz(uint32_t i) { return i ^ (((i >> 3) ^ (i >> 6) ^ (i >> 9)) & 7u); }
__device__ __forceinline__ uint32_t base_of(uint32_t t, int sh) {
    return ((t >> sh) << (sh + 3)) | (t & ((1u << sh) - 1u));
}
__device__ __forceinline__ void put8(double2* buf, uint32_t t, int sh, const double2 (&v)[8]) {
    const uint32_t b = swz(base_of(t, sh));
#pragma unroll
    for (int s = 0; s < 8; ++s) buf[b ^ swz(static_cast<uint32_t>(s) << sh)] = v[s];
}
__device__ __forceinline__ void get8(const double2* buf, uint32_t t, int sh, double2 (&v)[8]) {
    const uint32_t b = swz(base_of(t, sh));
#pragma unroll
    for (int s = 0; s < 8; ++s) v[s] = buf[b ^ swz(static_cast<uint32_t>(s) << sh)];
}

// (1 - i t X) on slot bit k
__device__ __forceinline__ void mix_slot(double2 (&v)[8], int k, double t) {
#pragma unroll
    for (int s = 0; s < 8; ++s)
        if (!(s & (1 << k))) {
            const double2 a = v[s], b = v[s | (1 << k)];
            v[s] = make_double2(fma(t, b.y, a.x), fma(-t, b.x, a.y));
            v[s | (1 << k)] = make_double2(fma(t, a.y, b.x), fma(-t, a.x, b.y));
        }
}
// Im sum over pairs of slot bit k of conj(f0) v1 + conj(f1) v0
__device__ __forceinline__ double overlap_slot(const double2 (&v)[8], const double2 (&f)[8], int k, double acc) {
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const double2 p = v[s ^ (1 << k)];
        acc = fma(f[s].x, p.y, acc);
        acc = fma(-f[s].y, p.x, acc);
    }
    return acc;
}

// Cut sizes of the 8 slot combinations of one thread: z0 (slot bits 0) and the
// qubits q[0..2] the slot bits stand for.  nb: adjacency bit planes, nb[k * 32 + u].
__device__ __forceinline__ void cuts8(uint32_t z0, const int (&q)[3], const uint32_t* nb, int planes, int n, int (&c)[8]) {
    int c0 = 0, d[3] = {0, 0, 0}, j01 = 0, j02 = 0, j12 = 0;
    for (int k = 0; k < planes; ++k) {
        const uint32_t* N = nb + 32 * k;
        int ck = 0;
        for (int u = 0; u < n; ++u) ck += ((z0 >> u) & 1u) ? __popc(~z0 & N[u]) : 0;
        c0 += ck << k;
#pragma unroll
        for (int b = 0; b < 3; ++b) d[b] += (__popc(N[q[b]]) - 2 * __popc(z0 & N[q[b]])) << k;
        j01 += static_cast<int>((N[q[0]] >> q[1]) & 1u) << k;
        j02 += static_cast<int>((N[q[0]] >> q[2]) & 1u) << k;
        j12 += static_cast<int>((N[q[1]] >> q[2]) & 1u) << k;
    }
    c[0] = c0;
    c[1] = c0 + d[0];
    c[2] = c0 + d[1];
    c[3] = c[1] + d[1] - 2 * j01;
    c[4] = c0 + d[2];
    c[5] = c[1] + d[2] - 2 * j02;
    c[6] = c[2] + d[2] - 2 * j12;
    c[7] = c[3] + d[2] - 2 * (j02 + j12);
}

// What one pass does around its phase: mixers undone or applied on the way to it and after it.
struct PassWork {
    bool load, phase, up;                // load: from the pool, and a mixer before the phase; up: a mixer after it
    Mix md, mu;
    int k_down;                          // gates of the down mixer undone in earlier passes
    double amp0, fold;                   // load == false: the start amplitude; turn: the scale of psi, squared
};

// Accumulators of a pass, per thread.
// kForward: psi alone.  kTurn: the last forward pass, <C> and phi = C psi in place of a phase, then
// the first mixer undone on both.  kReverse: psi and phi.
enum PassMode { kForward, kTurn, kReverse };
struct PassSums {
    double e, g_down, g_up, gg;
};

// One pass over the register by groups of 2^(TB-3) threads, one tile each at a time.
// Set A: the tile is the low TB-1 index bits of a block of amplitudes and of the block of their
// complements (top tile bit), so its TB bits carry the mixers of qubits 0..TB-2 and of qubit n-1.
// Set B: the tile is the high bits TB-1..m-1 (local bits L..TB-1) and the low L bits, L = 2 TB - 1 - m.
template <int TB, PassMode MODE>
__device__ __noinline__ void qaoa_pass(bool set_a, const PassWork& w, int n, int E, const uint32_t* nb, int planes, const double2* s_ph,
                          double2* psi, double2* phi, double2* bufs, PassSums& acc) {
    constexpr bool two = MODE == kReverse, undo = MODE != kForward;
    constexpr uint32_t kGroup = 1u << (TB - 3);
    constexpr int kShift[4] = {0, 3, 6, TB - 3};
    const int m = n - 1;
    const uint32_t full = (1u << m) - 1u;
    const uint32_t group = threadIdx.x / kGroup, t = threadIdx.x % kGroup;
    const uint32_t n_groups = kQThreads / kGroup;
    double2* bv = bufs + static_cast<size_t>(group) * 2 * (1u << TB);
    double2* bf = bv + (1u << TB);
    const int L = set_a ? 0 : 2 * TB - 1 - m;    // local bits below L carry no mixer
    const int gmin = set_a ? 0 : (L >= 9 ? 3 : L / 3);
    const uint32_t n_tiles = 1u << (m - TB);
    auto zof = [&](uint32_t tile, uint32_t l) -> uint32_t {
        if (set_a) {
            const uint32_t z = (tile << (TB - 1)) | (l & ((1u << (TB - 1)) - 1u));
            return (l >> (TB - 1)) ? z ^ full : z;
        }
        return (l & ((1u << L) - 1u)) | (tile << L) | ((l >> L) << (TB - 1));
    };
    auto bar = [&] { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(kGroup) : "memory"); };
    // slot bit k of layout g carries a mixer of this pass; the others mix with t = 0 (a branch around
    // a mixer makes the compiler spill psi and phi)
    auto carries = [&](int g, int k) { return kShift[g] + k >= L && (g < 3 || kShift[3] + k >= 9); };
    for (uint32_t tile = group; tile < n_tiles; tile += n_groups) {
        double2 v[8], f[8];
        bar();   // the previous tile's last reads of the buffers are done
        if (MODE != kForward || w.load) {
            const uint32_t b = base_of(t, kShift[3]);
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const uint32_t z = zof(tile, b | (static_cast<uint32_t>(s) << kShift[3]));
                v[s] = *QSV_DBG(psi + z);
                f[s] = two ? *QSV_DBG(phi + z) : make_double2(0.0, 0.0);
            }
        } else {
#pragma unroll
            for (int s = 0; s < 8; ++s) v[s] = make_double2(w.amp0, 0.0);
        }
        // down: layouts 3 .. gmin (a thread rewrites only the slots it read last, so one barrier
        // separates a layout's writes from the next layout's reads)
        Power scale;
        if (MODE != kForward || w.load) {
            for (int k = 0; k < w.k_down; ++k) scale.times(w.md);
#pragma unroll
            for (int g = 3; g >= 0; --g)
                if (g >= gmin) {
                    if (two) {
                        double o = 0.0;
#pragma unroll
                        for (int k = 0; k < 3; ++k)
                            if (carries(g, k)) o = overlap_slot(v, f, k, o);
                        acc.g_down = fma(scale.value(), o, acc.g_down);
                    }
                    const double tt = two ? -w.md.t : w.md.t;
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        if (g < 3 || kShift[3] + k >= 9) {
                            const double tk = carries(g, k) ? tt : 0.0;
                            mix_slot(v, k, tk);
                            if (two) mix_slot(f, k, tk);
                            if (carries(g, k)) scale.times(w.md);
                        }
                    if (g > gmin) {
                        put8(bv, t, kShift[g], v);
                        if (two) put8(bf, t, kShift[g], f);
                        bar();
                        get8(bv, t, kShift[g ? g - 1 : 0], v);
                        if (two) get8(bf, t, kShift[g ? g - 1 : 0], f);
                    }
                }
        }
        // the diagonal step, in layout gmin
        int c[8];
        {
            const int sh = gmin == 3 ? kShift[3] : 3 * gmin;
            int q[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) q[k] = set_a || sh + k < L ? sh + k : sh + k - L + TB - 1;
            // the complemented half of a set A tile is cut as its complement (qubit n-1 at 1): slot bits stay 0
            const uint32_t l = base_of(t, sh);
            const uint32_t z0 = set_a ? (tile << (TB - 1)) | (l & ((1u << (TB - 1)) - 1u)) | ((l >> (TB - 1)) << m)
                                      : zof(tile, l);
            cuts8(z0, q, nb, planes, n, c);
        }
        if (MODE == kTurn) {
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const double cv = w.fold * static_cast<double>(c[s]);
                f[s] = make_double2(cv * v[s].x, cv * v[s].y);
                acc.e = fma(f[s].x, v[s].x, acc.e);
                acc.e = fma(f[s].y, v[s].y, acc.e);
            }
        } else if (two) {
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const double o = f[s].x * v[s].y - f[s].y * v[s].x;
                acc.gg = fma(scale.value() * static_cast<double>(E - 2 * c[s]), o, acc.gg);
            }
        }
        if (MODE != kTurn && w.phase) {
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const double2 ph = s_ph[c[s]];
                v[s] = cmul2(ph, v[s]);
                if (two) f[s] = cmul2(ph, f[s]);
            }
        }
        if (!w.up) continue;
        const double tt = undo ? -w.mu.t : w.mu.t;
        scale = Power();
#pragma unroll
        for (int g = 0; g < 4; ++g)
            if (g >= gmin) {
                if (undo) {
                    double o = 0.0;
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        if (carries(g, k)) o = overlap_slot(v, f, k, o);
                    acc.g_up = fma(scale.value(), o, acc.g_up);
                }
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    if (g < 3 || kShift[3] + k >= 9) {
                        const double tk = carries(g, k) ? tt : 0.0;
                        mix_slot(v, k, tk);
                        if (undo) mix_slot(f, k, tk);
                        if (carries(g, k)) scale.times(w.mu);
                    }
                if (g < 3) {
                    put8(bv, t, kShift[g], v);
                    if (undo) put8(bf, t, kShift[g], f);
                    bar();
                    get8(bv, t, kShift[g < 3 ? g + 1 : 3], v);
                    if (undo) get8(bf, t, kShift[g < 3 ? g + 1 : 3], f);
                }
            }
        {
            const uint32_t b = base_of(t, kShift[3]);
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const uint32_t z = zof(tile, b | (static_cast<uint32_t>(s) << kShift[3]));
                *QSV_DBG(psi + z) = v[s];
                if (undo) *QSV_DBG(phi + z) = f[s];
            }
        }
    }
}

// exp(-i gamma (E - 2 c)) * scale for c = 0..E (conjugated when undoing)
__device__ __forceinline__ void phase_table(double2* s_ph, int E, double gamma, double scale, bool undo) {
    for (int c = threadIdx.x; c <= E; c += blockDim.x) {
        double sn, cs;
        sincos(-gamma * static_cast<double>(E - 2 * c), &sn, &cs);
        s_ph[c] = make_double2(scale * cs, undo ? -scale * sn : scale * sn);
    }
    __syncthreads();
}

// An instance whose half register is streamed through tiles (m > 12).
template <int TB>
__device__ void qaoa_stream(const QaoaInst& I, const double* prm, const Mix* mix, double* grd, double* energy, const uint32_t* nb,
                            double2* s_ph, double2* psi, double2* bufs, double2* red, bool with_grad) {
    const int n = I.n, p = I.p, E = I.n_edges, m = n - 1;
    double2* phi = psi + (1ull << m);
    const int size_a = TB, size_b = m - TB + 1;
    PassSums acc{0, 0, 0, 0};
    Mix prev{};
    for (int k = 0; k <= p; ++k) {      // forward: finish mixer k-1, phase k, start mixer k
        PassWork w{};
        w.load = k > 0;
        w.md = prev;
        w.phase = k < p;
        w.up = k < p || with_grad;
        w.amp0 = 1.0;
        if (k < p) {
            w.mu = mix[k];
            phase_table(s_ph, E, *QSV_DBG(prm + 2 * k), k == 0 ? exp2(-0.5 * n) : prev.scn, false);
            prev = w.mu;
            qaoa_pass<TB, kForward>((k & 1) == 0, w, n, E, nb, I.layers, s_ph, psi, phi, bufs, acc);
        } else {
            w.mu = prev;
            w.fold = prev.scn * prev.scn;
            qaoa_pass<TB, kTurn>((k & 1) == 0, w, n, E, nb, I.layers, s_ph, psi, phi, bufs, acc);
        }
        __syncthreads();
    }
    const double2 en = qblock_sum(make_double2(acc.e, 0.0), red);
    if (threadIdx.x == 0) *QSV_DBG(energy) = 2.0 * en.x;
    if (!with_grad) return;
    double gb = acc.g_up;
    for (int r = p - 1; r >= 0; --r) {   // reverse: finish undoing mixer r, undo phase r, start undoing mixer r-1
        PassWork w{};
        const bool set_a = (r & 1) == 0;
        w.load = true;
        w.md = prev;
        w.k_down = set_a ? size_b : size_a;
        w.phase = w.up = r > 0;
        if (r > 0) {
            phase_table(s_ph, E, *QSV_DBG(prm + 2 * r), prev.scn, true);
            w.mu = mix[r - 1];
        }
        acc = PassSums{0, gb, 0, 0};
        qaoa_pass<TB, kReverse>(set_a, w, n, E, nb, I.layers, s_ph, psi, phi, bufs, acc);
        const double2 g = qblock_sum(make_double2(acc.g_down, acc.gg), red);
        if (threadIdx.x == 0) {
            *QSV_DBG(grd + 2 * r) = 4.0 * g.y;
            *QSV_DBG(grd + (2 * r + 1)) = 4.0 * g.x;
        }
        gb = acc.g_up;
        prev = w.mu;
    }
}

// An instance whose half register stays on chip (m <= 12): registers between layout changes, psi
// in `A` and phi in `B` at them.  Index bits at and above m hold zeros.
__device__ __noinline__ void qaoa_small(const QaoaInst& I, const double* prm, const Mix* mix, double* grd, double* energy, const uint32_t* nb, double2* s_ph,
                           double2* A, double2* B, double2* red, bool with_grad) {
    const int n = I.n, p = I.p, E = I.n_edges, m = n - 1;
    const uint32_t M = 1u << m, full = M - 1u, t = threadIdx.x;
    const int top = (m + 2) / 3 - 1;     // layouts 0..top, slot bits 3 g .. 3 g + 2
    double2 v[8], f[8];
    auto active = [&](int g) { return base_of(t, 3 * g) < M; };
    auto cuts = [&](int g, int (&c)[8]) {
        const int q[3] = {3 * g, 3 * g + 1, 3 * g + 2};
        cuts8(base_of(t, 3 * g), q, nb, I.layers, n, c);
    };
    // the places that layouts 0..top reach
    for (uint32_t i = t; i < (1u << (3 * (top + 1))); i += blockDim.x) A[i] = B[i] = make_double2(0.0, 0.0);
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        v[s] = make_double2(base_of(t, 0) + s < M ? 1.0 : 0.0, 0.0);
        f[s] = make_double2(0.0, 0.0);
    }
    __syncthreads();
    int g = 0;                            // the layout the registers are in
    // mixes every index bit, from the layout the registers are in to the other end, then the
    // pairs (z, ~z) of qubit n-1 in shared memory; `both`: undo on psi and phi, adding overlaps
    auto mixer = [&](const Mix& mx, auto both, double& over) {
        constexpr bool two = decltype(both)::value;
        const double tt = two ? -mx.t : mx.t;
        const int dir = g == 0 ? 1 : -1, end = g == 0 ? top : 0;
        Power scale;
        for (;;) {
            if (active(g)) {
                double o = 0.0;
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    if (two && 3 * g + k < m) o = overlap_slot(v, f, k, o);
                over = fma(scale.value(), o, over);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const double tk = 3 * g + k < m ? tt : 0.0;
                    mix_slot(v, k, tk);
                    if (two) mix_slot(f, k, tk);
                }
            }
            for (int k = 0; k < 3; ++k)
                if (3 * g + k < m) scale.times(mx);
            if (active(g)) {
                put8(A, t, 3 * g, v);
                if (two) put8(B, t, 3 * g, f);
            }
            __syncthreads();
            if (g == end) break;
            g += dir;
            if (active(g)) {
                get8(A, t, 3 * g, v);
                if (two) get8(B, t, 3 * g, f);
            }
        }
        double o = 0.0;
        for (uint32_t i = t; i < (M >> 1); i += blockDim.x) {
            const uint32_t i0 = swz(i), i1 = swz(i ^ full);
            const double2 a = A[i0], b = A[i1];
            A[i0] = make_double2(fma(tt, b.y, a.x), fma(-tt, b.x, a.y));
            A[i1] = make_double2(fma(tt, a.y, b.x), fma(-tt, a.x, b.y));
            if (two) {
                const double2 fa = B[i0], fb = B[i1];
                o += fa.x * b.y - fa.y * b.x + fb.x * a.y - fb.y * a.x;
                B[i0] = make_double2(fma(tt, fb.y, fa.x), fma(-tt, fb.x, fa.y));
                B[i1] = make_double2(fma(tt, fa.y, fb.x), fma(-tt, fa.x, fb.y));
            }
        }
        over = fma(scale.value(), o, over);
        __syncthreads();
        if (active(g)) {
            get8(A, t, 3 * g, v);
            if (two) get8(B, t, 3 * g, f);
        }
        // the next writes go to the slots just read: no barrier needed before them
    };
    Mix prev{};
    double none = 0.0;
    int c[8];
    for (int r = 0; r < p; ++r) {
        phase_table(s_ph, E, *QSV_DBG(prm + 2 * r), r == 0 ? exp2(-0.5 * n) : prev.scn, false);
        if (active(g)) {
            cuts(g, c);
#pragma unroll
            for (int s = 0; s < 8; ++s) v[s] = cmul2(s_ph[c[s]], v[s]);
        }
        prev = mix[r];
        mixer(prev, std::false_type{}, none);
    }
    double e = 0.0;
    if (active(g)) {
        cuts(g, c);
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            const double cv = prev.scn * prev.scn * static_cast<double>(c[s]);
            f[s] = make_double2(cv * v[s].x, cv * v[s].y);
            e = fma(f[s].x, v[s].x, e);
            e = fma(f[s].y, v[s].y, e);
        }
    }
    const double2 en = qblock_sum(make_double2(e, 0.0), red);
    if (threadIdx.x == 0) *QSV_DBG(energy) = 2.0 * en.x;
    if (!with_grad) return;
    for (int r = p - 1; r >= 0; --r) {
        double gb = 0.0, gg = 0.0;
        mixer(prev, std::true_type{}, gb);
        const double undone = prev.scn * prev.scn;     // psi and phi each lack scale^n
        phase_table(s_ph, E, *QSV_DBG(prm + 2 * r), prev.scn, true);
        if (active(g)) {
            cuts(g, c);
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const double o = f[s].x * v[s].y - f[s].y * v[s].x;
                gg = fma(undone * static_cast<double>(E - 2 * c[s]), o, gg);
                const double2 ph = s_ph[c[s]];
                v[s] = cmul2(ph, v[s]);
                f[s] = cmul2(ph, f[s]);
            }
        }
        const double2 sum = qblock_sum(make_double2(gb, gg), red);
        if (threadIdx.x == 0) {
            *QSV_DBG(grd + 2 * r) = 4.0 * sum.y;
            *QSV_DBG(grd + (2 * r + 1)) = 4.0 * sum.x;
        }
        if (r > 0) prev = mix[r - 1];
    }
}

// Tiles of 2^11 amplitudes, two groups of 256 threads that run apart (one loads while the other
// computes), up to 22 qubits; the high bits of 23 and 24 qubits need tiles of 2^12.
__global__ void __launch_bounds__(kQThreads, 1)
    k_qaoa_batch(const QaoaInst* __restrict__ inst, const int32_t* __restrict__ order, int n_inst,
                 const int32_t* __restrict__ edges, const double* __restrict__ params, double2* __restrict__ pool,
                 int64_t cta_slot, int* __restrict__ counter, double* __restrict__ energy, double* __restrict__ grads,
                 int with_grad) {
    extern __shared__ __align__(16) unsigned char qsm[];
    double2* bufs = reinterpret_cast<double2*>(qsm);
    __shared__ int s_w;
    __shared__ uint32_t s_nb[32 * kQMaxLayers];
    __shared__ int s_ed[2 * kQMaxEdges];
    __shared__ double2 s_ph[kQMaxEdges + 1];
    __shared__ Mix s_mix[kQMaxDepth];
    __shared__ double2 red[kQThreads / 32];
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_w = atomicAdd(QSV_DBG(counter), 1);
        __syncthreads();
        const int w = s_w;
        if (w >= n_inst) break;
        const int id = *QSV_DBG(order + w);
        const QaoaInst I = *QSV_DBG(inst + id);
        for (int u = threadIdx.x; u < 32 * kQMaxLayers; u += blockDim.x) s_nb[u] = 0;
        for (int e = threadIdx.x; e < 2 * I.n_edges; e += blockDim.x) s_ed[e] = *QSV_DBG(edges + (2 * I.edge_off + e));
        __syncthreads();
        if (threadIdx.x < 32 && I.layers == 1) {   // no edge twice: bits in any order
            for (int e = threadIdx.x; e < I.n_edges; e += 32) {
                const int a = s_ed[2 * e], b = s_ed[2 * e + 1];
                atomicXor(&s_nb[a], 1u << b);
                atomicXor(&s_nb[b], 1u << a);
            }
        } else if (threadIdx.x == 0) {   // adjacency with multiplicity: a ripple carry through the bit planes
            for (int e = 0; e < I.n_edges; ++e) {
                const int a = s_ed[2 * e], b = s_ed[2 * e + 1];
                for (int k = 0; k < kQMaxLayers; ++k) {
                    const bool carry = (s_nb[32 * k + a] >> b) & 1u;
                    s_nb[32 * k + a] ^= 1u << b;
                    s_nb[32 * k + b] ^= 1u << a;
                    if (!carry) break;
                }
            }
        }
        const double* prm = params + I.param_off;
        // Every layer's mixer angle, beside the first warp's adjacency: formed layer by layer they were half
        // a microsecond of chain each, felt where the register is narrow (8 qubits, p = 4: 74 -> 68 us alone,
        // 1000 of them 830 -> 795 us).
        if (threadIdx.x >= 32)
            for (int r = threadIdx.x - 32; r < I.p; r += blockDim.x - 32) s_mix[r] = mix_of(*QSV_DBG(prm + (2 * r + 1)), I.n);
        __syncthreads();
        double* grd = grads + I.param_off;
        double* en = energy + id;
        double2* psi = pool + (I.state_off >= 0 ? I.state_off : static_cast<int64_t>(blockIdx.x) * cta_slot);
        if (I.n - 1 <= kQSmallBits) qaoa_small(I, prm, s_mix, grd, en, s_nb, s_ph, bufs, bufs + kQTile, red, with_grad != 0);
        else if (I.n - 1 <= 21) qaoa_stream<11>(I, prm, s_mix, grd, en, s_nb, s_ph, psi, bufs, red, with_grad != 0);
        else qaoa_stream<12>(I, prm, s_mix, grd, en, s_nb, s_ph, psi, bufs, red, with_grad != 0);
    }
}

struct QaoaBatch {
    int device = 0;
    int n_inst = 0;
    size_t n_params = 0;
    cudaStream_t stream = nullptr;
    void* dev = nullptr;          // instances, order, edges, params, energy, grads, counter
    double2* pool = nullptr;
    int64_t cta_slot = 0;         // amplitudes per CTA in the pool where instances share slots
    QaoaInst* d_inst = nullptr;
    int32_t* d_order = nullptr;
    int32_t* d_edges = nullptr;
    double* d_params = nullptr;
    double* d_energy = nullptr;
    double* d_grads = nullptr;
    int* d_counter = nullptr;
    double* h_params = nullptr;   // pinned staging
    double* h_out = nullptr;      // pinned: energies then grads
    cudaGraph_t graph[2] = {nullptr, nullptr};
    cudaGraphExec_t exec[2] = {nullptr, nullptr};
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    int grid = 0;
};

void capture(QaoaBatch& q, int with_grad) {
    check_cuda(cudaStreamBeginCapture(q.stream, cudaStreamCaptureModeThreadLocal), "capture begin");
    cudaMemcpyAsync(q.d_params, q.h_params, q.n_params * sizeof(double), cudaMemcpyHostToDevice, q.stream);
    cudaMemsetAsync(q.d_counter, 0, sizeof(int), q.stream);
    const size_t smem = 2 * kQTile * sizeof(double2);
    k_qaoa_batch<<<q.grid, kQThreads, smem, q.stream>>>(q.d_inst, q.d_order, q.n_inst, q.d_edges, q.d_params, q.pool,
                                                         q.cta_slot, q.d_counter, q.d_energy, q.d_grads, with_grad);
    cudaMemcpyAsync(q.h_out, q.d_energy, q.n_inst * sizeof(double), cudaMemcpyDeviceToHost, q.stream);
    if (with_grad)
        cudaMemcpyAsync(q.h_out + q.n_inst, q.d_grads, q.n_params * sizeof(double), cudaMemcpyDeviceToHost, q.stream);
    check_cuda(cudaStreamEndCapture(q.stream, &q.graph[with_grad]), "capture end");
    check_cuda(cudaGraphInstantiate(&q.exec[with_grad], q.graph[with_grad], 0), "graph instantiate");
}

void release(QaoaBatch* q) {
    if (!q) return;
    cudaSetDevice(q->device);
    if (q->stream) cudaStreamSynchronize(q->stream);
    for (int i = 0; i < 2; ++i) {
        if (q->exec[i]) cudaGraphExecDestroy(q->exec[i]);
        if (q->graph[i]) cudaGraphDestroy(q->graph[i]);
    }
    if (q->dev) dev_free(q->dev);
    if (q->pool) dev_free(q->pool);
    if (q->h_params) cudaFreeHost(q->h_params);
    if (q->h_out) cudaFreeHost(q->h_out);
    if (q->e0) cudaEventDestroy(q->e0);
    if (q->e1) cudaEventDestroy(q->e1);
    if (q->stream) cudaStreamDestroy(q->stream);
    delete q;
}

}  // namespace

// ---------------------------------------------------------------- host entry points

void* qaoa_create(int device, int n_inst, const int32_t* n_qubits, const int32_t* depth, const int32_t* edge_ptr,
                  const int32_t* edges) {
    if (n_inst <= 0) throw std::invalid_argument("no instances");
    if (!n_qubits || !depth || !edge_ptr || !edges) throw std::invalid_argument("null instance arrays");
    check_cuda(cudaSetDevice(device), "cudaSetDevice");
    auto* q = new QaoaBatch();
    q->device = device;
    q->n_inst = n_inst;
    try {
        std::vector<QaoaInst> inst(n_inst);
        std::vector<double> cost(n_inst);
        int64_t pool_amps = 0, widest = 0;
        size_t n_params = 0;
        for (int i = 0; i < n_inst; ++i) {
            const int n = n_qubits[i], p = depth[i], E = edge_ptr[i + 1] - edge_ptr[i];
            if (n < 2 || n > kQMaxQubits) throw std::invalid_argument("QAOA instance width must be in [2, 24]");
            if (p < 1 || p > kQMaxDepth) throw std::invalid_argument("QAOA depth must be in [1, 64]");
            if (E < 0 || E > kQMaxEdges) throw std::invalid_argument("QAOA instance has too many edges");
            for (int e = edge_ptr[i]; e < edge_ptr[i + 1]; ++e) {
                const int u = edges[2 * e], v = edges[2 * e + 1];
                if (u < 0 || v < 0 || u >= n || v >= n || u == v)
                    throw std::invalid_argument("QAOA edge outside its instance or a self-loop");
            }
            std::map<std::pair<int, int>, int> times;
            int most = 1;
            for (int e = edge_ptr[i]; e < edge_ptr[i + 1]; ++e)
                most = std::max(most, ++times[std::minmax(edges[2 * e], edges[2 * e + 1])]);
            int planes = 0;
            while (most >> planes) ++planes;
            inst[i] = QaoaInst{n, p, E, edge_ptr[i], static_cast<int32_t>(n_params), planes, -1};
            if (n - 1 > kQSmallBits) {
                inst[i].state_off = pool_amps;
                pool_amps += 2ll << (n - 1);      // psi and phi of the half register
                widest = std::max<int64_t>(widest, 2ll << (n - 1));
            }
            n_params += 2 * static_cast<size_t>(p);
            cost[i] = std::ldexp(1.0, n) * (4.0 * p + 1.0);
        }
        q->n_params = n_params;
        int sms = 0;
        check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "sm count");
        q->grid = std::min(sms, n_inst);
        // the pool holds every instance's registers, or one slot of the widest per CTA where that is less
        if (widest * q->grid < pool_amps) {
            q->cta_slot = widest;
            pool_amps = widest * q->grid;
            for (QaoaInst& in : inst) in.state_off = -1;
        }
        std::vector<int32_t> order(n_inst);
        std::iota(order.begin(), order.end(), 0);
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cost[a] > cost[b]; });
        const size_t n_edges = static_cast<size_t>(edge_ptr[n_inst]);
        auto al = [](size_t b) { return (b + 255) & ~size_t{255}; };
        const size_t b_inst = al(n_inst * sizeof(QaoaInst)), b_order = al(n_inst * 4), b_edges = al(2 * n_edges * 4 + 4);
        const size_t b_params = al(n_params * 8), b_energy = al(n_inst * 8), b_grads = al(n_params * 8), b_cnt = 256;
        const size_t total = b_inst + b_order + b_edges + b_params + b_energy + b_grads + b_cnt;
        check_cuda(dev_malloc(&q->dev, total), "QAOA descriptors");
        uint8_t* d = static_cast<uint8_t*>(q->dev);
        q->d_inst = reinterpret_cast<QaoaInst*>(d);
        q->d_order = reinterpret_cast<int32_t*>(d + b_inst);
        q->d_edges = reinterpret_cast<int32_t*>(d + b_inst + b_order);
        q->d_params = reinterpret_cast<double*>(d + b_inst + b_order + b_edges);
        q->d_energy = reinterpret_cast<double*>(d + b_inst + b_order + b_edges + b_params);
        q->d_grads = reinterpret_cast<double*>(d + b_inst + b_order + b_edges + b_params + b_energy);
        q->d_counter = reinterpret_cast<int*>(d + b_inst + b_order + b_edges + b_params + b_energy + b_grads);
        if (pool_amps > 0) check_cuda(dev_malloc(&q->pool, static_cast<size_t>(pool_amps) * sizeof(double2)), "QAOA state pool");
        check_cuda(cudaMallocHost(reinterpret_cast<void**>(&q->h_params), std::max<size_t>(n_params, 1) * 8), "pinned params");
        check_cuda(cudaMallocHost(reinterpret_cast<void**>(&q->h_out), (n_inst + n_params) * 8), "pinned results");
        check_cuda(cudaStreamCreateWithFlags(&q->stream, cudaStreamNonBlocking), "stream");
        check_cuda(cudaEventCreate(&q->e0), "event");
        check_cuda(cudaEventCreate(&q->e1), "event");
        check_cuda(cudaMemcpy(q->d_inst, inst.data(), n_inst * sizeof(QaoaInst), cudaMemcpyHostToDevice), "upload");
        check_cuda(cudaMemcpy(q->d_order, order.data(), n_inst * 4, cudaMemcpyHostToDevice), "upload");
        if (n_edges) check_cuda(cudaMemcpy(q->d_edges, edges, 2 * n_edges * 4, cudaMemcpyHostToDevice), "upload");
        const size_t smem = 2 * kQTile * sizeof(double2);
        check_cuda(cudaFuncSetAttribute(k_qaoa_batch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(smem)), "smem attribute");
        capture(*q, 0);
        capture(*q, 1);
    } catch (...) {
        release(q);
        throw;
    }
    return q;
}

void qaoa_run(void* h, const double* params, int with_grad, double* energies, double* grads, double* ms) {
    auto* q = static_cast<QaoaBatch*>(h);
    if (!q) throw std::invalid_argument("null QAOA batch");
    if (!params || !energies || (with_grad && !grads)) throw std::invalid_argument("null argument");
    check_cuda(cudaSetDevice(q->device), "cudaSetDevice");
    const int g = with_grad ? 1 : 0;
    std::memcpy(q->h_params, params, q->n_params * 8);
    check_cuda(cudaEventRecord(q->e0, q->stream), "event");
    check_cuda(cudaGraphLaunch(q->exec[g], q->stream), "graph launch");
    check_cuda(cudaEventRecord(q->e1, q->stream), "event");
    check_cuda(cudaStreamSynchronize(q->stream), "QAOA batch");
    std::memcpy(energies, q->h_out, q->n_inst * 8);
    if (with_grad) std::memcpy(grads, q->h_out + q->n_inst, q->n_params * 8);
    if (ms) {
        float f = 0;
        check_cuda(cudaEventElapsedTime(&f, q->e0, q->e1), "elapsed");
        *ms = f;
    }
}

void qaoa_destroy(void* h) { release(static_cast<QaoaBatch*>(h)); }

}  // namespace qsv
