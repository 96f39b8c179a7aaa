// kern_traj_fused.cu — trajectories of small registers with each shot held in one CTA's shared
// memory from its first command to its final sample.
//
// For registers of up to 64 KiB (complex128 n <= 12, complex64 n <= 13) the batched executor's
// passes over the wide register in HBM are pure overhead: a shot fits on chip.  Here every CTA (or,
// for the narrowest, every warp) runs one shot: it loads the prefix state into shared memory, seeds
// the shot's MT19937 engine
// (std::mt19937(seed + shot)) in shared memory, and interprets the trajectory plan — fused
// gates, guarded gates, measurements, branches, noise channels — with block-wide passes over
// shared memory, then draws the final sample and writes the outcome and the classical register.
// The per-shot rules (guards, decisions, channel choices, the final CDF walk) are the batched
// executor's (traj.h), so both executors follow the reference's consumption of draws exactly.
#include <algorithm>
#include <cstring>

#include "traj.h"

namespace qsv {

namespace {

constexpr int kFsMaxBytes = 64 * 1024;   // widest register held in shared memory
// A shot per warp, eight to a block, against a shot per block (B200, feed-forward circuits of depth
// 8, 20000 shots, microseconds): 7 qubits 867 against 2160, 8 qubits 1262 against 2670, 9 qubits 2194
// against 3418, 10 qubits 5261 against 5145, and with noise on every gate 10 qubits 12996 against
// 26621 (a noise step is two reductions and a draw, all chain).  Too few shots to give every
// multiprocessor a block: 8 qubits 500 shots 268 against 242, 9 qubits 337 against 284, while 7
// qubits stay even (223 against 224).
constexpr int kFsWarpShots = 8;
constexpr int kFsWarpBytes = 2 * 1024;          // always
constexpr int kFsWarpBytesMany = 8 * 1024;      // with shots for every multiprocessor's block
constexpr int kFsWarpBytesNoise = 16 * 1024;    // the same, plans with noise
constexpr int kFsNarrowBytes = 16 * 1024;   // registers up to here: 128 threads a CTA, else 256
constexpr int kFsMaxCoef = 512;          // doubles of one step's coefficients (a 4-qubit block)
constexpr int kFsMtBytes = 4 * 624 + 16; // one MT19937 state, padded to keep the plan aligned
constexpr size_t kFsResidentMax = 104 * 1024;   // dynamic shared memory with the plan resident
constexpr size_t kFsApplyResidentMax = 200 * 1024;   // the same for the one-CTA gate sequence
// The one-CTA gate sequence takes 512 threads from 10 qubits: below, a step has fewer groups than
// that and the barrier of four warps is the cheaper one.
constexpr int kFsApplyWide = 10;

enum FsKind : uint8_t {
    FS_DENSE = 0,     // k <= 4 unitary on q[0..k) where (i & ctrl) == ctrl; matrix at coef
    FS_DIAG,          // k <= 8 diagonal on q[0..k); entries at coef
    FS_PHASE,         // i -> v i where (i & mask) == mask; v at coef
    FS_SWAP,          // swap q[0], q[1]
    FS_PROT,          // exp(-i theta/2 P): x = mask, z = zmask; (cos, sin) at coef
    FS_SCALE,         // every amplitude times v
    FS_MEASURE,       // q[0]; cbit; k = 1 for Reset
    FS_BRANCH,        // flag bit `flag` <- (cbits & mask) == zmask
    FS_PAULI_NOISE,   // channel kind k2 on q[0..k); parameters at coef
    FS_KRAUS_NOISE,   // k2 operators on q[0]; 8 doubles each at coef
    FS_ADJ,           // circuit batches: adjoint step on q[0..k) (k <= 2): slot cbit <- <phi| G |psi>, then
                      // D on both registers; G then D (2^k x 2^k each) at coef
};

struct alignas(16) FsStep {
    uint8_t kind = 0;
    uint8_t k = 0;
    uint8_t k2 = 0;
    uint8_t flag = 0;
    int32_t cbit = -1;
    uint32_t coef = 0;       // offset in the coefficient table (doubles)
    uint32_t ncoef = 0;      // doubles the step reads there (staged in shared memory)
    uint64_t fmask = 0, fwant = 0, cmask = 0, cwant = 0;   // guard
    uint64_t mask = 0, zmask = 0, ctrl = 0;
    uint64_t reserved = 0;   // keeps the size a multiple of 16 bytes
    // FS_DENSE and FS_ADJ: q[16..16+k2) are the step's qubits and controls, ascending
    uint8_t q[32] = {};
};

// The threads of one shot meet: a whole block, or one warp of a block that runs a shot per warp.
template <int NT>
__device__ __forceinline__ void fs_sync() {
    if constexpr (NT == 32) __syncwarp();
    else __syncthreads();
}

// N sums over the NT threads of a shot with one pair of barriers; red must hold N * NT / 32
// doubles.  Results valid in the shot's thread 0.
template <int NT, int N>
__device__ __forceinline__ void fs_sums(double v[N], double* red, uint32_t tid) {
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if constexpr (NT > 32) {
        if ((tid & 31) == 0)
#pragma unroll
            for (int k = 0; k < N; ++k) red[N * (tid >> 5) + k] = v[k];
        __syncthreads();
        if (tid == 0)
#pragma unroll
            for (int k = 0; k < N; ++k) {
                double t = 0.0;
                for (int w = 0; w < NT / 32; ++w) t += red[N * w + k];
                v[k] = t;
            }
        __syncthreads();   // red is free again
    }
}

template <typename T>
__device__ __forceinline__ vec2_t<T> cmul_d(double re, double im, vec2_t<T> a) {
    const double x = static_cast<double>(a.x), y = static_cast<double>(a.y);
    return mk<T>(static_cast<T>(re * x - im * y), static_cast<T>(re * y + im * x));
}

// Where amplitude i lies in shared memory: the bits above an eight-amplitude row (128 bytes, all
// banks once) are XORed into the place in the row, so that a warp whose lanes leave out a low
// qubit (the gate's own) still covers every bank.  Linear over XOR: slot(a | b) of disjoint bits
// is slot(a) ^ slot(b), one XOR per amplitude of a group.
template <typename T>
__device__ __forceinline__ uint32_t fs_slot(uint32_t i) {
    return sizeof(T) == 8 ? i ^ ((i >> 3) & 7u) : i ^ ((i >> 4) & 15u);
}

__device__ __forceinline__ uint32_t fs_insert(uint32_t g, uint32_t p) {   // a zero bit at position p
    return ((g >> p) << (p + 1)) | (g & ((1u << p) - 1u));
}

// The groups of a gate step: the gate's qubits and its controls ascending in q[16..16+k2), so
// that every index that is visited is one that the gate changes.
struct FsGroups {
    const FsStep& S;
    uint32_t p4, ctrl, npos;
    __device__ __forceinline__ FsGroups(const FsStep& s)
        : S(s), p4(*reinterpret_cast<const uint32_t*>(s.q + 16)), ctrl(static_cast<uint32_t>(s.ctrl)), npos(s.k2) {}
    template <int K>
    __device__ __forceinline__ uint32_t base(uint32_t g) const {
#pragma unroll
        for (int j = 0; j < K; ++j) g = fs_insert(g, (p4 >> (8 * j)) & 0xffu);
        for (uint32_t j = K; j < npos; ++j) g = fs_insert(g, S.q[16 + j]);
        return g | ctrl;
    }
};

template <typename T, int K>
__device__ __forceinline__ void fs_offsets(const FsStep& S, uint32_t off[1 << K]) {
    const uint32_t q4 = *reinterpret_cast<const uint32_t*>(S.q);
    off[0] = 0;
#pragma unroll
    for (int b = 0; b < K; ++b) {
        const uint32_t o = fs_slot<T>(1u << ((q4 >> (8 * b)) & 0xffu));
#pragma unroll
        for (int l = 0; l < (1 << b); ++l) off[l + (1 << b)] = off[l] ^ o;
    }
}

// G groups of 2^K amplitudes per thread, NT threads: each matrix entry is read once for all G.
// Several rows at a time: their independent FP64 chains hide the unit's latency.
template <typename T, int K, int NT, int G>
__device__ __forceinline__ void fs_rows(vec2_t<T>* a, const FsGroups& at, uint32_t groups, const uint32_t off[1 << K],
                                        const double2* __restrict__ rows, uint32_t tid) {
    constexpr int D = 1 << K;
    // all the rows of a wide block at once would spill
    constexpr int R = K == 1 ? D : K == 4 ? 2 : K == 3 || G == 1 ? 4 : 2;
    for (uint32_t g = tid; g < groups; g += G * NT) {
        uint32_t base[G];
        double xr[G][D], xi[G][D];
#pragma unroll
        for (int u = 0; u < G; ++u) {
            // past the end: the thread's first group once more (both are read before either is written)
            const uint32_t gu = u == 0 || g + u * NT < groups ? g + u * NT : g;
            base[u] = fs_slot<T>(at.template base<K>(gu));
#pragma unroll
            for (int x = 0; x < D; ++x) {
                const vec2_t<T> v = a[base[u] ^ off[x]];
                xr[u][x] = static_cast<double>(v.x);
                xi[u][x] = static_cast<double>(v.y);
            }
        }
#pragma unroll 1
        for (int y0 = 0; y0 < D; y0 += R) {
            uint32_t o0 = 0;
#pragma unroll
            for (int b = 1; b < D; b <<= 1)
                if (b >= R && (y0 & b)) o0 ^= off[b];
#pragma unroll
            for (int y = 0; y < R; ++y) {
                double re[G] = {}, im[G] = {};
#pragma unroll
                for (int x = 0; x < D; ++x) {
                    const double2 cf = rows[(y0 + y) * D + x];
#pragma unroll
                    for (int u = 0; u < G; ++u) {
                        re[u] = fma(cf.x, xr[u][x], re[u]);
                        re[u] = fma(-cf.y, xi[u][x], re[u]);
                        im[u] = fma(cf.x, xi[u][x], im[u]);
                        im[u] = fma(cf.y, xr[u][x], im[u]);
                    }
                }
#pragma unroll
                for (int u = 0; u < G; ++u)
                    a[base[u] ^ o0 ^ off[y]] = mk<T>(static_cast<T>(re[u]), static_cast<T>(im[u]));
            }
        }
    }
}

// One k-qubit unitary.  What bounds these steps is the shared memory's pipe, and most of what goes
// through it are the matrix entries, the same for all lanes: up to two qubits a thread takes two
// groups where the register has them.
template <typename T, int K, int NT>
__device__ __forceinline__ void fs_dense(vec2_t<T>* a, int n, const FsStep& S, const double* __restrict__ m,
                                         uint32_t tid) {
    uint32_t off[1 << K];
    fs_offsets<T, K>(S, off);
    const FsGroups at(S);
    const uint32_t groups = 1u << (n - static_cast<int>(at.npos));
    const double2* const rows = reinterpret_cast<const double2*>(m);
    if constexpr (K <= 2) {
        if (groups > NT) {
            fs_rows<T, K, NT, 2>(a, at, groups, off, rows, tid);
            return;
        }
    }
    fs_rows<T, K, NT, 1>(a, at, groups, off, rows, tid);
}

// The gate steps (dense, diagonal, phase, scale, swap, Pauli rotation) on the amplitudes at
// fs_slot places, by threads 0..NT of the step; false for the other kinds.
template <typename T, int NT>
__device__ __forceinline__ bool fs_gate(vec2_t<T>* a, int n, const FsStep& S, const double* c, uint32_t tid) {
    const uint32_t dim = 1u << n;
    switch (S.kind) {
        case FS_DENSE:
            switch (S.k) {
                case 1: fs_dense<T, 1, NT>(a, n, S, c, tid); break;
                case 2: fs_dense<T, 2, NT>(a, n, S, c, tid); break;
                case 3: fs_dense<T, 3, NT>(a, n, S, c, tid); break;
                default: fs_dense<T, 4, NT>(a, n, S, c, tid); break;
            }
            break;
        case FS_DIAG:
            for (uint32_t i = tid; i < dim; i += NT) {
                uint32_t l = 0;
                for (int b = 0; b < S.k; ++b) l |= ((i >> S.q[b]) & 1u) << b;
                vec2_t<T>& v = a[fs_slot<T>(i)];
                v = cmul_d<T>(c[2 * l], c[2 * l + 1], v);
            }
            break;
        case FS_PHASE: {
            const uint32_t mask = static_cast<uint32_t>(S.mask);
            for (uint32_t i = tid; i < dim; i += NT)
                if ((i & mask) == mask) {
                    vec2_t<T>& v = a[fs_slot<T>(i)];
                    v = cmul_d<T>(c[0], c[1], v);
                }
            break;
        }
        case FS_SCALE:
            for (uint32_t i = tid; i < dim; i += NT) a[i] = cmul_d<T>(c[0], c[1], a[i]);
            break;
        case FS_SWAP: {
            const uint32_t A = 1u << S.q[0], B = 1u << S.q[1];
            const uint32_t lo = min(S.q[0], S.q[1]), hi = max(S.q[0], S.q[1]);
            for (uint32_t g = tid; g < dim / 4; g += NT) {
                const uint32_t base = fs_insert(fs_insert(g, lo), hi);
                vec2_t<T>&va = a[fs_slot<T>(base | A)], &vb = a[fs_slot<T>(base | B)];
                const vec2_t<T> t = va;
                va = vb;
                vb = t;
            }
            break;
        }
        case FS_PROT: {
            // exp(-i theta/2 P) on pairs (i, i ^ x), i without the lowest bit of x
            const double cs = c[0], sn = c[1];
            const uint32_t x = static_cast<uint32_t>(S.mask), z = static_cast<uint32_t>(S.zmask);
            const uint32_t ny = static_cast<uint32_t>(__popc(x & z)), pb = x ? static_cast<uint32_t>(__ffs(x) - 1) : 0u;
            for (uint32_t g = tid; g < (x ? dim / 2 : dim); g += NT) {
                const uint32_t i = x ? fs_insert(g, pb) : g;
                const uint32_t j = i ^ x, si = fs_slot<T>(i), sj = fs_slot<T>(j);
                const vec2_t<T> ai = a[si], aj = a[sj];
                // s[i] = c ai - i sn phase(j) aj,  phase(j) = i^ny (-1)^popcount(j & z)
                const vec2_t<T> pj = tr_pauli_phase<T>(aj, ny + 1, __popc(j & z) & 1);
                const vec2_t<T> pi = tr_pauli_phase<T>(ai, ny + 1, __popc(i & z) & 1);
                a[si] = mk<T>(static_cast<T>(cs * static_cast<double>(ai.x) - sn * static_cast<double>(pj.x)),
                              static_cast<T>(cs * static_cast<double>(ai.y) - sn * static_cast<double>(pj.y)));
                if (x)
                    a[sj] = mk<T>(static_cast<T>(cs * static_cast<double>(aj.x) - sn * static_cast<double>(pi.x)),
                                  static_cast<T>(cs * static_cast<double>(aj.y) - sn * static_cast<double>(pi.y)));
            }
            break;
        }
        default:
            return false;
    }
    return true;
}

// What a shot keeps in shared memory besides its amplitudes and its engine's words.
template <int NT>
struct FsShot {
    double red[4 * (NT / 32)];
    double part[NT];
    double bc[10];
    uint64_t cbits, flags, bx, bz;
    uint32_t mt_idx, bny;
    int bflag, pad;
};

// A step costs a chain of a few hundred cycles (record, indices, the unit's latency, a barrier),
// shared-memory traffic second.  10 qubits, 20000 shots of about 140 steps: 8.54 ms with 64-bit
// indices, rows one at a time, whole engines seeded and twisted and 256 threads a shot; 4.9 ms now.
//
// Shots of NT threads, W of them to a block.  W > 1 is a shot per warp (NT = 32, resident plan): a
// register of a few amplitudes per lane waits for its chain of steps, draws and decisions, so what
// counts is how many chains a multiprocessor holds, and warps that share a plan need no barrier.
template <typename T, int NT, int W>
__global__ void __launch_bounds__(NT * W, NT == 128 ? 5 : 3) k_fs_run(
    const FsStep* __restrict__ steps, int n_steps, const double* __restrict__ coef, uint32_t n_coef, int resident,
    const vec2_t<T>* __restrict__ prefix, int n, uint32_t seed, uint64_t shot0, uint64_t n_shots,
    uint64_t* __restrict__ out_idx, uint64_t* __restrict__ out_cbits) {
    static_assert(W == 1 || NT == 32, "several shots per block: a warp each");
    // dynamic shared memory: per shot its amplitudes and its MT19937 words, then the plan
    // (resident) or one step's coefficients
    extern __shared__ __align__(16) unsigned char fs_smem[];
    const uint32_t tid = W == 1 ? threadIdx.x : threadIdx.x & (NT - 1);
    const uint32_t grp = W == 1 ? 0 : threadIdx.x / NT;
    const uint32_t dim = 1u << n;
    const size_t amp_area = (static_cast<size_t>(dim) * sizeof(vec2_t<T>) + 15) & ~size_t{15};
    vec2_t<T>* a = reinterpret_cast<vec2_t<T>*>(fs_smem + grp * amp_area);
    uint32_t* mtw = reinterpret_cast<uint32_t*>(fs_smem + W * amp_area + grp * kFsMtBytes);
    uint64_t* rsteps = reinterpret_cast<uint64_t*>(fs_smem + W * (amp_area + kFsMtBytes));
    double* rcoef = reinterpret_cast<double*>(rsteps + static_cast<size_t>(n_steps) * (sizeof(FsStep) / 8));
    __shared__ __align__(16) uint64_t sstep[sizeof(FsStep) / 8];   // streamed plans (W = 1): the current step
    double* const scoef = reinterpret_cast<double*>(rsteps);
    __shared__ FsShot<NT> shared_shot[W];
    FsShot<NT>& H = shared_shot[grp];
    const MtView g{mtw, 1, &H.mt_idx};
    static_assert(sizeof(FsStep) % 16 == 0, "FsStep is staged as 8-byte words and keeps rcoef aligned");

    if (resident) {
        const uint64_t* src = reinterpret_cast<const uint64_t*>(steps);
        const size_t words = static_cast<size_t>(n_steps) * (sizeof(FsStep) / 8);
        for (size_t w = threadIdx.x; w < words; w += NT * W) rsteps[w] = __ldg(QSV_DBG(src + w));
        for (uint32_t w = threadIdx.x; w < n_coef; w += NT * W) rcoef[w] = __ldg(QSV_DBG(coef + w));
        if (W > 1) __syncthreads();
    }

    // persistent blocks: shots first, first + stride, ...
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * W;
    for (uint64_t shot = static_cast<uint64_t>(blockIdx.x) * W + grp; shot < n_shots; shot += stride) {
    for (uint32_t i = tid; i < dim; i += NT) a[fs_slot<T>(i)] = *QSV_DBG(prefix + i);
    if (tid == 0) {
        g.seed(seed + static_cast<uint32_t>(shot0 + shot));
        H.cbits = 0;
        H.flags = 0;
    }
    fs_sync<NT>();

    for (int si = 0; si < n_steps; ++si) {
        if (!resident) {
            const uint64_t* src = reinterpret_cast<const uint64_t*>(steps + si);
            for (int w = tid; w < static_cast<int>(sizeof(FsStep) / 8); w += NT)
                sstep[w] = __ldg(QSV_DBG(src + w));
            fs_sync<NT>();
        }
        const FsStep& S = resident ? *reinterpret_cast<const FsStep*>(rsteps + si * (sizeof(FsStep) / 8))
                                   : *reinterpret_cast<const FsStep*>(sstep);
        if ((H.flags & S.fmask) != S.fwant || (H.cbits & S.cmask) != S.cwant) {   // uniform in the CTA
            if (!resident) fs_sync<NT>();                                      // sstep is read
            continue;
        }
        const double* c = rcoef + S.coef;
        if (!resident) {
            for (uint32_t w = tid; w < S.ncoef; w += NT) scoef[w] = __ldg(QSV_DBG(coef + (S.coef + w)));
            fs_sync<NT>();
            c = scoef;
        }
        if (!fs_gate<T, NT>(a, n, S, c, tid)) switch (S.kind) {
            case FS_MEASURE: {
                const uint32_t q = S.q[0], ob = fs_slot<T>(1u << q);
                double acc = 0.0;
                for (uint32_t gi = tid; gi < dim / 2; gi += NT)
                    acc += tr_norm2<T>(a[fs_slot<T>(fs_insert(gi, q))]);
                fs_sums<NT, 1>(&acc, H.red, tid);
                const double p0 = acc;
                if (tid == 0) {
                    double sc = 0.0;
                    const bool one = tr_decide(p0, g, &sc);
                    H.bflag = one ? 1 : 0;
                    H.bc[0] = sc;
                    if (S.cbit >= 0) H.cbits = one ? (H.cbits | (1ull << S.cbit)) : (H.cbits & ~(1ull << S.cbit));
                }
                fs_sync<NT>();
                const int one = H.bflag;
                const double sc = H.bc[0];
                for (uint32_t gi = tid; gi < dim / 2; gi += NT) {
                    const uint32_t i = fs_slot<T>(fs_insert(gi, q)), i1 = i ^ ob;
                    const vec2_t<T> keep = a[one ? i1 : i];
                    const vec2_t<T> v = mk<T>(static_cast<T>(static_cast<double>(keep.x) * sc),
                                              static_cast<T>(static_cast<double>(keep.y) * sc));
                    const bool up = one && !S.k;
                    a[up ? i1 : i] = v;
                    a[up ? i : i1] = mk<T>(T(0), T(0));
                }
                break;
            }
            case FS_BRANCH:
                if (tid == 0) {
                    const uint64_t holds = (H.cbits & S.mask) == S.zmask ? 1ull : 0ull;
                    H.flags = (H.flags & ~(1ull << S.flag)) | (holds << S.flag);
                }
                break;
            case FS_PAULI_NOISE: {
                if (tid == 0) {
                    TrQubits tq;
                    tq.k = S.k;
                    for (int b = 0; b < 32; ++b) tq.q[b] = S.q[b];
                    uint64_t x, z;
                    uint32_t ny;
                    tr_choose_pauli(S.k2, c, tq, g, x, z, ny);
                    H.bx = x;
                    H.bz = z;
                    H.bny = ny;
                }
                fs_sync<NT>();
                const uint32_t x = static_cast<uint32_t>(H.bx), z = static_cast<uint32_t>(H.bz);
                const uint32_t ny = H.bny;
                if (!(x | z)) break;
                if (x == 0) {
                    for (uint32_t j = tid; j < dim; j += NT) {
                        vec2_t<T>& v = a[fs_slot<T>(j)];
                        v = tr_pauli_phase<T>(v, ny, __popc(j & z) & 1);
                    }
                } else {
                    const uint32_t hb = 31u - static_cast<uint32_t>(__clz(x)), ox = fs_slot<T>(x);
                    for (uint32_t gi = tid; gi < dim / 2; gi += NT) {
                        const uint32_t j = fs_insert(gi, hb), j2 = j ^ x, sj = fs_slot<T>(j);
                        const vec2_t<T> va = a[sj], vb = a[sj ^ ox];
                        a[sj ^ ox] = tr_pauli_phase<T>(va, ny, __popc(j & z) & 1);
                        a[sj] = tr_pauli_phase<T>(vb, ny, __popc(j2 & z) & 1);
                    }
                }
                break;
            }
            case FS_KRAUS_NOISE: {
                const uint32_t q = S.q[0], ob = fs_slot<T>(1u << q);
                double r00 = 0.0, r11 = 0.0, rr = 0.0, ri = 0.0;
                for (uint32_t gi = tid; gi < dim / 2; gi += NT) {
                    const uint32_t i0 = fs_slot<T>(fs_insert(gi, q));
                    const vec2_t<T> va = a[i0], vb = a[i0 ^ ob];
                    const double ar = va.x, ai = va.y, br = vb.x, bi = vb.y;
                    r00 += ar * ar + ai * ai;
                    r11 += br * br + bi * bi;
                    rr += ar * br + ai * bi;
                    ri += ai * br - ar * bi;
                }
                double rho[4] = {r00, r11, rr, ri};
                fs_sums<NT, 4>(rho, H.red, tid);
                r00 = rho[0];
                r11 = rho[1];
                rr = rho[2];
                ri = rho[3];
                if (tid == 0) H.bflag = tr_choose_kraus(r00, r11, rr, ri, c, S.k2, g, H.bc) ? 1 : 0;
                fs_sync<NT>();
                if (!H.bflag) break;
                const double m0 = H.bc[0], m1 = H.bc[1], m2 = H.bc[2], m3 = H.bc[3], m4 = H.bc[4], m5 = H.bc[5], m6 = H.bc[6],
                             m7 = H.bc[7];
                for (uint32_t gi = tid; gi < dim / 2; gi += NT) {
                    const uint32_t i0 = fs_slot<T>(fs_insert(gi, q));
                    const vec2_t<T> va = a[i0], vb = a[i0 ^ ob];
                    const double ar = va.x, ai = va.y, br = vb.x, bi = vb.y;
                    a[i0] = mk<T>(static_cast<T>((m0 * ar - m1 * ai) + (m2 * br - m3 * bi)),
                                  static_cast<T>((m0 * ai + m1 * ar) + (m2 * bi + m3 * br)));
                    a[i0 ^ ob] = mk<T>(static_cast<T>((m4 * ar - m5 * ai) + (m6 * br - m7 * bi)),
                                       static_cast<T>((m4 * ai + m5 * ar) + (m6 * bi + m7 * br)));
                }
                break;
            }
            default:
                break;
        }
        fs_sync<NT>();
    }

    // final sample: per-thread runs of consecutive amplitudes, their sums in index order, the
    // first index whose running sum reaches u * total (the last one when rounding never does).
    // The sums before each run are kept, so the run is found by bisection: they never decrease.
    const uint32_t per = dim >= NT ? dim / NT : 1;
    const uint32_t lo = tid * per;
    double run = 0.0;
    if (lo < dim)
        for (uint32_t i = lo; i < lo + per; ++i) run += tr_norm2<T>(a[fs_slot<T>(i)]);
    H.part[tid] = run;
    fs_sync<NT>();
    if (tid == 0) {
    const uint32_t runs = dim >= NT ? NT : dim;
    double total = 0.0;
#pragma unroll 8
    for (uint32_t t = 0; t < runs; ++t) {
        total += H.part[t];
        H.part[t] = total;
    }
    const double thr = g.canonical() * total;
    uint32_t t0 = 0, t1 = runs;   // the first run whose sum through it is not below thr
    while (t0 < t1) {
        const uint32_t t = (t0 + t1) / 2;
        if (H.part[t] < thr) t0 = t + 1;
        else t1 = t;
    }
    uint64_t idx = dim - 1;
    double acc = t0 ? H.part[t0 - 1] : 0.0;
    // past the run only when the sum amplitude by amplitude rounds below the run's
    for (uint32_t i = t0 * per; i < dim; ++i) {
        acc += tr_norm2<T>(a[fs_slot<T>(i)]);
        if (acc >= thr) {
            idx = i;
            break;
        }
    }
    *QSV_DBG(out_idx + shot) = idx;
    *QSV_DBG(out_cbits + shot) = H.cbits;
    }
    fs_sync<NT>();   // the next shot overwrites the amplitudes, H.part[] and the engine
    }
}

// A whole gate sequence on a small register in one CTA: the register is loaded into shared
// memory, every step applied there, and written back in place.  Replaces one launch per gate
// (each a few microseconds of launch latency for a few kilobytes of work) by one launch.  One
// multiprocessor's FP64 rate bounds it from 11 qubits: a 12-qubit ansatz of ten layers takes 128 us
// with 512 threads, two groups a thread and 32-bit places, 178 with 256 threads a group each.
template <typename T, int NT>
__global__ void __launch_bounds__(NT) k_fs_apply(const FsStep* __restrict__ steps, int n_steps,
                                                        const double* __restrict__ coef, uint32_t n_coef,
                                                        int resident, vec2_t<T>* __restrict__ state, int n) {
    extern __shared__ __align__(16) unsigned char fa_smem[];
    vec2_t<T>* a = reinterpret_cast<vec2_t<T>*>(fa_smem);
    const uint32_t dim = 1u << n;
    const size_t amp_area = (static_cast<size_t>(dim) * sizeof(vec2_t<T>) + 15) & ~size_t{15};
    uint64_t* rsteps = reinterpret_cast<uint64_t*>(fa_smem + amp_area);
    double* rcoef = reinterpret_cast<double*>(rsteps + static_cast<size_t>(n_steps) * (sizeof(FsStep) / 8));
    __shared__ __align__(16) uint64_t sstep[sizeof(FsStep) / 8];
    __shared__ __align__(16) double scoef[kFsMaxCoef];
    if (resident) {
        const uint64_t* src = reinterpret_cast<const uint64_t*>(steps);
        const size_t words = static_cast<size_t>(n_steps) * (sizeof(FsStep) / 8);
        for (size_t w = threadIdx.x; w < words; w += NT) rsteps[w] = __ldg(QSV_DBG(src + w));
        for (uint32_t w = threadIdx.x; w < n_coef; w += NT) rcoef[w] = __ldg(QSV_DBG(coef + w));
    }
    for (uint32_t i = threadIdx.x; i < dim; i += NT) a[fs_slot<T>(i)] = *QSV_DBG(state + i);
    __syncthreads();
    for (int si = 0; si < n_steps; ++si) {
        const double* c;
        const FsStep* S;
        if (resident) {
            S = reinterpret_cast<const FsStep*>(rsteps + si * (sizeof(FsStep) / 8));
            c = rcoef + S->coef;
        } else {
            const uint64_t* src = reinterpret_cast<const uint64_t*>(steps + si);
            for (int w = threadIdx.x; w < static_cast<int>(sizeof(FsStep) / 8); w += NT)
                sstep[w] = __ldg(QSV_DBG(src + w));
            __syncthreads();
            S = reinterpret_cast<const FsStep*>(sstep);
            for (uint32_t w = threadIdx.x; w < S->ncoef; w += NT) scoef[w] = __ldg(coef + S->coef + w);
            __syncthreads();
            c = scoef;
        }
        fs_gate<T, NT>(a, n, *S, c, threadIdx.x);
        __syncthreads();
    }
    for (uint32_t i = threadIdx.x; i < dim; i += NT) *QSV_DBG(state + i) = a[fs_slot<T>(i)];
}

// the places where a group's index takes zeros: the step's qubits and controls, ascending
void set_positions(FsStep& f) {
    uint64_t m = f.ctrl;
    for (int b = 0; b < f.k; ++b) m |= 1ull << f.q[b];
    f.k2 = 0;
    for (; m && f.k2 < 16; m &= m - 1) f.q[16 + f.k2++] = static_cast<uint8_t>(__builtin_ctzll(m));
}

// host: the plan's steps as FsSteps; false when a step has no shared-memory form
bool encode(const TrPlan& plan, std::vector<FsStep>& out, std::vector<double>& coef) {
    // every step's coefficients start on a 16-byte boundary (the dense rows are read as double2)
    auto start = [&](FsStep& f, const TrGuard& g) {
        f.fmask = g.fmask;
        f.fwant = g.fwant;
        f.cmask = g.cmask;
        f.cwant = g.cwant;
        if (coef.size() & 1) coef.push_back(0.0);
        f.coef = static_cast<uint32_t>(coef.size());
    };
    auto push_c = [&](c128 v) {
        coef.push_back(v.real());
        coef.push_back(v.imag());
    };
    auto op_step = [&](const Op& o, const TrGuard& g) -> bool {
        FsStep f;
        start(f, g);
        switch (o.kind) {
            case OP_NOP: return true;
            case OP_DENSE:
                if (o.k < 1 || o.k > 4) return false;
                f.kind = FS_DENSE;
                f.k = static_cast<uint8_t>(o.k);
                for (int b = 0; b < o.k; ++b) f.q[b] = static_cast<uint8_t>(o.qubits[b]);
                for (int b = 0; b < o.k; ++b)
                    if ((o.ctrl >> o.qubits[b]) & 1ull) return true;   // controlled on a target: never applies
                f.ctrl = o.ctrl;
                set_positions(f);
                for (const c128& v : o.m) push_c(v);
                break;
            case OP_CTRL1: {
                const uint64_t tb = 1ull << o.target;
                if (o.mask & tb) return true;   // the control set includes the target: never applies
                f.kind = FS_DENSE;
                f.k = 1;
                f.q[0] = static_cast<uint8_t>(o.target);
                f.ctrl = o.mask;
                set_positions(f);
                for (int e = 0; e < 4; ++e) push_c(o.m.at(e));
                break;
            }
            case OP_DIAG:
                if (o.k < 1 || o.k > 8) return false;
                f.kind = FS_DIAG;
                f.k = static_cast<uint8_t>(o.k);
                for (int b = 0; b < o.k; ++b) f.q[b] = static_cast<uint8_t>(o.qubits[b]);
                for (const c128& v : o.m) push_c(v);
                break;
            case OP_PHASE:
                f.kind = FS_PHASE;
                f.mask = o.mask;
                push_c(o.m.at(0));
                break;
            case OP_SCALE:
                f.kind = FS_SCALE;
                push_c(o.m.at(0));
                break;
            case OP_SWAP:
                f.kind = FS_SWAP;
                f.q[0] = static_cast<uint8_t>(o.qubits[0]);
                f.q[1] = static_cast<uint8_t>(o.qubits[1]);
                break;
            case OP_PAULI_ROT:
                f.kind = FS_PROT;
                f.mask = o.mask;
                f.zmask = o.zmask;
                push_c(o.m.at(0));
                break;
            default:
                return false;   // permutations
        }
        f.ncoef = static_cast<uint32_t>(coef.size()) - f.coef;
        out.push_back(f);
        return true;
    };
    auto finish = [&](FsStep& f) { f.ncoef = static_cast<uint32_t>(coef.size()) - f.coef; };
    for (const TrStep& st : plan.steps) {
        switch (st.kind) {
            case TrStep::OPS:
            case TrStep::MOPS:
                for (const Op& o : st.ops)
                    if (!op_step(o, st.kind == TrStep::OPS ? TrGuard{} : st.g)) return false;
                break;
            case TrStep::MDENSE: {
                FsStep f;
                start(f, st.g);
                f.kind = FS_DENSE;
                f.k = static_cast<uint8_t>(st.k);
                for (int b = 0; b < st.k; ++b) f.q[b] = static_cast<uint8_t>(__builtin_ctzll(st.args.off[1 << b]));
                set_positions(f);
                for (int e = 0; e < (1 << (2 * st.k)); ++e) {
                    coef.push_back(plan.mats[st.moff + e].re);
                    coef.push_back(plan.mats[st.moff + e].im);
                }
                finish(f);
                out.push_back(f);
                break;
            }
            case TrStep::MSCALE: {
                FsStep f;
                start(f, st.g);
                f.kind = FS_SCALE;
                push_c(st.phase);
                finish(f);
                out.push_back(f);
                break;
            }
            case TrStep::MEASURE: {
                FsStep f;
                start(f, st.g);
                f.kind = FS_MEASURE;
                f.q[0] = static_cast<uint8_t>(st.qubit);
                f.cbit = st.cbit;
                f.k = st.reset ? 1 : 0;
                finish(f);
                out.push_back(f);
                break;
            }
            case TrStep::BRANCH: {
                FsStep f;
                start(f, TrGuard{});
                f.kind = FS_BRANCH;
                f.flag = static_cast<uint8_t>(st.flag);
                f.mask = st.bmask;
                f.zmask = st.bwant;
                finish(f);
                out.push_back(f);
                break;
            }
            case TrStep::NOISE: {
                FsStep f;
                start(f, st.g);
                f.k = static_cast<uint8_t>(st.nq.k);
                for (int b = 0; b < 32; ++b) f.q[b] = st.nq.q[b];
                if (st.noise == NOISE_KRAUS) {
                    f.kind = FS_KRAUS_NOISE;
                    f.k2 = static_cast<uint8_t>(st.n_ops);
                    coef.insert(coef.end(), plan.noise_prm.begin() + st.poff,
                                plan.noise_prm.begin() + st.poff + 8 * st.n_ops);
                } else {
                    f.kind = FS_PAULI_NOISE;
                    f.k2 = static_cast<uint8_t>(st.noise);
                    const size_t np = st.noise == NOISE_PAULI ? 3 : st.noise == NOISE_PAULI2 ? 15 : 1;
                    coef.insert(coef.end(), plan.noise_prm.begin() + st.poff, plan.noise_prm.begin() + st.poff + np);
                }
                finish(f);
                out.push_back(f);
                break;
            }
        }
    }
    for (const FsStep& f : out) {
        if (f.ncoef > static_cast<uint32_t>(kFsMaxCoef)) return false;
        // the kernel reads dense rows as double2 from f.coef and stages ncoef doubles
        if ((f.coef & 1u) || static_cast<size_t>(f.coef) + f.ncoef > coef.size())
            throw std::logic_error("fused trajectory plan: misplaced coefficients");
    }
    return true;
}

}  // namespace

template <typename T>
bool run_trajectories_fused(const TrPlan& plan, int n, const vec2_t<T>* d_prefix, uint32_t seed, size_t n_shots,
                            uint64_t* out_idx, uint64_t* out_cbits, cudaStream_t st, Workspace& ws,
                            uint64_t* launches) {
    const size_t amp_bytes = sizeof(vec2_t<T>) << n;
    if (amp_bytes > static_cast<size_t>(kFsMaxBytes)) return false;
    std::vector<FsStep> steps;
    std::vector<double> coef;
    if (!encode(plan, steps, coef)) return false;
    if (coef.empty()) coef.push_back(0.0);

    constexpr uint64_t kChunk = 1ull << 20;   // shots per launch
    const uint64_t chunk = std::min<uint64_t>(kChunk, n_shots);
    const size_t steps_bytes = steps.size() * sizeof(FsStep);
    const size_t coef_off = (steps_bytes + 15) & ~size_t{15};
    const size_t out_off = coef_off + ((coef.size() * sizeof(double) + 15) & ~size_t{15});
    uint8_t* p = static_cast<uint8_t*>(ws.shots(out_off + 16 * chunk));
    FsStep* d_steps = reinterpret_cast<FsStep*>(p);
    double* d_coef = reinterpret_cast<double*>(p + coef_off);
    uint64_t* d_out = reinterpret_cast<uint64_t*>(p + out_off);
    uint64_t* d_cb = d_out + chunk;
    uint64_t* h = reinterpret_cast<uint64_t*>(ws.host_result(2 * chunk));
    if (!steps.empty())
        check_cuda(cudaMemcpyAsync(d_steps, steps.data(), steps_bytes, cudaMemcpyHostToDevice, st), "steps H2D");
    check_cuda(cudaMemcpyAsync(d_coef, coef.data(), coef.size() * sizeof(double), cudaMemcpyHostToDevice, st),
               "coefficients H2D");
    // the plan stays in shared memory when it fits next to the amplitudes, else each step is
    // staged from global memory as it comes
    const size_t prog_bytes = steps_bytes + coef.size() * sizeof(double);
    const size_t amp_area = (amp_bytes + 15) & ~size_t{15};
    const size_t shot_area = amp_area + kFsMtBytes;
    int dev = 0, sms = 0, per_sm = 0;
    check_cuda(cudaGetDevice(&dev), "device");
    check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "sm count");
    bool noise = false;
    for (const FsStep& f : steps) noise |= f.kind == FS_PAULI_NOISE || f.kind == FS_KRAUS_NOISE;
    const bool many = n_shots >= static_cast<size_t>(kFsWarpShots) * static_cast<size_t>(sms);
    const int warp_bytes = !many ? kFsWarpBytes : noise ? kFsWarpBytesNoise : kFsWarpBytesMany;
    // eight shots and their plan take what one block may have beside the kernel's own shared memory
    bool warps = amp_bytes <= static_cast<size_t>(warp_bytes);
    if (warps) {
        int block_max = 0;
        check_cuda(cudaDeviceGetAttribute(&block_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev), "block shared memory");
        cudaFuncAttributes own{};
        check_cuda(cudaFuncGetAttributes(&own, k_fs_run<T, 32, kFsWarpShots>), "fused trajectory kernel");
        warps = kFsWarpShots * shot_area + prog_bytes + own.sharedSizeBytes <= static_cast<size_t>(block_max);
    }
    const int resident = warps || shot_area + prog_bytes <= kFsResidentMax ? 1 : 0;
    const int per_cta = warps ? kFsWarpShots : 1;
    const size_t smem = per_cta * shot_area + (resident ? prog_bytes : kFsMaxCoef * sizeof(double));
    const int threads = warps ? 32 * kFsWarpShots : amp_bytes <= static_cast<size_t>(kFsNarrowBytes) ? 128 : 256;
    const auto kern = warps ? k_fs_run<T, 32, kFsWarpShots> : threads == 128 ? k_fs_run<T, 128, 1> : k_fs_run<T, 256, 1>;
    check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
               "fused trajectory smem");
    check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                    cudaSharedmemCarveoutMaxShared), "fused trajectory carveout");
    check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem), "occupancy");
    const uint64_t resident_ctas = static_cast<uint64_t>(sms) * std::max(per_sm, 1);
    for (uint64_t s0 = 0; s0 < n_shots; s0 += chunk) {
        const uint64_t nb = std::min<uint64_t>(chunk, n_shots - s0);
        const unsigned grid = static_cast<unsigned>(std::min<uint64_t>((nb + per_cta - 1) / per_cta, resident_ctas));
        kern<<<grid, threads, smem, st>>>(d_steps, static_cast<int>(steps.size()), d_coef,
                                          static_cast<uint32_t>(coef.size()), resident, d_prefix, n, seed, s0, nb,
                                          d_out, d_cb);
        check_cuda(cudaGetLastError(), "fused trajectory launch");
        check_cuda(cudaMemcpyAsync(h, d_out, 8 * nb, cudaMemcpyDeviceToHost, st), "D2H");
        check_cuda(cudaMemcpyAsync(h + chunk, d_cb, 8 * nb, cudaMemcpyDeviceToHost, st), "D2H");
        check_cuda(cudaStreamSynchronize(st), "fused trajectories");   // the host copies and the
        std::memcpy(out_idx + s0, h, 8 * nb);                          // step upload are done
        std::memcpy(out_cbits + s0, h + chunk, 8 * nb);
        if (launches) ++*launches;
    }
    return true;
}

template <typename T>
bool apply_ops_small(const std::vector<Op>& ops, vec2_t<T>* s, int n, cudaStream_t st, Workspace& ws) {
    const size_t amp_bytes = sizeof(vec2_t<T>) << n;
    if (amp_bytes > static_cast<size_t>(kFsMaxBytes) || ops.size() < 2) return false;
    TrPlan plan;
    plan.steps.emplace_back();
    plan.steps.back().kind = TrStep::OPS;
    plan.steps.back().ops = ops;
    std::vector<FsStep> steps;
    std::vector<double> coef;
    if (!encode(plan, steps, coef)) return false;
    if (steps.empty()) return true;
    if (coef.empty()) coef.push_back(0.0);
    const size_t steps_bytes = steps.size() * sizeof(FsStep);
    const size_t coef_off = (steps_bytes + 15) & ~size_t{15};
    std::vector<unsigned char> blob(coef_off + coef.size() * sizeof(double));
    std::memcpy(blob.data(), steps.data(), steps_bytes);
    std::memcpy(blob.data() + coef_off, coef.data(), coef.size() * sizeof(double));
    unsigned char* d = static_cast<unsigned char*>(ws.shots(blob.size()));
    // pageable source: staged before cudaMemcpyAsync returns; stream order protects the buffer
    check_cuda(cudaMemcpyAsync(d, blob.data(), blob.size(), cudaMemcpyHostToDevice, st), "gate program H2D");
    const size_t amp_area = (amp_bytes + 15) & ~size_t{15};
    const size_t prog_bytes = steps_bytes + coef.size() * sizeof(double);
    const int resident = amp_area + prog_bytes <= kFsApplyResidentMax ? 1 : 0;
    const size_t smem = amp_area + (resident ? prog_bytes : 0);
    auto launch = [&](auto kern, int threads) {
        check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
                   "small-register smem");
        kern<<<1, threads, smem, st>>>(reinterpret_cast<const FsStep*>(d), static_cast<int>(steps.size()),
                                       reinterpret_cast<const double*>(d + coef_off),
                                       static_cast<uint32_t>(coef.size()), resident, s, n);
    };
    if (n < kFsApplyWide) launch(k_fs_apply<T, 128>, 128);
    else launch(k_fs_apply<T, 512>, 512);
    check_cuda(cudaGetLastError(), "small-register launch");
    return true;
}

template bool apply_ops_small<double>(const std::vector<Op>&, double2*, int, cudaStream_t, Workspace&);
template bool apply_ops_small<float>(const std::vector<Op>&, float2*, int, cudaStream_t, Workspace&);

template bool run_trajectories_fused<double>(const TrPlan&, int, const double2*, uint32_t, size_t, uint64_t*,
                                             uint64_t*, cudaStream_t, Workspace&, uint64_t*);
template bool run_trajectories_fused<float>(const TrPlan&, int, const float2*, uint32_t, size_t, uint64_t*,
                                            uint64_t*, cudaStream_t, Workspace&, uint64_t*);

// ---------------------------------------------------------------- circuit batches
//
// Many circuits of up to 12 qubits (complex128), each with its own observable and parameter
// values, in one persistent launch: a CTA takes the next instance from a queue (widest first),
// keeps |psi> and |phi> = H|psi> in shared memory, runs the forward gate steps, <H>, and — for
// gradients — the reverse sweep of run_gradient_core (qarp_simulator.cpp:1519-1605): for each
// parametric command, last first, <phi| G |psi> into its slot and the command's dagger applied
// to both registers; other commands' daggers to both.  The reference evaluates such batches one
// circuit at a time (QarpSimulator::batch_expectation, qarp_simulator.cpp:971-984; the engine
// sweep, _qarp_engine.py:450-503).

namespace {

constexpr int kCbMaxQubits = 12;   // both registers in shared memory
constexpr int kCbNarrow = 10;      // registers below it: 32 KiB a CTA, several per multiprocessor
constexpr int kCbMaxWide = 16;     // wider members: the CTA's pair in a global scratch slot (L2)

struct CbInstDev {
    int32_t n, pad;
    uint32_t f0, f1;        // forward steps
    uint32_t r0, r1;        // reverse steps
    uint32_t t0, t1;        // Pauli terms
    uint32_t slot0, nslot;  // adjoint slots
};

// A sum over the warp, in every lane.
__device__ __forceinline__ double2 cb_warp_sum2(double2 v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    return v;
}

// An adjoint step on q[0..K): this thread's part of <phi| G |psi>, and D applied to both
// registers, from one read of each group.  G and D: 2^K x 2^K entries each at m.
template <int K, int NT>
__device__ __forceinline__ double2 cb_adjoint(double2* psi, double2* phi, int n, const FsStep& S,
                                              const double* __restrict__ m) {
    constexpr int D = 1 << K;
    uint32_t off[D];
    fs_offsets<double, K>(S, off);
    const FsGroups at(S);
    const uint32_t groups = 1u << (n - K);
    const double2* const gm = reinterpret_cast<const double2*>(m);
    const double2* const dm = gm + D * D;
    double ar = 0.0, ai = 0.0;
    auto times = [&](const double2* mat, int y, const double2* v) {   // row y of mat, times v
        double2 o = make_double2(0.0, 0.0);
#pragma unroll
        for (int x = 0; x < D; ++x) {
            const double2 cf = mat[y * D + x];
            o.x = fma(cf.x, v[x].x, o.x);
            o.x = fma(-cf.y, v[x].y, o.x);
            o.y = fma(cf.x, v[x].y, o.y);
            o.y = fma(cf.y, v[x].x, o.y);
        }
        return o;
    };
    for (uint32_t g = threadIdx.x; g < groups; g += NT) {
        const uint32_t base = fs_slot<double>(at.base<K>(g));
        double2 p[D], f[D];
#pragma unroll
        for (int x = 0; x < D; ++x) {
            p[x] = psi[base ^ off[x]];
            f[x] = phi[base ^ off[x]];
        }
        auto row = [&](int y, double2 fy, uint32_t oy) {   // conj(f) * (G psi)
            const double2 gp = times(gm, y, p);
            ar = fma(fy.x, gp.x, ar);
            ar = fma(fy.y, gp.y, ar);
            ai = fma(fy.x, gp.y, ai);
            ai = fma(-fy.y, gp.x, ai);
            psi[base ^ oy] = times(dm, y, p);
            phi[base ^ oy] = times(dm, y, f);
        };
        if constexpr (K < 2) {
#pragma unroll
            for (int y = 0; y < D; ++y) row(y, f[y], off[y]);
        } else {   // one row at a time: all of them at once would spill
#pragma unroll 1
            for (int y = 0; y < D; ++y) {
                const double2 lo = (y & 1) ? f[1] : f[0], hi = (y & 1) ? f[3] : f[2];
                row(y, (y & 2) ? hi : lo, ((y & 1) ? off[1] : 0u) ^ ((y & 2) ? off[2] : 0u));
            }
        }
    }
    return make_double2(ar, ai);
}

// Instances [i0, i1) of one width class, NT threads a CTA, both registers of up to `sm_qubits`
// qubits in shared memory.  What a narrow instance waits for is the chain of its steps, not
// arithmetic: the next step's coefficients and the record after it are fetched while a step runs,
// one barrier a step, and an adjoint step's sums over the warps are added up by one warp while the
// others go on.  The reverse sweep's plain gates run on psi and phi at once, half of the threads
// each.  512 hardware-efficient ansaetze of 6..12 qubits with gradients: 1.46 ms as one launch of one
// instance per multiprocessor, each step staged before it ran; 0.60 ms as three classes side by side
// (alone: 0.41, 0.36 and 0.15 ms for 12, 10..11 and 6..9 qubits).
template <int NT>
__global__ void __launch_bounds__(NT) k_cb_run(const CbInstDev* __restrict__ inst, int i0, int i1,
                                               const FsStep* __restrict__ steps, const double* __restrict__ coef,
                                               const uint64_t* __restrict__ tx, const uint64_t* __restrict__ tz,
                                               const double2* __restrict__ tc, int with_grad,
                                               int* __restrict__ queue, double* __restrict__ energy,
                                               double2* __restrict__ slots, double2* __restrict__ wide,
                                               int wide_qubits, int sm_qubits) {
    extern __shared__ __align__(16) unsigned char cb_smem[];
    double2* const sm_psi = reinterpret_cast<double2*>(cb_smem);
    constexpr int kWords = sizeof(FsStep) / 8, kPer = (kFsMaxCoef + NT - 1) / NT, kWarps = NT / 32;
    static_assert(kWords <= 32 && kWarps <= 32, "a record by one warp, the warps' sums by one");
    __shared__ __align__(16) uint64_t srec[3][kWords];
    __shared__ __align__(16) double scoef[2][kFsMaxCoef];
    __shared__ double2 red[2][kWarps];
    __shared__ int cur;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (;;) {
        if (tid == 0) cur = atomicAdd(QSV_DBG(queue), 1);
        __syncthreads();
        const int i = i0 + cur;
        if (i >= i1) break;
        const CbInstDev I = *QSV_DBG(inst + i);
        const int n = I.n;
        const uint32_t dim = 1u << n;
        // registers of up to sm_qubits qubits in shared memory, wider ones in this CTA's
        // scratch slot (2 x 2^wide_qubits amplitudes; the host sized it for the widest member)
        double2* psi = sm_psi;
        if (n > sm_qubits) {
            psi = wide + (static_cast<uint64_t>(blockIdx.x) << (wide_qubits + 1));
            if (!QSV_DBG_RANGE_OK(psi, 32ull << wide_qubits)) {   // the debug build's check of the slot
                __syncthreads();
                continue;
            }
        }
        double2* phi = psi + (n > sm_qubits ? (1ull << wide_qubits) : (1ull << sm_qubits));
        for (uint32_t j = tid; j < dim; j += NT) psi[j] = make_double2(j == 0 ? 1.0 : 0.0, 0.0);   // slot 0 is amplitude 0
        const uint32_t s1 = with_grad ? I.r1 : I.f1;   // forward steps, then reverse steps: f1 == r0
        const auto rec_word = [&](uint32_t s) -> uint64_t {
            return tid < kWords && s < s1 ? __ldg(QSV_DBG(reinterpret_cast<const uint64_t*>(steps + s) + tid)) : 0ull;
        };
        // the first step's record and coefficients, and the second's record
        {
            const uint64_t w0 = rec_word(I.f0), w1 = rec_word(I.f0 + 1);
            if (tid < kWords) {
                srec[0][tid] = w0;
                srec[1][tid] = w1;
            }
            __syncthreads();
            const FsStep& F = *reinterpret_cast<const FsStep*>(srec[0]);
            if (I.f0 < s1)
                for (uint32_t w = tid; w < F.ncoef && w < static_cast<uint32_t>(kFsMaxCoef); w += NT)
                    scoef[0][w] = __ldg(QSV_DBG(coef + (F.coef + w)));
            __syncthreads();
        }
        int slot = 0, buf = 0, par = 0;
        // one step: `body` on its record and coefficients between the next ones' loads and stores
        auto step = [&](uint32_t s, auto body) {
            const int next = slot == 2 ? 0 : slot + 1, after = next == 2 ? 0 : next + 1;
            const FsStep& N = *reinterpret_cast<const FsStep*>(srec[next]);
            const uint64_t w2 = rec_word(s + 2);
            double pc[kPer];
            const uint32_t nc = s + 1 < s1 ? min(N.ncoef, static_cast<uint32_t>(kFsMaxCoef)) : 0u;
#pragma unroll
            for (int u = 0; u < kPer; ++u) {
                const uint32_t w = tid + u * NT;
                pc[u] = w < nc ? __ldg(QSV_DBG(coef + (N.coef + w))) : 0.0;
            }
            body(*reinterpret_cast<const FsStep*>(srec[slot]), scoef[buf]);
            if (tid < kWords) srec[after][tid] = w2;   // read last in the step before this one
#pragma unroll
            for (int u = 0; u < kPer; ++u) {
                const uint32_t w = tid + u * NT;
                if (w < nc) scoef[buf ^ 1][w] = pc[u];
            }
            __syncthreads();
            slot = next;
            buf ^= 1;
        };
        for (uint32_t s = I.f0; s < I.f1; ++s)
            step(s, [&](const FsStep& S, const double* c) { fs_gate<double, NT>(psi, n, S, c, tid); });
        // phi = H psi: phi[j] = sum_t c_t (-1)^popcount((j ^ x_t) & z_t) psi[j ^ x_t]
        double er = 0.0;
        for (uint32_t j = tid; j < dim; j += NT) {
            double fr = 0.0, fi = 0.0;
            for (uint32_t t = I.t0; t < I.t1; ++t) {
                const uint32_t x = static_cast<uint32_t>(__ldg(QSV_DBG(tx + t))), z = static_cast<uint32_t>(__ldg(QSV_DBG(tz + t)));
                const double2 c = __ldg(QSV_DBG(tc + t));
                const double2 v = psi[fs_slot<double>(j ^ x)];
                const double sg = (__popc((j ^ x) & z) & 1) ? -1.0 : 1.0;
                fr = fma(sg, c.x * v.x - c.y * v.y, fr);
                fi = fma(sg, c.x * v.y + c.y * v.x, fi);
            }
            const uint32_t sj = fs_slot<double>(j);
            phi[sj] = make_double2(fr, fi);
            const double2 p = psi[sj];
            er = fma(p.x, fr, er);
            er = fma(p.y, fi, er);
        }
        const double2 we = cb_warp_sum2(make_double2(er, 0.0));
        if (lane == 0) red[par][warp] = we;
        __syncthreads();
        // the warps' sums of the last reduction, added up by warp 0 (red[par] is written again
        // two reductions, so at least one barrier, later)
        auto collect = [&]() -> double2 {
            const double2 v = lane < kWarps ? red[par][lane] : make_double2(0.0, 0.0);
            return cb_warp_sum2(v);
        };
        if (warp == 0) {
            const double2 e = collect();
            if (lane == 0) *QSV_DBG(energy + I.pad) = e.x;   // at the caller's instance index
        }
        par ^= 1;
        if (with_grad) {
            for (uint32_t s = I.r0; s < I.r1; ++s) {
                int out = -1;
                step(s, [&](const FsStep& S, const double* c) {
                    if (S.kind == FS_ADJ) {
                        const double2 v = S.k == 0   ? cb_adjoint<0, NT>(psi, phi, n, S, c)
                                          : S.k == 1 ? cb_adjoint<1, NT>(psi, phi, n, S, c)
                                                     : cb_adjoint<2, NT>(psi, phi, n, S, c);
                        const double2 w = cb_warp_sum2(v);
                        if (lane == 0) red[par][warp] = w;
                        out = S.cbit;
                    } else {
                        fs_gate<double, NT / 2>(tid < NT / 2 ? psi : phi, n, S, c, tid & (NT / 2 - 1));
                    }
                });
                if (out >= 0) {
                    if (warp == 0) {
                        const double2 ip = collect();
                        if (lane == 0) *QSV_DBG(slots + (I.slot0 + static_cast<uint32_t>(out))) = ip;
                    }
                    par ^= 1;
                }
            }
        }
        __syncthreads();   // the registers and `cur` are free for the next instance
    }
}

struct CbInstHost {
    int n = 0;
    int n_params = 0;
    uint32_t f0 = 0, f1 = 0, r0 = 0, r1 = 0, t0 = 0, t1 = 0, slot0 = 0;
    uint32_t coef0 = 0, coef1 = 0;   // the instance's coefficient range
    std::vector<int32_t> slot_cmd;   // per slot: the parametric command
    std::vector<c128> slot_pref;
    std::vector<int32_t> dep_ptr, dep_param;
    std::vector<double> dep_alpha;
};

// the forward steps, reverse steps and coefficients of one instance (its parameters in place)
void cb_encode(const std::vector<Cmd>& cmds, int n, const int32_t* dep_ptr, bool grad, std::vector<FsStep>& fwd,
               std::vector<FsStep>& rev, std::vector<double>& coef, std::vector<c128>* prefs) {
    TrPlan fp;
    fp.steps.emplace_back();
    fp.steps.back().kind = TrStep::OPS;
    for (const Cmd& c : fuse_for_dispatch(cmds, n, 3, 0))
        for (Op& o : lower(c, n)) fp.steps.back().ops.push_back(std::move(o));
    if (!encode(fp, fwd, coef)) throw capability_error("circuit batch: a command has no shared-memory form");
    if (!grad) return;
    int slot = 0;
    for (size_t idx = cmds.size(); idx-- > 0;) {
        const Cmd& c = cmds[idx];
        if (dep_ptr[idx + 1] > dep_ptr[idx]) {
            c128 pref;
            std::vector<c128> G;
            int k = 0;
            if (!generator(c, &pref, &G, &k))
                throw capability_error("run_gradient: gate '" + std::to_string(c.gate) +
                                       "' carries a symbolic parameter but has no adjoint generator rule");
            std::vector<c128> D;
            if (k == 0) {
                const double th = -c.p.at(0);
                D = {c128(std::cos(th), std::sin(th))};
            } else {
                D = local_unitary(dagger(c));
            }
            FsStep f;
            if (coef.size() & 1) coef.push_back(0.0);
            f.kind = FS_ADJ;
            f.k = static_cast<uint8_t>(k);
            for (int b = 0; b < k; ++b) f.q[b] = static_cast<uint8_t>(c.q[b]);
            set_positions(f);
            f.cbit = slot++;
            f.coef = static_cast<uint32_t>(coef.size());
            for (const c128& v : G) { coef.push_back(v.real()); coef.push_back(v.imag()); }
            for (const c128& v : D) { coef.push_back(v.real()); coef.push_back(v.imag()); }
            f.ncoef = static_cast<uint32_t>(coef.size()) - f.coef;
            rev.push_back(f);
            if (prefs) prefs->push_back(pref);
        } else {
            TrPlan rp;
            rp.steps.emplace_back();
            rp.steps.back().kind = TrStep::OPS;
            for (Op& o : lower(dagger(c), n)) rp.steps.back().ops.push_back(std::move(o));
            if (!encode(rp, rev, coef)) throw capability_error("circuit batch: a command has no shared-memory form");
        }
    }
}

}  // namespace

struct CircuitBatch {
    int device = 0;
    cudaStream_t stream = nullptr;
    std::vector<CbInstHost> inst;
    std::vector<FsStep> steps;
    std::vector<double> coef;
    std::vector<uint64_t> tx, tz;
    std::vector<double> tc;
    uint32_t n_slots = 0;
    bool grad = false;
    // device side, built by finalize
    unsigned char* dev = nullptr;
    double2* wide = nullptr;           // members above 12 qubits: one register pair per CTA
    int wide_qubits = 0;
    double* host_coef = nullptr;       // pinned: the graph's source of coefficients
    double* host_out = nullptr;        // pinned: energies then slots
    size_t off_inst = 0, off_steps = 0, off_coef = 0, off_tx = 0, off_tz = 0, off_tc = 0, off_queue = 0,
           off_energy = 0, off_slots = 0, total = 0;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaStream_t side[2] = {};         // the narrower classes' branches of the graph
    cudaEvent_t fork = nullptr, join[2] = {};

    ~CircuitBatch() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        if (dev) dev_free(dev);
        if (wide) dev_free(wide);
        if (host_coef) cudaFreeHost(host_coef);
        if (host_out) cudaFreeHost(host_out);
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        if (fork) cudaEventDestroy(fork);
        for (cudaEvent_t e : join)
            if (e) cudaEventDestroy(e);
        for (cudaStream_t t : side)
            if (t) cudaStreamDestroy(t);
        if (stream) cudaStreamDestroy(stream);
    }
};

void* cbatch_create(int device, bool with_gradient) {
    auto* b = new CircuitBatch();
    b->device = device;
    b->grad = with_gradient;
    return b;
}

int cbatch_add(void* bp, const std::vector<Cmd>& cmds, int n, const int32_t* dep_ptr, const int32_t* dep_param,
               const double* dep_alpha, int n_params, const PauliTerms& terms) {
    CircuitBatch* b = static_cast<CircuitBatch*>(bp);
    if (b->exec) throw std::invalid_argument("circuit batch: instances are added before the first run");
    if (n < 1 || n > kCbMaxWide)
        throw capability_error("circuit batch: registers of 1.." + std::to_string(kCbMaxWide) + " qubits");
    CbInstHost h;
    h.n = n;
    h.n_params = b->grad ? n_params : 0;
    std::vector<FsStep> fwd, rev;
    const size_t c0 = b->coef.size();
    cb_encode(cmds, n, dep_ptr, b->grad, fwd, rev, b->coef, &h.slot_pref);
    h.coef0 = static_cast<uint32_t>(c0);
    h.coef1 = static_cast<uint32_t>(b->coef.size());
    h.f0 = static_cast<uint32_t>(b->steps.size());
    b->steps.insert(b->steps.end(), fwd.begin(), fwd.end());
    h.f1 = h.r0 = static_cast<uint32_t>(b->steps.size());
    b->steps.insert(b->steps.end(), rev.begin(), rev.end());
    h.r1 = static_cast<uint32_t>(b->steps.size());
    if (b->grad) {
        for (size_t idx = cmds.size(); idx-- > 0;)
            if (dep_ptr[idx + 1] > dep_ptr[idx]) h.slot_cmd.push_back(static_cast<int32_t>(idx));
        h.dep_ptr.assign(dep_ptr, dep_ptr + cmds.size() + 1);
        h.dep_param.assign(dep_param, dep_param + dep_ptr[cmds.size()]);
        h.dep_alpha.assign(dep_alpha, dep_alpha + dep_ptr[cmds.size()]);
    }
    h.slot0 = b->n_slots;
    b->n_slots += static_cast<uint32_t>(h.slot_cmd.size());
    h.t0 = static_cast<uint32_t>(b->tx.size());
    for (size_t g = 0; g < terms.gx.size(); ++g)
        for (int32_t t = terms.gstart[g]; t < terms.gstart[g + 1]; ++t) {
            b->tx.push_back(terms.gx[g]);
            b->tz.push_back(terms.z[t]);
            b->tc.push_back(terms.c[2 * t]);
            b->tc.push_back(terms.c[2 * t + 1]);
        }
    h.t1 = static_cast<uint32_t>(b->tx.size());
    b->inst.push_back(std::move(h));
    return static_cast<int>(b->inst.size()) - 1;
}

// new parameter values for instance idx: the same structure, so only its coefficients change
void cbatch_set(void* bp, int idx, const std::vector<Cmd>& cmds) {
    CircuitBatch* b = static_cast<CircuitBatch*>(bp);
    if (idx < 0 || idx >= static_cast<int>(b->inst.size())) throw std::invalid_argument("circuit batch: no such instance");
    CbInstHost& h = b->inst[static_cast<size_t>(idx)];
    std::vector<FsStep> fwd, rev;
    std::vector<double> coef;
    std::vector<c128> prefs;
    cb_encode(cmds, h.n, h.dep_ptr.empty() ? nullptr : h.dep_ptr.data(), b->grad && !h.dep_ptr.empty(), fwd, rev,
              coef, &prefs);
    if (coef.size() != h.coef1 - h.coef0 || fwd.size() != h.f1 - h.f0 || rev.size() != h.r1 - h.r0)
        throw std::invalid_argument("circuit batch: the new stream's structure differs from the instance's");
    for (size_t s = 0; s < fwd.size(); ++s)
        if (fwd[s].kind != b->steps[h.f0 + s].kind || fwd[s].coef + h.coef0 != b->steps[h.f0 + s].coef)
            throw std::invalid_argument("circuit batch: the new stream's structure differs from the instance's");
    std::copy(coef.begin(), coef.end(), b->coef.begin() + h.coef0);
    h.slot_pref = prefs;
    if (b->host_coef) std::copy(coef.begin(), coef.end(), b->host_coef + h.coef0);
}

namespace {

void cb_finalize(CircuitBatch* b) {
    check_cuda(cudaSetDevice(b->device), "cudaSetDevice");
    check_cuda(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking), "batch stream");
    check_cuda(cudaEventCreate(&b->e0), "event");
    check_cuda(cudaEventCreate(&b->e1), "event");
    // every step reads its coefficients from the batch-wide table (encode appended each
    // instance's to it, so the offsets are absolute already): check that every read stays in it
    for (const FsStep& f : b->steps)
        if (static_cast<size_t>(f.coef) + f.ncoef > b->coef.size() || f.ncoef > static_cast<uint32_t>(kFsMaxCoef))
            throw std::logic_error("circuit batch: a step's coefficients lie outside the table");
    for (const CbInstHost& h : b->inst)
        for (uint32_t t = h.t0; t < h.t1; ++t)
            if (t >= b->tx.size()) throw std::logic_error("circuit batch: a term lies outside the table");
    // by width class, costliest instances first: the queues' order
    auto width_class = [](int n) { return n >= kCbMaxQubits ? 0 : n >= kCbNarrow ? 1 : 2; };
    std::vector<size_t> order(b->inst.size());
    for (size_t i = 0; i < order.size(); ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](size_t a, size_t c) {
        const int ca = width_class(b->inst[a].n), cc = width_class(b->inst[c].n);
        if (ca != cc) return ca < cc;
        const double wa = std::ldexp(1.0, b->inst[a].n) * (b->inst[a].r1 - b->inst[a].f0 + b->inst[a].t1 - b->inst[a].t0);
        const double wc = std::ldexp(1.0, b->inst[c].n) * (b->inst[c].r1 - b->inst[c].f0 + b->inst[c].t1 - b->inst[c].t0);
        return wa > wc;
    });
    std::vector<CbInstDev> idev;
    for (size_t oi : order) {
        const CbInstHost& h = b->inst[oi];
        CbInstDev d{};
        d.n = h.n;
        d.pad = static_cast<int32_t>(oi);   // the caller's index: results are written there
        d.f0 = h.f0; d.f1 = h.f1; d.r0 = h.r0; d.r1 = h.r1; d.t0 = h.t0; d.t1 = h.t1;
        d.slot0 = h.slot0; d.nslot = static_cast<uint32_t>(h.slot_cmd.size());
        idev.push_back(d);
    }
    if (b->coef.empty()) b->coef.push_back(0.0);
    if (b->tx.empty()) { b->tx.push_back(0); b->tz.push_back(0); b->tc.push_back(0.0); b->tc.push_back(0.0); }
    auto align = [](size_t x) { return (x + 255) & ~size_t{255}; };
    const size_t n_inst = b->inst.size();
    b->off_inst = 0;
    b->off_steps = align(idev.size() * sizeof(CbInstDev));
    b->off_coef = b->off_steps + align(std::max<size_t>(b->steps.size(), 1) * sizeof(FsStep));
    b->off_tx = b->off_coef + align(b->coef.size() * sizeof(double));
    b->off_tz = b->off_tx + align(b->tx.size() * 8);
    b->off_tc = b->off_tz + align(b->tz.size() * 8);
    b->off_queue = b->off_tc + align(b->tc.size() * 8);
    b->off_energy = b->off_queue + 256;
    b->off_slots = b->off_energy + align(n_inst * 8);
    b->total = b->off_slots + align(std::max<uint32_t>(b->n_slots, 1) * 16);
    check_cuda(dev_malloc(&b->dev, b->total), "circuit batch buffers");
    check_cuda(cudaMallocHost(&b->host_coef, b->coef.size() * sizeof(double)), "pinned coefficients");
    check_cuda(cudaMallocHost(&b->host_out, (n_inst + 2 * std::max<uint32_t>(b->n_slots, 1)) * sizeof(double)),
               "pinned results");
    std::copy(b->coef.begin(), b->coef.end(), b->host_coef);
    auto up = [&](size_t off, const void* src, size_t bytes) {
        if (bytes) check_cuda(cudaMemcpyAsync(b->dev + off, src, bytes, cudaMemcpyHostToDevice, b->stream), "batch upload");
    };
    up(b->off_inst, idev.data(), idev.size() * sizeof(CbInstDev));
    up(b->off_steps, b->steps.data(), b->steps.size() * sizeof(FsStep));
    up(b->off_tx, b->tx.data(), b->tx.size() * 8);
    up(b->off_tz, b->tz.data(), b->tz.size() * 8);
    up(b->off_tc, b->tc.data(), b->tc.size() * 8);
    check_cuda(cudaStreamSynchronize(b->stream), "batch upload");
    int sms = 0;
    check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device), "sm count");
    // Three classes by width, a launch each, side by side: how many instances share a multiprocessor
    // is what their registers leave of its shared memory.
    struct Class { int sm_qubits; decltype(&k_cb_run<128>) kern; int threads; size_t i0, i1; unsigned grid; };
    Class cls[3] = {{kCbMaxQubits, k_cb_run<512>, 512, 0, 0, 0},
                    {kCbMaxQubits - 1, k_cb_run<256>, 256, 0, 0, 0},
                    {kCbNarrow - 1, k_cb_run<128>, 128, 0, 0, 0}};
    size_t at = 0;
    for (int k = 0; k < 3; ++k) {
        Class& c = cls[k];
        c.i0 = at;
        while (at < n_inst && width_class(idev[at].n) == k) ++at;
        c.i1 = at;
        if (c.i0 == c.i1) continue;
        const size_t smem = 2 * (size_t{1} << c.sm_qubits) * sizeof(double2);
        check_cuda(cudaFuncSetAttribute(c.kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
                   "batch smem");
        check_cuda(cudaFuncSetAttribute(c.kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                        cudaSharedmemCarveoutMaxShared), "batch carveout");
        int per_sm = 0;
        check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, c.kern, c.threads, smem), "occupancy");
        c.grid = static_cast<unsigned>(std::min<size_t>(c.i1 - c.i0, static_cast<size_t>(sms) * std::max(per_sm, 1)));
    }
    // the first class that has instances runs on the batch's own stream, each further one beside it
    int branches = 0;
    for (const Class& c : cls) branches += c.grid > 0;
    if (branches > 1) check_cuda(cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming), "event");
    for (int k = 0; k + 1 < branches; ++k) {
        check_cuda(cudaEventCreateWithFlags(&b->join[k], cudaEventDisableTiming), "event");
        check_cuda(cudaStreamCreateWithFlags(&b->side[k], cudaStreamNonBlocking), "batch stream");
    }
    b->wide_qubits = 0;
    for (const CbInstHost& h : b->inst)
        if (h.n > kCbMaxQubits) b->wide_qubits = std::max(b->wide_qubits, h.n);
    if (b->wide_qubits) {
        const size_t bytes = static_cast<size_t>(cls[0].grid) * (size_t{32} << b->wide_qubits);
        check_cuda(dev_malloc(&b->wide, bytes), "circuit batch wide registers");
    }
    // one graph: coefficients up, queue reset, the persistent kernel, results down
    check_cuda(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal), "batch capture");
    check_cuda(cudaMemcpyAsync(b->dev + b->off_coef, b->host_coef, b->coef.size() * sizeof(double),
                               cudaMemcpyHostToDevice, b->stream), "batch coefficients");
    check_cuda(cudaMemsetAsync(b->dev + b->off_queue, 0, 3 * sizeof(int), b->stream), "batch queue");
    if (branches > 1) check_cuda(cudaEventRecord(b->fork, b->stream), "batch fork");
    for (int c = 0, branch = 0; c < 3; ++c) {
        if (!cls[c].grid) continue;
        cudaStream_t on = branch == 0 ? b->stream : b->side[branch - 1];
        if (branch) check_cuda(cudaStreamWaitEvent(on, b->fork, 0), "batch fork");
        cls[c].kern<<<cls[c].grid, cls[c].threads, 2 * (size_t{1} << cls[c].sm_qubits) * sizeof(double2), on>>>(
            reinterpret_cast<const CbInstDev*>(b->dev + b->off_inst), static_cast<int>(cls[c].i0),
            static_cast<int>(cls[c].i1), reinterpret_cast<const FsStep*>(b->dev + b->off_steps),
            reinterpret_cast<const double*>(b->dev + b->off_coef),
            reinterpret_cast<const uint64_t*>(b->dev + b->off_tx), reinterpret_cast<const uint64_t*>(b->dev + b->off_tz),
            reinterpret_cast<const double2*>(b->dev + b->off_tc), b->grad ? 1 : 0,
            reinterpret_cast<int*>(b->dev + b->off_queue) + c, reinterpret_cast<double*>(b->dev + b->off_energy),
            reinterpret_cast<double2*>(b->dev + b->off_slots), b->wide, b->wide_qubits, cls[c].sm_qubits);
        check_cuda(cudaGetLastError(), "batch launch");
        if (branch) {
            check_cuda(cudaEventRecord(b->join[branch - 1], on), "batch join");
            check_cuda(cudaStreamWaitEvent(b->stream, b->join[branch - 1], 0), "batch join");
        }
        ++branch;
    }
    check_cuda(cudaMemcpyAsync(b->host_out, b->dev + b->off_energy, n_inst * sizeof(double), cudaMemcpyDeviceToHost,
                               b->stream), "batch energies");
    if (b->n_slots)
        check_cuda(cudaMemcpyAsync(b->host_out + n_inst, b->dev + b->off_slots, b->n_slots * 16,
                                   cudaMemcpyDeviceToHost, b->stream), "batch slots");
    check_cuda(cudaStreamEndCapture(b->stream, &b->graph), "batch capture");
    check_cuda(cudaGraphInstantiate(&b->exec, b->graph, 0), "batch graph");
}

}  // namespace

void cbatch_run(void* bp, double* energies, double* grads, double* device_ms) {
    CircuitBatch* b = static_cast<CircuitBatch*>(bp);
    if (b->inst.empty()) return;
    if (!b->exec) cb_finalize(b);
    check_cuda(cudaSetDevice(b->device), "cudaSetDevice");
    check_cuda(cudaEventRecord(b->e0, b->stream), "event");
    check_cuda(cudaGraphLaunch(b->exec, b->stream), "batch graph launch");
    check_cuda(cudaEventRecord(b->e1, b->stream), "event");
    check_cuda(cudaStreamSynchronize(b->stream), "circuit batch");
    if (device_ms) {
        float ms = 0;
        check_cuda(cudaEventElapsedTime(&ms, b->e0, b->e1), "event");
        *device_ms = ms;
    }
    const size_t n_inst = b->inst.size();
    // the kernel wrote results at the caller's instance index (CbInstDev::pad)
    if (energies) std::copy(b->host_out, b->host_out + n_inst, energies);
    if (grads && b->grad) {
        size_t g0 = 0;
        for (const CbInstHost& h : b->inst) {
            for (int p = 0; p < h.n_params; ++p) grads[g0 + static_cast<size_t>(p)] = 0.0;
            for (size_t s = 0; s < h.slot_cmd.size(); ++s) {
                const double* ipd = b->host_out + n_inst + 2 * (h.slot0 + s);
                const c128 ip(ipd[0], ipd[1]);
                const double base = 2.0 * std::real(h.slot_pref[s] * ip);
                const int32_t i = h.slot_cmd[s];
                for (int32_t d = h.dep_ptr[i]; d < h.dep_ptr[i + 1]; ++d)
                    grads[g0 + static_cast<size_t>(h.dep_param[d])] += h.dep_alpha[d] * base;
            }
            g0 += static_cast<size_t>(h.n_params);
        }
    }
}

void cbatch_destroy(void* bp) { delete static_cast<CircuitBatch*>(bp); }

}  // namespace qsv
