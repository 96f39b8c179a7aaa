// kern_pauli.cu — <psi|H|psi> of a Pauli sum with real coefficients over one register.
//
// Reference counterpart: pauli_transition with bra == ket
// (src/qarpx/src/simulator/pauli_expectation.cpp:34-167).
//
// A term's X mask x pairs the amplitudes i and i ^ x, and the two contributions of a pair are
// complex conjugates, so each pair is formed once: q = conj(psi[i ^ x]) psi[i], of which a term
// with an even number of Ys takes Re q and one with an odd number Im q, times 2 and its signs.
//
// The register is read in tiles of 2^12 amplitudes (any 12 qubits that include 0..2), a tile's
// amplitudes in the registers of 256 threads (16 each) and once more in shared memory.  A group
// of terms whose x lies inside the tile's qubits finds every partner there: the one-kernel form
// read each partner from L2 instead (10 TB/s of L2 reads at 26 qubits, its bound).  The host
// covers the groups with passes, a tile choice each (cover_groups): 551 terms of weight <= 4 over
// 26 qubits take 14 passes, one register read each.  Groups no pass is worth reading the
// register for go to one last pass that fetches partners from global memory.
//
// The 16 amplitudes of a thread differ in the four slot qubits.  Where x contains a slot qubit the
// pairs are (slot bit 0, its partner): 8 shared-memory reads for the thread's 8 pairs, no lane
// idle.  Otherwise a warp qubit of x switches half the warps off, and an x on lane qubits alone
// visits each pair from both ends at half weight.  The signs of the 8 pairs follow from the term's
// Z bits on the three other slot qubits (its class, one of 8 sign patterns compiled in): a term costs a
// popcount and an addition, a class seven additions for 8 pairs.
//
// 26 qubits, 551 terms in 254 groups: 12.7 ms; 26.8 ms in the one-kernel form, which still serves
// transitions between two registers and complex coefficients.  Bound: issue slots (header, class and
// sign work around 8 reads and 16 FMAs a group) with 16 warps an SM; the amplitudes take the registers.
#include <algorithm>
#include <cstring>
#include <vector>

#include "kernels.h"

namespace qsv {

namespace {

constexpr int kPThreads = 256;
constexpr int kPTile = 12;
constexpr int kPLow = 3;       // qubits 0..2 in every tile: 128-byte (complex64: 64-byte) runs
constexpr int kPCover = 4;     // a shared-memory pass takes at least this many groups: it costs a
                               // read of the register, about what 3 groups cost from global memory
constexpr int kPCtas = 2;      // CTAs per SM (128 registers a thread, 64 KiB)

// The terms of one X mask that take Re q, or those that take Im q (a thread that held both products
// would spill).
struct __align__(16) PairGroup {
    uint32_t code;             // bits 0..11: x on the tile's local bits (shared-memory passes); 12..15: variant
                               // (0..3 pairs across that slot bit, 3 also slots 0..7, 4 slots 8..15, + 5 for Im q);
                               // 16: transform; 24..31: threads with one of these bits have no pair
    int32_t t0, t1, pad;       // its terms
};
struct PairOutside {
    uint64_t x;                // the whole X mask (global passes)
    uint64_t skip_tile;        // tiles with this index bit have no pair
};
// A term, ordered by class within its group.
struct __align__(16) PairTerm {
    double c;
    uint32_t zt;               // Z bits on thread bits
    uint32_t cls;              // Z bits on the variant's slot bits, | kRunEnd on the last of a class
};
constexpr int kMaxGroups = 384, kMaxTerms = 1024;   // of one launch: they lie in shared memory
constexpr uint32_t kRunEnd = 8;
constexpr int kTransformRuns = 4;   // from this many classes an 8-point transform (24 additions) gives
                                    // every class sum; below, 7 additions a class
struct PairTable {                  // one launch's part of the uploaded tables
    const PairGroup* group;
    const PairOutside* outside;
    const PairTerm* term;
    const uint64_t* zo;             // per term: Z bits outside the tile
    int32_t n_groups, n_terms;
};
struct PairPass {
    uint8_t slot_q[4];         // qubits of the slot bits
    uint8_t tid_q[8];          // qubits of the thread bits (lanes, then warps)
    uint8_t sorted[kPTile];    // the tile's qubits, ascending
};

__device__ __forceinline__ double2 wide(double2 v) { return v; }
__device__ __forceinline__ double2 wide(float2 v) { return make_double2(v.x, v.y); }

template <int K>
__device__ __forceinline__ double class_sum(const double (&q)[8]) {
    constexpr bool s0 = K & 1, s1 = K & 2, s2 = K & 4;
    const double a = s0 ? q[0] - q[1] : q[0] + q[1], b = s0 ? q[2] - q[3] : q[2] + q[3];
    const double c = s0 ? q[4] - q[5] : q[4] + q[5], d = s0 ? q[6] - q[7] : q[6] + q[7];
    const double e = s1 ? a - b : a + b, f = s1 ? c - d : c + d;
    return s2 ? e - f : e + f;
}

// e + the terms [j, end) of one group: their coefficients (the tile's sign already on them), signed for
// this thread, summed by class, times the class sums of q.  A term is read while the one before it is
// summed (the table ends in a spare entry).
__device__ __forceinline__ double term_sums(const PairTerm* term, int j, int end, bool wht, double (&q)[8], uint32_t tid,
                                            double e) {
    if (wht) {
#pragma unroll
        for (int h = 1; h < 8; h <<= 1)
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (!(k & h)) {
                    const double x = q[k], y = q[k | h];
                    q[k] = x + y;
                    q[k | h] = x - y;
                }
    }
    int4 t = *reinterpret_cast<const int4*>(term + j);
    while (j < end) {
        double w = 0.0;
        uint32_t cls;
        do {
            const int4 now = t;
            ++j;
            t = *reinterpret_cast<const int4*>(term + j);
            cls = static_cast<uint32_t>(now.w);
            w += __hiloint2double(now.y ^ (__popc(static_cast<uint32_t>(now.z) & tid) << 31), now.x);
        } while (!(cls & kRunEnd));
        double s;
        if (wht) {
            switch (cls & 7u) {
                case 0: s = q[0]; break;
                case 1: s = q[1]; break;
                case 2: s = q[2]; break;
                case 3: s = q[3]; break;
                case 4: s = q[4]; break;
                case 5: s = q[5]; break;
                case 6: s = q[6]; break;
                default: s = q[7]; break;
            }
        } else {
            switch (cls & 7u) {
                case 0: s = class_sum<0>(q); break;
                case 1: s = class_sum<1>(q); break;
                case 2: s = class_sum<2>(q); break;
                case 3: s = class_sum<3>(q); break;
                case 4: s = class_sum<4>(q); break;
                case 5: s = class_sum<5>(q); break;
                case 6: s = class_sum<6>(q); break;
                default: s = class_sum<7>(q); break;
            }
        }
        e = fma(w, s, e);
    }
    return e;
}

// q[m] = Re or Im of conj(partner) own for the variant's 8 slots
template <int V, bool IM, typename T, typename Fetch>
__device__ __forceinline__ void pair_products(const vec2_t<T> (&v)[16], Fetch fetch, double (&q)[8]) {
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        constexpr int b = V < 4 ? V : 3;
        const int s = (((m >> b) << (b + 1)) | (m & ((1 << b) - 1))) | (V == 4 ? 8 : 0);
        const double2 o = wide(v[s]), w = wide(fetch(s));
        q[m] = IM ? fma(w.x, o.y, -(w.y * o.x)) : fma(w.x, o.x, w.y * o.y);
    }
}

template <typename T, bool GLOBAL>
__global__ void __launch_bounds__(kPThreads, kPCtas)
    k_pauli_pairs(const vec2_t<T>* __restrict__ psi, const __grid_constant__ PairPass pass, uint64_t n_tiles,
                  PairTable tab, double* __restrict__ partials) {
    extern __shared__ __align__(16) unsigned char psm[];
    PairGroup* group_s = reinterpret_cast<PairGroup*>(psm);
    PairTerm* term_s = reinterpret_cast<PairTerm*>(group_s + tab.n_groups);
    uint64_t* zo_s = reinterpret_cast<uint64_t*>(term_s + tab.n_terms + 1);
    vec2_t<T>* tile_s = reinterpret_cast<vec2_t<T>*>(zo_s + ((tab.n_terms + 1) & ~1));
    __shared__ double red[kPThreads / 32];
    const uint32_t tid = threadIdx.x;
    uint64_t toff = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) toff |= static_cast<uint64_t>((tid >> k) & 1u) << pass.tid_q[k];
    auto slot_off = [&](int s) {
        uint64_t o = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if ((s >> k) & 1) o |= 1ull << pass.slot_q[k];
        return o;
    };
    for (int g = tid; g < tab.n_groups; g += kPThreads) group_s[g] = *QSV_DBG(tab.group + g);
    for (int j = tid; j < tab.n_terms; j += kPThreads) {
        term_s[j] = *QSV_DBG(tab.term + j);
        zo_s[j] = *QSV_DBG(tab.zo + j);
    }
    if (tid == 0) term_s[tab.n_terms] = PairTerm{};
    uint64_t signed_for = 0;     // the tile whose signs the coefficients carry
    double e = 0.0;
    for (uint64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        uint64_t tb = tile;
#pragma unroll
        for (int k = 0; k < kPTile; ++k) {
            const uint64_t low = tb & ((1ull << pass.sorted[k]) - 1ull);
            tb = ((tb ^ low) << 1) | low;
        }
        const vec2_t<T>* src = psi + (tb | toff);
        vec2_t<T> v[16];
#pragma unroll
        for (int s = 0; s < 16; ++s) v[s] = *QSV_DBG(src + slot_off(s));
        __syncthreads();     // the previous tile's readers are done
        if (!GLOBAL) {
#pragma unroll
            for (int s = 0; s < 16; ++s) tile_s[tid | (s << 8)] = v[s];
        }
        for (int j = tid; j < tab.n_terms; j += kPThreads)
            if (__popcll(zo_s[j] & (tb ^ signed_for)) & 1) term_s[j].c = -term_s[j].c;
        signed_for = tb;
        __syncthreads();
        for (int g = blockIdx.y; g < tab.n_groups; g += gridDim.y) {
            const int4 gr = *reinterpret_cast<const int4*>(group_s + g);
            const uint32_t code = static_cast<uint32_t>(gr.x);
            if (tid & (code >> 24)) continue;      // whole warps: a warp bit
            uint64_t from = 0;
            if (GLOBAL) {
                const PairOutside* po = QSV_DBG(tab.outside + g);
                if (tb & __ldg(&po->skip_tile)) continue;
                from = (tb | toff) ^ __ldg(&po->x);
            }
            double q[8];
            const uint32_t at = tid ^ (code & 0xfffu);
            auto fetch = [&](int s) -> vec2_t<T> {
                if (GLOBAL) return *QSV_DBG(psi + (from ^ slot_off(s)));
                return tile_s[at ^ (static_cast<uint32_t>(s) << 8)];
            };
            switch ((code >> 12) & 15u) {
                case 0: pair_products<0, false, T>(v, fetch, q); break;
                case 1: pair_products<1, false, T>(v, fetch, q); break;
                case 2: pair_products<2, false, T>(v, fetch, q); break;
                case 3: pair_products<3, false, T>(v, fetch, q); break;
                case 4: pair_products<4, false, T>(v, fetch, q); break;
                case 5: pair_products<0, true, T>(v, fetch, q); break;
                case 6: pair_products<1, true, T>(v, fetch, q); break;
                case 7: pair_products<2, true, T>(v, fetch, q); break;
                case 8: pair_products<3, true, T>(v, fetch, q); break;
                default: pair_products<4, true, T>(v, fetch, q); break;
            }
            e = term_sums(term_s, gr.y, gr.z, code & 0x10000u, q, tid, e);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if ((tid & 31u) == 0) red[tid >> 5] = e;
    __syncthreads();
    if (tid == 0) {
        double sum = 0.0;
#pragma unroll
        for (int w = 0; w < kPThreads / 32; ++w) sum += red[w];
        *QSV_DBG(partials + (static_cast<uint64_t>(blockIdx.y) * gridDim.x + blockIdx.x)) = sum;
    }
}

// sum of all partials, one block, fixed order
__global__ void __launch_bounds__(1024) k_pauli_final(const double* __restrict__ partials, unsigned n, double* __restrict__ out) {
    __shared__ double red[32];
    double a = 0.0;
    for (unsigned i = threadIdx.x; i < n; i += blockDim.x) a += *QSV_DBG(partials + i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < 32; ++w) s += red[w];
        *QSV_DBG(out) = s;
    }
}

int popc(uint64_t v) { return __builtin_popcountll(v); }

struct Cover {
    uint64_t tile = 0;            // the pass's tile qubits
    bool global = false;
    std::vector<int> groups;
};

// Tile choices that cover the groups' X masks.  Each tile starts at qubits 0..2 and takes in, again
// and again, the group that needs the fewest further qubits (of those the widest, first in order);
// what the last qubits are is free.  A tile that covers fewer than kPCover groups ends the list and
// the groups left go to one pass that reads partners from global memory.
std::vector<Cover> cover_groups(const std::vector<uint64_t>& gx, int n, bool shared) {
    std::vector<Cover> out;
    std::vector<int> rem(gx.size());
    for (size_t i = 0; i < rem.size(); ++i) rem[i] = static_cast<int>(i);
    auto fill = [&](uint64_t t) {
        for (int q = 0; q < n && popc(t) < kPTile; ++q) t |= 1ull << q;
        return t;
    };
    while (shared && !rem.empty()) {
        uint64_t t = (1ull << kPLow) - 1;
        while (popc(t) < kPTile) {
            int best = -1, need = 64, width = -1;
            for (int i : rem) {
                const int k = popc(gx[i] & ~t);
                if (k == 0 || k > need) continue;
                const int w = popc(gx[i]);
                if (k < need || w > width) best = i, need = k, width = w;
            }
            if (best < 0 || popc(t) + need > kPTile) break;
            t |= gx[best];
        }
        Cover c;
        c.tile = fill(t);
        std::vector<int> left;
        for (int i : rem) ((gx[i] & ~c.tile) ? left : c.groups).push_back(i);
        if (static_cast<int>(c.groups.size()) < kPCover && n > kPTile) break;
        out.push_back(std::move(c));
        rem.swap(left);
    }
    if (!rem.empty()) {
        // slot qubits where the masks have most bits; the other tile qubits are the lowest
        Cover c;
        c.global = true;
        c.groups = rem;
        uint64_t slots = 0;
        std::vector<int> open = rem;
        for (int s = 0; s < 4; ++s) {
            int best = -1, most = -1;
            for (int q = n - 1; q >= 5; --q) {
                if ((slots >> q) & 1) continue;
                int k = 0;
                for (int i : open) k += static_cast<int>((gx[i] >> q) & 1);
                if (k > most) most = k, best = q;
            }
            slots |= 1ull << best;
            std::vector<int> rest;
            for (int i : open)
                if (!((gx[i] >> best) & 1)) rest.push_back(i);
            open.swap(rest);
        }
        c.tile = fill(slots);
        out.push_back(std::move(c));
    }
    return out;
}

}  // namespace

// From 12 qubits up, psi against itself, every coefficient real: true with the energy in *out.
template <typename T>
bool pauli_energy(const vec2_t<T>* psi, int n, const PauliTerms& terms, cudaStream_t st, Workspace& ws, double* out) {
    if (n < kPTile || n > 63) return false;
    const int n_groups = static_cast<int>(terms.gx.size());
    for (int g = 0; g < n_groups; ++g)
        for (int j = terms.gstart[g]; j < terms.gstart[g + 1]; ++j)
            if (terms.c[2 * j + (popc(terms.gx[g] & terms.z[j]) & 1 ? 0 : 1)] != 0.0) return false;
    const uint64_t n_tiles = 1ull << (n - kPTile);
    int dev = 0;
    check_cuda(cudaGetDevice(&dev), "device");
    int sms = 0;
    check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "sm count");
    const uint64_t slots = static_cast<uint64_t>(sms) * kPCtas;
    // Up to 21 qubits the register sits in L2 (32 MiB) and one pass reading every partner from there is
    // the faster: 21 qubits, 541 terms 709 us against 736 us in shared-memory passes; 22 qubits 1273
    // against 1083 us.
    constexpr int kPSharedQubits = 22;
    const std::vector<Cover> covers = cover_groups(terms.gx, n, n == kPTile || n >= kPSharedQubits);
    std::vector<PairGroup> hg;
    std::vector<PairOutside> ho;
    std::vector<PairTerm> ht;
    std::vector<uint64_t> hz;
    struct Launch {
        PairPass pass{};
        bool global = false;
        unsigned gx = 1, gy = 1;
        int n_groups = 0, n_terms = 0;
        size_t g0 = 0, t0 = 0;      // first entries in the tables
    };
    std::vector<Launch> launches;
    for (const Cover& c : covers) {
        PairPass pass{};
        // thread bits 0..2 are qubits 0..2; slots, then warps, go where they split most groups' pairs
        std::vector<int> q, tile;
        for (int b = 0; b < n; ++b)
            if ((c.tile >> b) & 1) tile.push_back(b);
        for (int k = 0; k < kPTile; ++k) pass.sorted[k] = static_cast<uint8_t>(tile[k]);
        std::vector<int> order;      // slots 0..3, then warps 0..2
        uint64_t used = (1ull << kPLow) - 1;
        if (c.global)
            for (int b = 0; b < 5; ++b) used |= 1ull << b;     // whole lanes of consecutive amplitudes
        std::vector<int> open = c.groups;
        for (int s = 0; s < 7; ++s) {
            int best = -1, most = -1;
            for (int b : tile) {
                if ((used >> b) & 1) continue;
                int k = 0;
                for (int i : open) k += static_cast<int>((terms.gx[i] >> b) & 1);
                if (k > most) most = k, best = b;
            }
            order.push_back(best);
            used |= 1ull << best;
            std::vector<int> rest;
            for (int i : open)
                if (!((terms.gx[i] >> best) & 1)) rest.push_back(i);
            open.swap(rest);
        }
        for (int s = 0; s < 4; ++s) pass.slot_q[s] = static_cast<uint8_t>(order[s]);
        int lane = 0;
        for (int b : tile)
            if (std::find(order.begin(), order.end(), b) == order.end()) pass.tid_q[lane++] = static_cast<uint8_t>(b);
        for (int w = 0; w < 3; ++w) pass.tid_q[5 + w] = static_cast<uint8_t>(order[4 + w]);
        auto open_launch = [&] {
            launches.emplace_back();
            launches.back().pass = pass;
            launches.back().global = c.global;
            launches.back().g0 = hg.size();
            launches.back().t0 = ht.size();
        };
        open_launch();
        struct Term {
            PairTerm t;
            uint64_t zo;
        };
        // one group, its pairs formed by `variant`; terms beyond a launch's table go to the next one
        auto emit = [&](int gi, uint32_t variant, double weight, uint32_t skip_tid, uint64_t skip_tile) {
            const uint64_t x = terms.gx[gi];
            uint32_t code = variant << 12 | skip_tid << 24;
            for (int k = 0; k < 8; ++k) code |= static_cast<uint32_t>((x >> pass.tid_q[k]) & 1) << k;
            for (int k = 0; k < 4; ++k) code |= static_cast<uint32_t>((x >> pass.slot_q[k]) & 1) << (8 + k);
            const int sel = variant < 4 ? static_cast<int>(variant) : 3;
            std::vector<Term> part[2];
            for (int j = terms.gstart[gi]; j < terms.gstart[gi + 1]; ++j) {
                const uint64_t z = terms.z[j];
                const int odd = popc(x & z) & 1;
                Term t{};
                for (int k = 0; k < 8; ++k) t.t.zt |= static_cast<uint32_t>((z >> pass.tid_q[k]) & 1) << k;
                int at = 0;
                for (int k = 0; k < 4; ++k)
                    if (k != sel) t.t.cls |= static_cast<uint32_t>((z >> pass.slot_q[k]) & 1) << at++;
                t.zo = z & ~c.tile;
                // Re((cr + i ci) q) = cr Re q - ci Im q
                t.t.c = weight * (odd ? -terms.c[2 * j + 1] : terms.c[2 * j]);
                if (variant == 4 && ((z >> pass.slot_q[3]) & 1)) t.t.c = -t.t.c;
                part[odd].push_back(t);
            }
            for (auto& p : part)
                std::stable_sort(p.begin(), p.end(), [](const Term& a, const Term& b) { return a.t.cls < b.t.cls; });
            for (int odd = 0; odd < 2; ++odd)
                for (size_t done = 0; done < part[odd].size();) {
                    if (launches.back().n_groups == kMaxGroups || launches.back().n_terms == kMaxTerms) open_launch();
                    Launch& l = launches.back();
                    PairGroup pg{};
                    pg.code = code + (odd ? 5u << 12 : 0u);
                    pg.t0 = l.n_terms;
                    const size_t stop = std::min(part[odd].size(), done + static_cast<size_t>(kMaxTerms - l.n_terms));
                    int runs = 0;
                    for (; done < stop; ++done) {
                        Term t = part[odd][done];
                        const bool end = done + 1 == stop || part[odd][done + 1].t.cls != t.t.cls;
                        runs += end;
                        if (end) t.t.cls |= kRunEnd;
                        ht.push_back(t.t);
                        hz.push_back(t.zo);
                        ++l.n_terms;
                    }
                    if (runs >= kTransformRuns) pg.code |= 0x10000u;
                    pg.t1 = l.n_terms;
                    hg.push_back(pg);
                    ho.push_back(PairOutside{x, skip_tile});
                    ++l.n_groups;
                }
        };
        for (int gi : c.groups) {
            const uint64_t x = terms.gx[gi];
            int slot = -1, warp = -1;
            for (int k = 0; k < 4 && slot < 0; ++k)
                if ((x >> pass.slot_q[k]) & 1) slot = k;
            for (int k = 5; k < 8 && warp < 0; ++k)
                if ((x >> pass.tid_q[k]) & 1) warp = k;
            if (slot >= 0) {
                emit(gi, static_cast<uint32_t>(slot), 2.0, 0, 0);
            } else {
                // pairs visited from one end (a warp or tile bit of x), or from both at half weight
                const uint64_t outside = x & ~c.tile;
                const uint32_t st_ = warp >= 0 ? 1u << warp : 0;
                const uint64_t so = warp < 0 && outside ? outside & (~outside + 1) : 0;
                const double w = st_ || so ? 2.0 : 1.0;
                emit(gi, 3, w, st_, so);
                emit(gi, 4, w, st_, so);
            }
        }
    }
    // few tiles: several CTAs share one, each with its part of the groups
    const uint64_t want = 4 * slots;
    uint64_t n_part = 0;
    for (Launch& l : launches) {
        l.gx = static_cast<unsigned>(n_tiles >= want ? slots : n_tiles);
        // each CTA that shares a tile reads it: where the tiles alone fill the chip, a part is worth that
        // from kPCover groups (22 qubits, one term: 56.6 -> 44.9 us; 50 with a kernel per amplitude)
        const uint64_t most = n_tiles >= slots ? (l.n_groups + kPCover - 1) / kPCover : l.n_groups;
        l.gy = n_tiles >= want ? 1u
                               : static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>((want + n_tiles - 1) / n_tiles, most)));
        n_part += static_cast<uint64_t>(l.gx) * l.gy;
    }
    std::vector<uint8_t> host;
    auto put = [&](const void* src, size_t bytes) {
        const size_t at = host.size();
        host.resize((at + bytes + 15) & ~size_t{15});
        std::memcpy(host.data() + at, src, bytes);
        return at;
    };
    const size_t at_g = put(hg.data(), hg.size() * sizeof(PairGroup)), at_o = put(ho.data(), ho.size() * sizeof(PairOutside));
    const size_t at_t = put(ht.data(), ht.size() * sizeof(PairTerm)), at_z = put(hz.data(), hz.size() * sizeof(uint64_t));
    uint8_t* dev_tab = static_cast<uint8_t*>(ws.matrix(host.size()));
    // pageable source: the call returns once it is staged
    check_cuda(cudaMemcpyAsync(dev_tab, host.data(), host.size(), cudaMemcpyHostToDevice, st), "term upload");
    double* partials = static_cast<double*>(ws.scratch((n_part + 1) * sizeof(double)));
    auto table_bytes = [](int groups, int n_terms) {
        return static_cast<size_t>(groups) * sizeof(PairGroup) + (static_cast<size_t>(n_terms) + 1) * sizeof(PairTerm) +
               static_cast<size_t>((n_terms + 1) & ~1) * sizeof(uint64_t);
    };
    const size_t tile_bytes = sizeof(vec2_t<T>) << kPTile;
    check_cuda(cudaFuncSetAttribute(k_pauli_pairs<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(tile_bytes + table_bytes(kMaxGroups, kMaxTerms))), "shared memory");
    uint64_t at = 0;
    for (const Launch& l : launches) {
        const dim3 grid(l.gx, l.gy);
        const size_t smem = table_bytes(l.n_groups, l.n_terms) + (l.global ? 0 : tile_bytes);
        PairTable tab{reinterpret_cast<const PairGroup*>(dev_tab + at_g) + l.g0, reinterpret_cast<const PairOutside*>(dev_tab + at_o) + l.g0,
                      reinterpret_cast<const PairTerm*>(dev_tab + at_t) + l.t0, reinterpret_cast<const uint64_t*>(dev_tab + at_z) + l.t0,
                      l.n_groups, l.n_terms};
        if (l.global) k_pauli_pairs<T, true><<<grid, kPThreads, smem, st>>>(psi, l.pass, n_tiles, tab, partials + at);
        else k_pauli_pairs<T, false><<<grid, kPThreads, smem, st>>>(psi, l.pass, n_tiles, tab, partials + at);
        at += static_cast<uint64_t>(l.gx) * l.gy;
    }
    k_pauli_final<<<1, 1024, 0, st>>>(partials, static_cast<unsigned>(n_part), partials + n_part);
    check_cuda(cudaGetLastError(), "energy launch");
    double* h = ws.host_result(2);
    check_cuda(cudaMemcpyAsync(h, partials + n_part, sizeof(double), cudaMemcpyDeviceToHost, st), "result copy");
    check_cuda(cudaStreamSynchronize(st), "energy");
    *out = h[0];
    return true;
}

template bool pauli_energy<double>(const double2*, int, const PauliTerms&, cudaStream_t, Workspace&, double*);
template bool pauli_energy<float>(const float2*, int, const PauliTerms&, cudaStream_t, Workspace&, double*);

}  // namespace qsv
