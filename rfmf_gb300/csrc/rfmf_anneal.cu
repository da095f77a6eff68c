// rfmf_anneal.cu -- the RFMF sweep kernel for GB300 (sm_103a).
//
// Method (gt-tinker/rfmf, src/anneal_kernels.cu:262-491): per sweep, every
// vertex v draws a Q20 Gumbel key from Philox4x32-10 (key = chain seed,
// counter = (sweep, v>>3)), scores gum + beta*delta(v) with delta(v) the exact
// cut gain of flipping v, and the best score of each group g = v mod P (ties
// to the smallest v) wins; the P winners then flip, exactly as if flipped one
// after another in group order.
//
// GB300 design (not the reference's):
//   * A persistent CTA takes work items of up to K chains of ONE graph.  The
//     graph's CSR is staged once per item into shared memory by bulk async
//     copies (cp.async.bulk + mbarrier) in a compact format (2 bytes per entry
//     for +-1 weights), and K warp groups (W warps each) run K chains side by
//     side on that one copy.  Chains never synchronise with each other: a
//     chain's barriers are __syncwarp (W == 1) or a named barrier of its own.
//   * All mutable chain state stays in shared memory for the whole window:
//     D[v] = spin[v]*S[v] (the per-vertex gain; as an int8 field S with a
//     bias that one xor with the spin mask turns into D when the max weighted
//     degree B <= 127, else int32 D), the spins as mask bytes and bits, and
//     the best-so-far spins as bits.  Graphs too big for shared memory walk
//     their CSR in HBM instead, in the most compact entry form they allow
//     (2, 4 or 8 bytes); the chain state stays resident.
//   * SELECT reads only D.  The sweep-uniform part of the Philox counter is
//     hoisted (rounds 1-3 lose 3 multiplies and 3 xors per block) and three
//     vertex blocks are in flight per thread.
//   * The group argmax keeps eight register accumulators per thread (one per
//     Philox lane j), the block stride chosen so that each lands in one group.
//     For P <= 128 each warp passes its 256 accumulators through shared memory
//     and reduces them without atomics; the winners stay in registers (one-warp
//     chains) or pass through one partial per warp and group.  Larger P, int64
//     scores, strides that a chain's threads do not reach, and chains with no
//     room for the scratch go through shared-memory slots with atomics.
//   * FLIP has no winner-winner correction walk.  With D kept per vertex,
//     negating the winners' D and scattering 2*w*s_b*s_x into D[x] over the
//     winners' rows leaves every winner holding D_final, and the cut gain of
//     the whole flip set is exactly (sum delta_pre - sum D_final) / 2: the
//     same integer the reference's corr[] formulation (src/anneal_kernels.cu:
//     133-192, 420-440) adds up.  Compact rows are walked as vectors of four
//     entries, 8-byte pairs four loads at a time.
#include <cuda_runtime.h>

#include <climits>
#include <cstdint>
#include <type_traits>

#include "rfmf_device.h"

// Gain bytes this translation unit compiles the kernels for (each leaves the
// other width's helpers unreferenced).
#ifndef RFMF_GAIN_BYTES
#define RFMF_GAIN_BYTES 1
#endif
#pragma nv_diag_suppress 177

namespace rfmf {

namespace {

// Published Philox4x32 constants (Salmon et al. 2011).
constexpr uint32_t kM0 = 0xD2511F53u;
constexpr uint32_t kM1 = 0xCD9E8D57u;
constexpr uint32_t kW0 = 0x9E3779B9u;
constexpr uint32_t kW1 = 0xBB67AE85u;

// Bound on mbarrier polls while a CSR bulk copy lands (each poll may suspend
// the thread for a hardware-chosen interval); past it the CTA stops taking
// work and the launch reports kDevCopyTimeout.
constexpr int kMaxCopyPolls = 1 << 22;

// max |Gumbel key| (Q20 table plus the field's upper bits).
constexpr int64_t kGumMaxMag = 3617486 + 127;

__device__ __forceinline__ void mulwide(uint32_t a, uint32_t b, uint32_t& hi, uint32_t& lo) {
    const uint64_t p = static_cast<uint64_t>(a) * b;
    hi = static_cast<uint32_t>(p >> 32);
    lo = static_cast<uint32_t>(p);
}

// Philox round keys, k0[r] = seed_lo + r*W0, k1[r] = seed_hi + r*W1.
struct ChainKeys {
    uint32_t k0[10];
    uint32_t k1[10];
};

// A value that is the same in every lane of the (converged) warp, as one the
// compiler knows to be uniform: redux.sync delivers to a uniform register,
// where a chain's constants cost no per-thread registers.
__device__ __forceinline__ uint32_t uniform(uint32_t x) { return __reduce_or_sync(0xFFFFFFFFu, x); }
__device__ __forceinline__ int32_t uniform(int32_t x) { return static_cast<int32_t>(uniform(static_cast<uint32_t>(x))); }
__device__ __forceinline__ uint64_t uniform(uint64_t x) {
    return (static_cast<uint64_t>(uniform(static_cast<uint32_t>(x >> 32))) << 32) | uniform(static_cast<uint32_t>(x));
}
__device__ __forceinline__ int64_t uniform(int64_t x) { return static_cast<int64_t>(uniform(static_cast<uint64_t>(x))); }
template <class T>
__device__ __forceinline__ T* uniform(T* x) { return reinterpret_cast<T*>(uniform(reinterpret_cast<uint64_t>(x))); }
__device__ __forceinline__ ChainKeys make_keys(uint64_t seed) {
    ChainKeys k;
    uint32_t a = uniform(static_cast<uint32_t>(seed)), b = uniform(static_cast<uint32_t>(seed >> 32));
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        k.k0[r] = a;
        k.k1[r] = b;
        a += kW0;
        b += kW1;
    }
    return k;
}

// Per-sweep constants.  The Philox counter is (step_lo, step_hi, b, 0): words
// 0, 1 and 3 are the same for every vertex block of a sweep.
struct SweepConst {
    uint32_t A;   // round-1 xor for word 0:  step_hi ^ k0[0]
    uint32_t Cc;  // round-2 xor for word 0:  hi(M1 * w2_r1) ^ k0[1]
    uint32_t Dc;  // round-2 xor for word 2:  lo(M0 * step_lo) ^ k1[1]
    uint32_t E;   // round-3 xor for word 0:  lo(M1 * w2_r1) ^ k0[2]
};

__device__ __forceinline__ SweepConst make_sweep(uint64_t step, const ChainKeys& k) {
    const uint32_t slo = static_cast<uint32_t>(step);
    const uint32_t shi = static_cast<uint32_t>(step >> 32);
    uint32_t hi0, lo0;
    mulwide(kM0, slo, hi0, lo0);
    const uint32_t w2r1 = hi0 ^ k.k1[0];   // counter word 3 (block >> 32) is 0
    uint32_t hi1, lo1;
    mulwide(kM1, w2r1, hi1, lo1);
    SweepConst c;
    c.A = shi ^ k.k0[0];
    c.Cc = hi1 ^ k.k0[1];
    c.Dc = lo0 ^ k.k1[1];
    c.E = lo1 ^ k.k0[2];
    return c;
}

// Philox4x32-10 of counter (step, b, 0) under the chain key; bit-identical to
// philox4x32_10(gumbelBlockCounter(step, b), key) of src/philox.cuh:77-119.
__device__ __forceinline__ void philox_block(uint32_t b, const SweepConst& c,
                                             const ChainKeys& k, uint32_t x[4]) {
    uint32_t hi, lo;
    mulwide(kM1, b, hi, lo);                  // round 1
    uint32_t v0 = hi ^ c.A;
    uint32_t v1 = lo;
    mulwide(kM0, v0, hi, lo);                 // round 2
    v0 = v1 ^ c.Cc;
    uint32_t v2 = hi ^ c.Dc;
    uint32_t v3 = lo;
    uint32_t h0, l0, h1, l1;
    mulwide(kM0, v0, h0, l0);                 // round 3
    mulwide(kM1, v2, h1, l1);
    v0 = h1 ^ c.E;
    v1 = l1;
    v2 = h0 ^ v3 ^ k.k1[2];
    v3 = l0;
#pragma unroll
    for (int r = 3; r < 10; ++r) {            // rounds 4..10
        mulwide(kM0, v0, h0, l0);
        mulwide(kM1, v2, h1, l1);
        v0 = h1 ^ v1 ^ k.k0[r];
        v1 = l1;
        v2 = h0 ^ v3 ^ k.k1[r];
        v3 = l0;
    }
    x[0] = v0;
    x[1] = v1;
    x[2] = v2;
    x[3] = v3;
}

// 11-bit field of lane j (src/philox.cuh:121-126).
__device__ __forceinline__ uint32_t field(const uint32_t x[4], int j) {
    return ((j & 1) ? (x[j >> 1] >> 16) : x[j >> 1]) & 0x7FFu;
}

// Packed argmax key [biased score : 32 | ~v : 32]: unsigned order = score
// order, ties to the smaller v; 0 is the empty slot (src/philox.cuh:128-152).
__device__ __forceinline__ unsigned long long pack_key(int32_t score, int32_t v) {
    return (static_cast<unsigned long long>(static_cast<uint32_t>(score) ^ 0x80000000u) << 32) |
           static_cast<unsigned long long>(~static_cast<uint32_t>(v));
}

__device__ __forceinline__ int32_t key_vertex(unsigned long long key) {
    return static_cast<int32_t>(~static_cast<uint32_t>(key));
}

__device__ __forceinline__ int spin_of(const uint32_t* bits, int v) {
    return (bits[v >> 5] >> (v & 31)) & 1;
}

__device__ __forceinline__ void raise_error(const DevLaunch& L, int code, int item) {
    if (atomicCAS(L.error, 0, code) == 0) *L.errorItem = item;
}

// Barrier of one chain's warp group: __syncwarp for one warp, else named
// barrier grp+1 over the group's 32W threads (barrier 0 is __syncthreads).
__device__ __forceinline__ void group_sync(int grp, int T) {
    if (T == 32) {
        __syncwarp();
    } else {
        asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "r"(T) : "memory");
    }
}

// ------------------------------------------------------- gain storage
// A chain keeps one value per vertex and its spin as a mask byte (sb: 0x00
// for +1, 0xFF for -1).  D[v] = spin[v] * S[v] is the gain SELECT scores,
// S[v] = sum_u w(v,u) spin[u].
//
// int32 gains: D itself, plain words (a row walk reads the neighbour's spin
// to know the sign of its change).
struct D32 {
    static constexpr bool kField = false;
    static constexpr int32_t kBias = 0;
    // Stored values (D + kBias) of block b; D32 stores D itself.
    __device__ static __forceinline__ void load8raw(const unsigned char* D, const unsigned char*, int b, int32_t d[8]) {
        const int4 a = *reinterpret_cast<const int4*>(D + 32 * b);
        const int4 c = *reinterpret_cast<const int4*>(D + 32 * b + 16);
        d[0] = a.x; d[1] = a.y; d[2] = a.z; d[3] = a.w;
        d[4] = c.x; d[5] = c.y; d[6] = c.z; d[7] = c.w;
    }
    __device__ static __forceinline__ void load8(const unsigned char* D, const unsigned char* sb, int b, int32_t d[8]) {
        load8raw(D, sb, b, d);
    }
    __device__ static __forceinline__ int32_t get(const unsigned char* D, const unsigned char*, int v) {
        return reinterpret_cast<const int32_t*>(D)[v];
    }
    __device__ static __forceinline__ int32_t get_as(const unsigned char* D, uint32_t, int v) {
        return reinterpret_cast<const int32_t*>(D)[v];
    }
    __device__ static __forceinline__ void set(unsigned char* D, const unsigned char*, int v, int32_t d) {
        reinterpret_cast<int32_t*>(D)[v] = d;
    }
    // Vertex v (gain d, mask byte m before) flips.
    __device__ static __forceinline__ void flip(unsigned char* D, int v, int32_t d, uint32_t) {
        reinterpret_cast<int32_t*>(D)[v] = -d;
    }
    __device__ static __forceinline__ void add(unsigned char* D, int v, int32_t delta) {
        atomicAdd(reinterpret_cast<int*>(D) + v, delta);
    }
};

// Byte k of x sign-extended to 32 bits: prmt with selector nibbles whose msb
// requests sign replication (the __byte_perm intrinsic drops that bit).
template <int k>
__device__ __forceinline__ int32_t sbyte(uint32_t x) {
    int32_t r;
    if constexpr (k == 3) {
        r = static_cast<int32_t>(x) >> 24;
    } else {
        constexpr uint32_t sel = static_cast<uint32_t>(k) | ((8u | k) << 4) | ((8u | k) << 8) |
                                 ((8u | k) << 12);
        asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(x), "n"(sel));
    }
    return r;
}

// Byte k of x zero-extended to 32 bits, as a dot product with a unit byte: it
// issues on the FMA pipe, while a byte permute or a shift would take the ALU
// pipe that bounds SELECT (see score8_key).
template <int k>
__device__ __forceinline__ int32_t ubyte(uint32_t x) {
    int32_t r;
    asm("dp4a.u32.u32 %0, %1, %2, 0;" : "=r"(r) : "r"(x), "r"(1u << (8 * k)));
    return r;
}

// c + b * (half k of x, 16 bits), b < 256, on the FMA pipe: b arrives as byte k.
__device__ __forceinline__ uint32_t add_half(uint32_t x, uint32_t bytes, uint32_t c) {
    uint32_t r;
    asm("dp2a.lo.u32.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(x), "r"(bytes), "r"(c));
    return r;
}

// int8 gains (|S| <= B <= 127): the byte q holds S + 128 while the vertex's
// spin is +1 and S + 127 while it is -1, so that q ^ mask is D + 128 either
// way (255 - (S + 127) = -S + 128).  SELECT pays one 8-byte mask load and two
// xors per block of 8 vertices; a flipped vertex changes its neighbours' q by
// 2 * w * (its new spin) whatever their spins are, so FLIP's row walk needs
// no load of the neighbour's spin (one of its three dependent shared-memory
// accesses per entry, each with ~3 bank-conflict wavefronts).
// Changes are shifted 32-bit atomic adds on the containing word.  They commute
// and the word is the exact sum of its bytes' values times powers of 256, so
// whatever carries happen on the way, once a sweep's adds are all in (the only
// time a byte is read) every byte is back in [0, 255].
struct D8 {
    static constexpr bool kField = true;
    static constexpr int32_t kBias = 128;
    __device__ static __forceinline__ uint2 words(const unsigned char* D, const unsigned char* sb, int b) {
        const uint2 w = *reinterpret_cast<const uint2*>(D + 8 * b);
        const uint2 m = *reinterpret_cast<const uint2*>(sb + 8 * b);
        return make_uint2(w.x ^ m.x, w.y ^ m.y);
    }
    // D + 128 of block b's vertices (no sign handling: callers fold the bias
    // into a constant).
    __device__ static __forceinline__ void load8raw(const unsigned char* D, const unsigned char* sb, int b,
                                                    int32_t d[8]) {
        const uint2 w = words(D, sb, b);
        d[0] = ubyte<0>(w.x);
        d[1] = ubyte<1>(w.x);
        d[2] = ubyte<2>(w.x);
        d[3] = ubyte<3>(w.x);
        d[4] = ubyte<0>(w.y);
        d[5] = ubyte<1>(w.y);
        d[6] = ubyte<2>(w.y);
        d[7] = ubyte<3>(w.y);
    }
    __device__ static __forceinline__ void load8(const unsigned char* D, const unsigned char* sb, int b, int32_t d[8]) {
        const uint2 w = words(D, sb, b);
        const uint32_t a = w.x ^ 0x80808080u, c = w.y ^ 0x80808080u;
        d[0] = sbyte<0>(a);
        d[1] = sbyte<1>(a);
        d[2] = sbyte<2>(a);
        d[3] = sbyte<3>(a);
        d[4] = sbyte<0>(c);
        d[5] = sbyte<1>(c);
        d[6] = sbyte<2>(c);
        d[7] = sbyte<3>(c);
    }
    __device__ static __forceinline__ int32_t get(const unsigned char* D, const unsigned char* sb, int v) {
        return static_cast<int32_t>(D[v] ^ sb[v]) - 128;
    }
    // The same for a vertex whose spin is known (neg: -1).
    __device__ static __forceinline__ int32_t get_as(const unsigned char* D, uint32_t neg, int v) {
        return static_cast<int32_t>(D[v] ^ (neg ? 0xFFu : 0u)) - 128;
    }
    __device__ static __forceinline__ void set(unsigned char* D, const unsigned char* sb, int v, int32_t d) {
        D[v] = static_cast<unsigned char>((d + 128) ^ sb[v]);
    }
    // Vertex v (gain d, mask byte m before) flips: S stays, D changes sign.
    __device__ static __forceinline__ void flip(unsigned char* D, int v, int32_t d, uint32_t m) {
        D[v] = static_cast<unsigned char>((128 - d) ^ (m ^ 0xFFu));
    }
    __device__ static __forceinline__ void add(unsigned char* D, int v, int32_t delta) {
        atomicAdd(reinterpret_cast<unsigned int*>(D + (v & ~3)),
                  static_cast<unsigned int>(delta) << (8 * (v & 3)));
    }
};

// ------------------------------------------------------------ CSR access
struct CsrView {
    const uint32_t* off;   // row words (compact formats) or plain offsets
    const void* ent;
};

// A word of the CSR: from the CTA's shared-memory copy, or from HBM through
// the read-only path.
template <bool kHbm, class T>
__device__ __forceinline__ T csr_load(const T* p) {
    if constexpr (kHbm) return __ldg(p);
    else return *p;
}

template <int kFmt>
struct Csr {
    static constexpr bool kHbm = csr_in_hbm(kFmt);
    static constexpr bool kPlain = kFmt == kCsrGlobal;                          // {col, w} pairs, rows not padded
    static constexpr bool kUnit = kFmt == kCsrUnit16 || kFmt == kCsrGlobal16;   // 16-bit entries
    // Row v as two words: plain offsets, or row words (first entry | padding,
    // next row's).
    __device__ static __forceinline__ void row(const CsrView& c, int v, uint32_t& lo, uint32_t& hi) {
        lo = csr_load<kHbm>(c.off + v);
        hi = csr_load<kHbm>(c.off + v + 1);
    }
    // The row's entries [i, end).
    __device__ static __forceinline__ void entries(const CsrView& c, int v, uint32_t& i, uint32_t& end) {
        row(c, v, i, end);
        if constexpr (!kPlain) {
            end = (end & ~3u) - (i & 3u);
            i &= ~3u;
        }
    }
    __device__ static __forceinline__ void entry(const CsrView& c, uint32_t i, int& col, int& w) {
        if constexpr (kPlain) {
            const int2 e = csr_load<kHbm>(static_cast<const int2*>(c.ent) + i);
            col = e.x;
            w = e.y;
        } else if constexpr (kUnit) {
            const uint32_t e = csr_load<kHbm>(static_cast<const unsigned short*>(c.ent) + i);
            col = static_cast<int>(e & 0x7FFFu);
            w = 1 - 2 * static_cast<int>(e >> 15);
        } else {
            const uint32_t e = csr_load<kHbm>(static_cast<const unsigned int*>(c.ent) + i);
            col = static_cast<int>(e & 0xFFFFu);
            w = static_cast<int32_t>(e) >> 16;
        }
    }
    // Vector q: entries 4q .. 4q + 3 (two to a word for 16-bit entries).
    using Vec = typename std::conditional<kUnit, uint2, uint4>::type;
    __device__ static __forceinline__ Vec vec(const CsrView& c, uint32_t q) {
        return csr_load<kHbm>(static_cast<const Vec*>(c.ent) + q);
    }
};

// ------------------------------------------------------------ chain region
struct ChainSmem {
    unsigned char* D;
    uint32_t* bits;
    uint32_t* best;
    unsigned char* sb;           // spins as mask bytes (0x00 = +1, 0xFF = -1), kept equal to bits
    unsigned long long* slots;   // int32 mode: packed keys
    long long* scores;           // int64 mode: max score per group (aliases slots)
    int32_t* ids;                // int64 mode: winner id per group
    int32_t* win;                // winners of the current sweep
    int64_t* red;                // one partial per warp of the group
};

__device__ __forceinline__ ChainSmem carve_chain(unsigned char* base, const DevLaunch& L,
                                                 int dbytes) {
    const ChainLayout c = chain_layout(L.maxN, L.maxWords, L.pmax, L.warpsPerChain, dbytes, L.layout);
    ChainSmem s;
    s.D = base + c.d;
    s.bits = reinterpret_cast<uint32_t*>(base + c.bits);
    s.best = reinterpret_cast<uint32_t*>(base + c.best);
    s.sb = base + c.sb;
    s.slots = reinterpret_cast<unsigned long long*>(base + c.slots);
    s.scores = reinterpret_cast<long long*>(base + c.slots);
    s.ids = reinterpret_cast<int32_t*>(base + c.ids);
    s.win = reinterpret_cast<int32_t*>(base + c.win);
    s.red = reinterpret_cast<int64_t*>(base + c.red);
    return s;
}

// Exact int64 sum over a chain's warp group; every thread gets the total.
// (The partials buffer is rewritten only after two more group barriers.)
__device__ __forceinline__ int64_t group_sum(int64_t v, const ChainSmem& s, int t, int T, int grp) {
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, m);
    if (T == 32) return v;
    if ((t & 31) == 0) s.red[t >> 5] = v;
    group_sync(grp, T);
    int64_t tot = 0;
    for (int w = 0; w < (T >> 5); ++w) tot += s.red[w];
    return tot;
}

// Exact warp sums with redux.sync.  int8 gains: the winners' gains of a sweep
// sum to at most 2 * 127 * P, far inside int32.  int32 gains: a lane's v is split
// into its low 24 bits, whose sum over 32 lanes is below 2^29, and the rest, whose
// sum stays in int32 while |v| < 2^50: a lane adds at most 2 * 2^31 a winner, and
// the fewer than 2^17 vertices that a chain's shared memory holds over 32 lanes.
__device__ __forceinline__ int32_t warp_sum(int32_t v) { return __reduce_add_sync(0xFFFFFFFFu, v); }
__device__ __forceinline__ int64_t warp_sum(int64_t v) {
    const int32_t lo = __reduce_add_sync(0xFFFFFFFFu, static_cast<int32_t>(v & 0xFFFFFF));
    const int32_t hi = __reduce_add_sync(0xFFFFFFFFu, static_cast<int32_t>(v >> 24));
    return (static_cast<int64_t>(hi) << 24) + lo;
}

// ---------------------------------------------------------------- SELECT
// Scores every vertex from pre-sweep D and leaves the winner of every group
// g < P in the chain's slots (int32 mode: packed key; int64 mode: ids[g]).
// Slots start each sweep at their empty value (reset by FLIP's reader).

// Per-phase constants, recomputed only when P changes (no integer division
// or modulo by P inside a sweep).
//
// kPathWarp: P <= 128 and private groups.  The block loop strides by S blocks,
// 8 S a multiple of P, so that every (lane, j) accumulator belongs to one
// group; each warp reduces its 256 accumulators to P winners (warp_argmax) and
// the winners stay in registers (one-warp chains) or pass through one 8-byte
// partial per warp and group (wider ones).  S is T when 8 T % P == 0 (any
// power of two), else the largest multiple of P / gcd(P, 8) up to T, the
// remaining threads idle in SELECT; when that is above 32, a one-warp chain
// plays its ceil(S / 32) warps one after another.
// Other P go through the group slots: kPathPrivate when 8 T % P == 0 (one
// atomic per accumulator), else kPathVertex (one atomic per vertex).
enum PhasePath : int { kPathWarp = 0, kPathPrivate = 1, kPathVertex = 2 };

struct PhaseCfg {
    int P;
    int path;       // PhasePath
    int laneShift;  // FLIP: log2 of the lanes that share one winner's row
    int rows;       // FLIP: rows a thread takes part in on kPathWarp (1 to 4)
    int S;          // block stride (T but on kPathWarp; above 32 a one-warp chain
                    //    plays several warps)
    int shares;     // 256 mod P: how far each warp's groups are shifted from the one
                    //    before; 0 on kPathWarp's main path
    int warpG;      // kPathWarp: (256 warp) mod P
};

__device__ __forceinline__ int key_bits(int n, int T) {
    const int iters = ((n + 7) / 8 + T - 1) / T;
    int kb = 4;
    while ((1 << kb) < iters) ++kb;
    return kb;
}

// kbMax: bits the chain's keys can spare for the block iteration; `slots`:
// the group slots are wanted (int64 scores, chains without argmax scratch).
__device__ __forceinline__ PhaseCfg phase_cfg(int P, int n, int t, int T, bool one, int kbMax, bool slots) {
    PhaseCfg c;
    c.P = P;
    c.S = T;
    const int twos = P & -P;
    const int s0 = P / (twos < 8 ? twos : 8);
    int S = T;
    if ((8 * T) % P != 0) S = s0 <= T ? T / s0 * s0 : (one ? s0 : 0);
    const bool warp = !slots && P <= 128 && S > 0 && key_bits(n, S > 0 ? S : 1) <= kbMax;
    c.S = uniform(warp ? S : T);
    const bool priv = (8 * T) % P == 0 && key_bits(n, T) <= kbMax;
    c.path = uniform(static_cast<int>(warp ? kPathWarp : priv ? kPathPrivate : kPathVertex));
    c.shares = uniform(256 % P);
    c.warpG = uniform((8 * (t & ~31)) % P);
    int sh = 0;
    while ((2 << sh) * P <= T && sh < 5) ++sh;
    c.laneShift = uniform(sh);
    c.rows = uniform((P + T - 1) / T);
    return c;
}

// Compact int32 argmax key.  A thread visits its vertex blocks b = t + k*T
// for k = 0, 1, ... (at most 2^kb of them); lane j of block k gets
//   key = score * 2^kb + (2^kb - 1 - k),   score = gum + beta * delta,
// so one integer max per vertex keeps the best score and, among equal
// scores, the smallest k, i.e. the smallest vertex (v = 8(t + kT) + j grows
// with k).  With f the 11-bit field and i = f & 15,
//   gum * 2^kb = LUT[i] * 2^kb + (f >> 4) * 2^kb
//              = (LUT[i] * 2^kb - i * 2^(kb-4)) + f * 2^(kb-4)     (kb >= 4)
// so key = TK[i] + f * 2^(kb-4) + (beta * 2^kb) * delta + (2^kb - 1 - k) with a
// 16-entry table TK.  The host enables this path only when
// (betaMax * B + max|gum| + 1) * 2^kb < 2^31 for every chain, so every key and
// partial sum is exact in int32; otherwise the launch takes the int64 path.
//
// Instruction budget per vertex: TK lives in a register (lane L holds
// TK[L & 15]) and is read with one shuffle whose source lane is the Philox
// word itself (a shuffle takes its source lane modulo 32, and lanes L and
// L + 16 hold the same entry, so the low word needs no masking and the high
// one a single shift); beta * gain is one multiply-add; the field is a mask
// folded into the add + max when kb == 4, else its multiple is added by a
// 16-bit dot product.
//
// Measured on GB300, cycles per warp instruction and scheduler: logic, shifts,
// permutes, max and add-max 2 on the ALU pipe; 32-bit multiply-add and the dot
// products 2 on the FMA pipe; a wide or high multiply 4 on the FMA pipe and 2
// on the ALU pipe.  A block of 8 vertices' Philox takes 74 ALU / 72 FMA
// cycles; its scoring adds 44 / 32, having moved the byte extraction of int8
// gains off the ALU pipe (60 / 16 before; the loop alone at four warps per
// scheduler 143 -> 134 cycles a block).  Adding some of the fields with dot
// products too (114 / 112 on paper) was slower, 138.
struct KeyCfg {
    int kb;          // bits of the block-iteration field
    uint32_t mulF;   // 2^(kb-4), the field's multiple; below 256 (a chain of 2^19 vertices would not fit)
    int32_t tkLane;  // TK[lane & 15]
    int full;        // block iterations of a stride S over all blocks: `full`,
    int extra;       //   and one more for the threads below `extra`
};

__device__ __forceinline__ KeyCfg key_cfg(int n, int S, int t, const int32_t* lut) {
    KeyCfg kc;
    kc.kb = uniform(key_bits(n, S));
    kc.mulF = 1u << (kc.kb - 4);
    kc.full = uniform(((n + 7) >> 3) / S);
    kc.extra = uniform(((n + 7) >> 3) % S);
    const int i = t & 15;
    kc.tkLane = lut[i] * (1 << kc.kb) - i * static_cast<int32_t>(kc.mulF) + (1 << kc.kb) - 1;
    return kc;
}

// The most block-iteration bits the compact keys of a chain can carry: its
// largest score is betaMax * B + max|gum|.
__device__ __forceinline__ int key_room(int32_t betaMax, int64_t B) {
    const int64_t top = static_cast<int64_t>(betaMax) * B + kGumMaxMag + 1;
    int kb = 0;
    while (kb < 12 && (top << (kb + 1)) < 2147483647) ++kb;
    return kb;
}

// Keys of one block's 8 vertices folded into acc; lanes j >= lim are skipped
// (the shuffles still run on every lane: the caller keeps the warp converged).
// `tkb` is this lane's TK[lane & 15] plus the block's constant part
// (2^kb - 1 - k) - bias * beta * 2^kb, so the shuffle delivers TK[i] with the
// constant already added and d holds the stored (biased) gains.  All sums are
// modular int32: only the final key is in range, and it is exact.  kF0: kb ==
// 4, the field's multiple is the field itself.
template <bool kMasked, bool kF0>
__device__ __forceinline__ void score8_key(int32_t acc[8], const uint32_t x[4], const int32_t d[8],
                                           int32_t betaK, int32_t tkb, const KeyCfg& kc, int lim) {
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const uint32_t xs = x[w] >> 16;
        const int32_t tk0 = __shfl_sync(0xFFFFFFFFu, tkb, static_cast<int>(x[w]));
        const int32_t tk1 = __shfl_sync(0xFFFFFFFFu, tkb, static_cast<int>(xs));
        const int32_t k0 = static_cast<int32_t>(static_cast<uint32_t>(betaK) * static_cast<uint32_t>(d[2 * w]) +
                                                static_cast<uint32_t>(tk0));
        const int32_t k1 = static_cast<int32_t>(static_cast<uint32_t>(betaK) * static_cast<uint32_t>(d[2 * w + 1]) +
                                                static_cast<uint32_t>(tk1));
        if constexpr (kF0) {
            if (!kMasked || 2 * w < lim)
                acc[2 * w] = __viaddmax_s32(k0, static_cast<int32_t>(x[w] & 0x7FFu), acc[2 * w]);
            if (!kMasked || 2 * w + 1 < lim)
                acc[2 * w + 1] = __viaddmax_s32(k1, static_cast<int32_t>(xs & 0x7FFu), acc[2 * w + 1]);
        } else {
            const uint32_t f = x[w] & 0x07FF07FFu;
            const int32_t s0 = static_cast<int32_t>(add_half(f, kc.mulF, static_cast<uint32_t>(k0)));
            const int32_t s1 = static_cast<int32_t>(add_half(f, kc.mulF << 8, static_cast<uint32_t>(k1)));
            if (!kMasked || 2 * w < lim) acc[2 * w] = max(acc[2 * w], s0);
            if (!kMasked || 2 * w + 1 < lim) acc[2 * w + 1] = max(acc[2 * w + 1], s1);
        }
    }
}

// NB vertex blocks b, b + T, ... (block iterations k, k + 1, ...) scored with
// their Philox draws in flight together.  kTail: the last of them may be
// ragged: a lane past the last block scores that block's place again with
// lim = 0, one on a partial block has lim = n & 7.
template <int NB, bool kTail, bool kF0, class DP>
__device__ __forceinline__ void score_blocks(int32_t acc[8], const ChainSmem& s, const SweepConst& sc,
                                             const ChainKeys& keys, int b, int T, int n, int32_t betaK,
                                             int32_t tkb, const KeyCfg& kc) {
    uint32_t x[NB][4];
    int last = b + (NB - 1) * T, lim = 8;
    if (kTail) {
        const int nfull = n >> 3, nblk = (n + 7) >> 3;
        lim = (last < nfull) ? 8 : ((last == nfull) ? (n & 7) : 0);
        last = (last < nblk) ? last : nblk - 1;
    }
#pragma unroll
    for (int q = 0; q < NB; ++q)
        philox_block(static_cast<uint32_t>(q == NB - 1 ? last : b + q * T), sc, keys, x[q]);
    // Each block's gains are loaded just before it is scored so that three
    // blocks' Philox words fit the registers.
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        int32_t d[8];
        DP::load8raw(s.D, s.sb, q == NB - 1 ? last : b + q * T, d);
        if (kTail && q == NB - 1) score8_key<true, kF0>(acc, x[q], d, betaK, tkb - q, kc, lim);
        else score8_key<false, kF0>(acc, x[q], d, betaK, tkb - q, kc, 8);
    }
}

// The block loop of select32: the warp's iterations (uniform, so the table
// shuffles run converged), three in flight, the last one to three together:
// all of them full but the very last.  One iteration alone takes 250 cycles
// on GB300 against 180 each for two or three in flight, so the remainder is
// never walked one by one.
template <bool kF0, class DP>
__device__ __forceinline__ void select_blocks(int32_t acc[8], const ChainSmem& s, const SweepConst& sc,
                                              const ChainKeys& keys, int n, int t, int T, int left,
                                              int32_t betaK, int32_t tkb, const KeyCfg& kc) {
    int b = t;
    for (; left > 3; left -= 3, b += 3 * T, tkb -= 3)
        score_blocks<3, false, kF0, DP>(acc, s, sc, keys, b, T, n, betaK, tkb, kc);
    if (left == 3) score_blocks<3, true, kF0, DP>(acc, s, sc, keys, b, T, n, betaK, tkb, kc);
    else if (left == 2) score_blocks<2, true, kF0, DP>(acc, s, sc, keys, b, T, n, betaK, tkb, kc);
    else if (left == 1) score_blocks<1, true, kF0, DP>(acc, s, sc, keys, b, T, n, betaK, tkb, kc);
}

// The winner of one group among a warp's 256 accumulators: its compact key
// and the accumulator it came from (8 * lane + j).  Equal keys mean equal
// score and block iteration, so the smaller accumulator is the smaller vertex.
__device__ __forceinline__ bool beats(int32_t ka, int32_t aa, int32_t kb, int32_t ab) {
    return ka > kb || (ka == kb && aa < ab);
}

// Per-warp scratch of warp_argmax: the 256 accumulators as words, j >= 4 in a
// second half that starts 16 banks later, so that both the vector stores
// (4 words per lane) and the transposed reads (lanes at consecutive
// accumulators) are free of bank conflicts.  Wider chains reuse it for the
// warp's partials (8 bytes per group, P <= 128).
constexpr int kHalf = 144;

// Groups of a warp's accumulators for P = 32 Q, or P <= 32 with Q = 1:
// accumulator a belongs to group a mod P; lane l gets the winners of groups
// l + 32 q (of group l mod P when P < 32, in every lane of that residue).
// The accumulators are transposed through shared memory, where eight reads
// and a register tree replace log2(256 / P) shuffles of each of the eight
// accumulators and a ballot per Philox lane to find the winning lane.  Wider
// chains used to merge their warps' winners with 64-bit shared atomic maxima
// (a compare-and-swap loop each), 1,900 to 2,900 cycles of a sweep on GB300.
// us per sweep before / with this and the settled gain (see run_chain):
// 1024 one-warp chains of ER n = 2000 P = 16 3.55 / 2.97, P = 128 7.55 / 6.75;
// 32 four-warp chains of ER n = 800 P = 16 2.93 / 1.94; 80 eight-warp chains
// of the 100x200 torus P = 16 4.36 / 3.75.
template <int Q>
__device__ __forceinline__ void warp_argmax(const int32_t acc[8], int32_t* scr, int lane, int P, int32_t key[4],
                                            int32_t at[4]) {
    *reinterpret_cast<int4*>(scr + 4 * lane) = make_int4(acc[0], acc[1], acc[2], acc[3]);
    *reinterpret_cast<int4*>(scr + kHalf + 4 * lane) = make_int4(acc[4], acc[5], acc[6], acc[7]);
    __syncwarp();
    const int32_t* mine = scr + 4 * (lane >> 3) + (lane & 3) + kHalf * ((lane >> 2) & 1);
    int32_t k[8], a[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        k[i] = mine[16 * i];   // accumulator lane + 32 i
        a[i] = lane + 32 * i;
    }
#pragma unroll
    for (int d = Q; d < 8; d *= 2) {
#pragma unroll
        for (int i = 0; i + d < 8; ++i) {
            if ((i / Q) % (2 * d / Q) == 0 && k[i + d] > k[i]) {
                k[i] = k[i + d];
                a[i] = a[i + d];
            }
        }
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        key[q] = k[q];
        at[q] = a[q];
    }
    if (Q == 1) {
        for (int m = 16; m >= P; m >>= 1) {
            const int32_t ok = __shfl_xor_sync(0xFFFFFFFFu, key[0], m);
            const int32_t oa = __shfl_xor_sync(0xFFFFFFFFu, at[0], m);
            if (beats(ok, oa, key[0], at[0])) {
                key[0] = ok;
                at[0] = oa;
            }
        }
    }
}

// Lanes that share a group of warp_argmax_any: 32 / P for a P below 16 that does
// not divide 32, never more (a division a sweep cost 110 cycles).
__constant__ unsigned char kShare[129] = {
    1, 15, 15, 10, 8, 6, 5, 4, 4, 3, 3, 2, 2, 2, 2, 2, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1,
    1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1,
    1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1,
    1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1,
};

// The same for any P <= 128: class c = a mod P (the group but for the warp's
// shift).  With P <= 32, 32 / P lanes share a class and fold pairwise into its
// first lane; four reads go out together.
//
// Accumulators lie at their own number here: lane-consecutive reads at any P,
// each address one add, where the halves of warp_argmax took seven
// instructions a read.  GB300, us per sweep before / now: 300 four-warp chains
// of a weighted ER n = 1500 P = 100 2.85 / 2.70, P = 12 1.90 / 1.77; 1024
// one-warp chains of ER n = 2000 P = 60 4.40 / 4.19, P = 5 2.98 / 2.80.
__device__ __forceinline__ void warp_argmax_any(const int32_t acc[8], int32_t* scr, int lane, int P, int share,
                                                int32_t key[4], int32_t at[4]) {
    *reinterpret_cast<int4*>(scr + 8 * lane) = make_int4(acc[0], acc[1], acc[2], acc[3]);
    *reinterpret_cast<int4*>(scr + 8 * lane + 4) = make_int4(acc[4], acc[5], acc[6], acc[7]);
    __syncwarp();
    const int width = share * P;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        key[q] = INT32_MIN;
        at[q] = 0;
        const int c = lane + 32 * q;
        if (c < width) {
#pragma unroll 1
            for (int a = c; a < 256; a += 4 * width) {
                int32_t k[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) k[i] = a + i * width < 256 ? scr[a + i * width] : INT32_MIN;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (k[i] > key[q]) {
                        key[q] = k[i];
                        at[q] = a + i * width;
                    }
                }
            }
        }
    }
    while (share > 1) {
        const int half = (share + 1) >> 1;
        const int32_t ok = __shfl_down_sync(0xFFFFFFFFu, key[0], half * P);
        const int32_t oa = __shfl_down_sync(0xFFFFFFFFu, at[0], half * P);
        if (lane < (share - half) * P && beats(ok, oa, key[0], at[0])) {
            key[0] = ok;
            at[0] = oa;
        }
        share = half;
    }
    if (lane >= P) key[0] = INT32_MIN;
}

// P = 1: fold the eight accumulators in registers, one warp max, and the
// lowest lane holding it; every lane gets the winner.
__device__ __forceinline__ void warp_argmax_one(const int32_t acc[8], int32_t& key, int32_t& at) {
    int32_t k[8];
    int jb[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) { k[j] = acc[j]; jb[j] = j; }
#pragma unroll
    for (int d = 1; d < 8; d *= 2) {
#pragma unroll
        for (int j = 0; j < 8; j += 2 * d)
            if (k[j + d] > k[j]) { k[j] = k[j + d]; jb[j] = jb[j + d]; }
    }
    key = __reduce_max_sync(0xFFFFFFFFu, k[0]);
    const int src = __ffs(__ballot_sync(0xFFFFFFFFu, k[0] == key)) - 1;
    at = 8 * src + __shfl_sync(0xFFFFFFFFu, jb[0], src);
}

// A wider chain's partial: one warp's winner of one group, ordered as an
// unsigned 64-bit number by key, then smaller vertex; 0 is none.  int8 gains
// carry the winner's spin sign and gain byte along (FLIP needs the gain from
// before any neighbour's flip, and so saves the barrier between reading it
// and scattering); v < 2^23 there (a chain keeps two bytes per vertex in
// shared memory).
template <class DP>
__device__ __forceinline__ unsigned long long make_partial(const ChainSmem& s, int32_t key, int v) {
    uint32_t lo;
    if constexpr (DP::kField) {
        const uint32_t m = s.sb[v];
        lo = ((~static_cast<uint32_t>(v) & 0x7FFFFFu) << 9) | ((m & 1u) << 8) |
             static_cast<uint32_t>(static_cast<unsigned char>(s.D[v] ^ m));
    } else {
        lo = ~static_cast<uint32_t>(v);
    }
    return (static_cast<unsigned long long>(static_cast<uint32_t>(key) ^ 0x80000000u) << 32) | lo;
}

// The accumulators of one warp over its `iters` block iterations at stride S
// (thread t of it).
template <bool kF0, class DP>
__device__ __forceinline__ void select_warp(int32_t acc[8], const ChainSmem& s, const SweepConst& sc,
                                            const ChainKeys& keys, int n, const KeyCfg& kc, int t, int S, int iters,
                                            int32_t beta) {
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = INT32_MIN;
    const int32_t betaK = beta * (1 << kc.kb);
    // Per-sweep part of the table register: (2^kb - 1) - bias * beta * 2^kb.
    const int32_t tkBase = static_cast<int32_t>(static_cast<uint32_t>(kc.tkLane) -
                                                static_cast<uint32_t>(DP::kBias) * static_cast<uint32_t>(betaK));
    select_blocks<kF0, DP>(acc, s, sc, keys, n, t, S, iters, betaK, tkBase, kc);
}

// The winners of a warp's P classes as its partials (wider chains) or in
// registers (v).
template <bool kOne, class DP>
__device__ __forceinline__ void warp_winners(const ChainSmem& s, const PhaseCfg& pc, const KeyCfg& kc, int32_t* scr,
                                             int first, int lane, int S, const int32_t key[4], const int32_t at[4],
                                             int32_t v[4]) {
    const int M = (1 << kc.kb) - 1;
    const int Q = (pc.P + 31) >> 5;
    if (!kOne) __syncwarp();   // the scratch is rewritten below
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (q >= Q) break;
        const int kk = M - (key[q] & M);
        v[q] = (key[q] != INT32_MIN) ? 8 * first + at[q] + 8 * kk * S : -1;
        if (!kOne) {
            const int c = lane + 32 * q;
            if (c < pc.P) {
                const int g = c + pc.warpG < pc.P ? c + pc.warpG : c + pc.warpG - pc.P;
                reinterpret_cast<unsigned long long*>(scr)[g] =
                    (v[q] >= 0) ? make_partial<DP>(s, key[q], v[q]) : 0ull;
            }
        }
    }
}

// SELECT off the main path: private groups at a stride S below T (or, for
// one-warp chains, above 32: the warps played one after another, each one's
// winners merged into a table with one lane per group), and the slots.  Code
// of its own: a variable stride in the main path's block loop cost every
// phase 8 to 13% on GB300.
template <bool kOne, class DP>
__device__ __forceinline__ void select32_general(const ChainSmem& s, const int32_t* lut, const KeyCfg& kc, int n,
                                                 const PhaseCfg& pc, int32_t beta, const SweepConst& sc,
                                                 const ChainKeys& keys, int t, int T, int32_t v[4]) {
    const int P = pc.P;
    if (pc.path == kPathVertex) {
        // One shared atomic per vertex, plain score.
        for (int bb = t; 8 * bb < n; bb += T) {
            uint32_t x[4];
            int32_t d[8];
            philox_block(static_cast<uint32_t>(bb), sc, keys, x);
            DP::load8(s.D, s.sb, bb, d);
            int g = (8 * bb) % P;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int vv = 8 * bb + j;
                if (vv < n) {
                    const uint32_t r = field(x, j);
                    const int32_t sv = lut[r & 15u] + static_cast<int32_t>(r >> 4) + beta * d[j];
                    atomicMax(&s.slots[g], pack_key(sv, vv));
                }
                if (++g == P) g = 0;
            }
        }
        return;
    }
    const int lane = t & 31, S = pc.S, M = (1 << kc.kb) - 1;
    int shift = 0;   // (256 round) mod P
    for (int first = t & ~31;; first += 32) {
        // Threads from S on idle: they score the last one's blocks and drop
        // them.
        int32_t acc[8], key[4], at[4];
        const int iters = first < S ? kc.full + (first < kc.extra ? 1 : 0) : 0;
        select_warp<false, DP>(acc, s, sc, keys, n, kc, first + lane < S ? first + lane : S - 1, S, iters, beta);
        if (pc.path == kPathPrivate) {
            int g = (8 * t) % P;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (acc[j] != INT32_MIN) {
                    const int kk = M - (acc[j] & M);
                    atomicMax(&s.slots[g], pack_key(acc[j] >> kc.kb, 8 * (t + kk * T) + j));
                }
                if (++g == P) g = 0;
            }
            return;
        }
        if (first + lane >= S) {
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] = INT32_MIN;
        }
        int32_t* scr = reinterpret_cast<int32_t*>(reinterpret_cast<unsigned char*>(s.slots) +
                                                  (kOne ? 0 : (t >> 5) * kWarpScratch));
        warp_argmax_any(acc, scr, lane, P, kShare[P], key, at);
        if (!kOne || S <= 32) {
            warp_winners<kOne, DP>(s, pc, kc, scr, first, lane, S, key, at, v);
            return;
        }
        unsigned long long* table = reinterpret_cast<unsigned long long*>(s.ids);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int c = lane + 32 * q;
            if (c < P) {
                const int g = c + shift < P ? c + shift : c + shift - P;
                const unsigned long long mine =
                    key[q] != INT32_MIN ? pack_key(key[q], 8 * first + at[q] + 8 * (M - (key[q] & M)) * S) : 0ull;
                if (first == 0 || mine > table[g]) table[g] = mine;
            }
        }
        const int step = pc.shares;
        shift = shift + step < P ? shift + step : shift + step - P;
        __syncwarp();
        if (first + 32 >= S) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int g = lane + 32 * q;
                const unsigned long long p = g < P ? table[g] : 0ull;
                v[q] = p ? key_vertex(p) : -1;
            }
            __syncwarp();
            return;
        }
    }
}

// SELECT of the int32 path.  On kPathWarp, on return lane l of a one-warp chain
// holds the winners v[q] of groups l + 32 q (-1: none) and a wider chain has
// its partials in place (a barrier is due); else the winners are packed keys
// in the group slots (a barrier is due).
template <bool kOne, class DP>
__device__ __forceinline__ void select32(const ChainSmem& s, const int32_t* lut, const KeyCfg& kc, int n,
                                         const PhaseCfg& pc, int32_t beta, const SweepConst& sc,
                                         const ChainKeys& keys, int t, int T, int32_t v[4]) {
    if (pc.path != kPathWarp || pc.shares != 0) {
        select32_general<kOne, DP>(s, lut, kc, n, pc, beta, sc, keys, t, T, v);
        return;
    }
    const int P = pc.P;
    const int lane = t & 31, first = kOne ? 0 : t & ~31;
    int32_t acc[8], key[4], at[4];
    const int iters = kc.full + (first < kc.extra ? 1 : 0);
    if (kc.kb == 4) select_warp<true, DP>(acc, s, sc, keys, n, kc, t, T, iters, beta);
    else select_warp<false, DP>(acc, s, sc, keys, n, kc, t, T, iters, beta);
    int32_t* scr = reinterpret_cast<int32_t*>(reinterpret_cast<unsigned char*>(s.slots) +
                                              (kOne ? 0 : (t >> 5) * kWarpScratch));
    if (P == 1) warp_argmax_one(acc, key[0], at[0]);
    else if (P <= 32) warp_argmax<1>(acc, scr, lane, P, key, at);
    else if (P == 64) warp_argmax<2>(acc, scr, lane, P, key, at);
    else warp_argmax<4>(acc, scr, lane, P, key, at);
    warp_winners<kOne, DP>(s, pc, kc, scr, first, lane, T, key, at, v);
}

// int64 scores (the reference's two-pass path, src/anneal_kernels.cu:348-378,
// taken when annealScoreSafeInt32 fails): max score per group, then the
// smallest v reaching it.
struct Acc64 {
    long long s[8];
    uint32_t b[8];
};

__device__ __forceinline__ void score8_64(Acc64& a, const uint32_t x[4], const int32_t d[8],
                                          int32_t beta, const int32_t* lut, uint32_t b, int lim) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (j < lim) {
            const uint32_t r = field(x, j);
            const long long sc = static_cast<long long>(lut[r & 15u] + static_cast<int32_t>(r >> 4)) +
                                 static_cast<long long>(beta) * d[j];
            if (sc > a.s[j]) { a.s[j] = sc; a.b[j] = b; }
        }
    }
}

template <class DP>
__device__ void select64(const ChainSmem& s, const int32_t* lut, int n, const PhaseCfg& pc,
                         int32_t beta, const SweepConst& sc, const ChainKeys& keys, int t, int T,
                         int grp) {
    const int P = pc.P;
    const bool priv = pc.path != kPathVertex;
    if (priv) {
        Acc64 a;
#pragma unroll
        for (int j = 0; j < 8; ++j) { a.s[j] = LLONG_MIN; a.b[j] = 0; }
        for (int b = t; 8 * b < n; b += T) {
            uint32_t x[4];
            int32_t d[8];
            philox_block(static_cast<uint32_t>(b), sc, keys, x);
            DP::load8(s.D, s.sb, b, d);
            const int lim = (n - 8 * b < 8) ? (n - 8 * b) : 8;
            score8_64(a, x, d, beta, lut, static_cast<uint32_t>(b), lim);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (a.s[j] != LLONG_MIN) atomicMax(&s.scores[(8 * t + j) % P], a.s[j]);
        group_sync(grp, T);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int g = (8 * t + j) % P;
            if (a.s[j] != LLONG_MIN && a.s[j] == s.scores[g])
                atomicMin(&s.ids[g], static_cast<int32_t>(8 * a.b[j] + j));
        }
    } else {
        for (int pass = 0; pass < 2; ++pass) {
            for (int b = t; 8 * b < n; b += T) {
                uint32_t x[4];
                int32_t d[8];
                philox_block(static_cast<uint32_t>(b), sc, keys, x);
                DP::load8(s.D, s.sb, b, d);
                int g = (8 * b) % P;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int v = 8 * b + j;
                    if (v < n) {
                        const uint32_t r = field(x, j);
                        const long long sv =
                            static_cast<long long>(lut[r & 15u] + static_cast<int32_t>(r >> 4)) +
                            static_cast<long long>(beta) * d[j];
                        if (pass == 0) atomicMax(&s.scores[g], sv);
                        else if (sv == s.scores[g]) atomicMin(&s.ids[g], v);
                    }
                    if (++g == P) g = 0;
                }
            }
            if (pass == 0) group_sync(grp, T);
        }
    }
}

// ------------------------------------------------------------------- FLIP
// One 16-bit entry (the low half of e): the neighbour's byte changes by +2 or
// -2, added into byte lane col & 3 of its word (the shift wraps at 32, so it
// needs no mask).  `nm`: 0x8000 when the winner's new spin is -1.
__device__ __forceinline__ void add_unit(unsigned char* D, uint32_t e, uint32_t nm) {
    const uint32_t val = ((e ^ nm) & 0x8000u) ? 0xFFFFFFFEu : 2u;
    atomicAdd(reinterpret_cast<unsigned int*>(D + (e & 0x7FFCu)), __funnelshift_l(0u, val, e << 3));
}

// One 32-bit entry w << 16 | col.  `neg`: the winner's new spin is -1.
template <class DP>
__device__ __forceinline__ void add_packed(const ChainSmem& s, uint32_t e, uint32_t neg) {
    const int c = static_cast<int>(e & 0xFFFFu), w2 = 2 * (static_cast<int32_t>(e) >> 16);
    const uint32_t x = DP::kField ? 0u : s.sb[c] & 1u;
    DP::add(s.D, c, (neg ^ x) ? -w2 : w2);
}

// A vector of four entries of a compact row.
template <class DP, int kFmt>
__device__ __forceinline__ void add_vec(const ChainSmem& s, const typename Csr<kFmt>::Vec& e, uint32_t neg) {
    if constexpr (!Csr<kFmt>::kUnit) {
        add_packed<DP>(s, e.x, neg);
        add_packed<DP>(s, e.y, neg);
        add_packed<DP>(s, e.z, neg);
        add_packed<DP>(s, e.w, neg);
    } else {
        const uint32_t h[4] = {e.x, e.x >> 16, e.y, e.y >> 16};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if constexpr (DP::kField) {
                add_unit(s.D, h[j], neg << 15);
            } else {
                const int c = static_cast<int>(h[j] & 0x7FFFu);
                DP::add(s.D, c, (((h[j] >> 15) ^ neg ^ s.sb[c]) & 1u) ? -2 : 2);
            }
        }
    }
}

// S[x] (or D[x]) changes over winner v's row after its flip: 2 w s_v for
// neighbour x, times the neighbour's spin for int32 gains.  `neg`: v's new
// spin is -1; lo, hi: its row words.  `lanes` threads share the row (this one
// is `sub`).
//
// Compact rows are walked as aligned vectors of four entries, the next one
// loaded ahead, without a remainder: the padding entries change v itself by a
// known amount, which its flip takes out again (own_padding).
template <class DP, int kFmt>
__device__ __forceinline__ void scatter_row(const ChainSmem& s, const CsrView& csr, uint32_t lo, uint32_t hi,
                                            uint32_t neg, int sub, int lanes) {
    using C = Csr<kFmt>;
    if constexpr (C::kPlain) {
        uint32_t i = lo + sub;
        for (; i + 3 * lanes < hi; i += 4 * lanes) {
            int c[4], w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) C::entry(csr, i + j * lanes, c[j], w[j]);
            uint32_t x[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = DP::kField ? 0u : s.sb[c[j]] & 1u;
#pragma unroll
            for (int j = 0; j < 4; ++j) DP::add(s.D, c[j], (neg ^ x[j]) ? -2 * w[j] : 2 * w[j]);
        }
        for (; i < hi; i += lanes) {
            int c, w;
            C::entry(csr, i, c, w);
            const uint32_t x = DP::kField ? 0u : s.sb[c] & 1u;
            DP::add(s.D, c, (neg ^ x) ? -2 * w : 2 * w);
        }
    } else {
        uint32_t q = (lo >> 2) + sub;
        const uint32_t end = hi >> 2;
        if (q >= end) return;
        typename C::Vec e = C::vec(csr, q);
        for (q += lanes; q < end; q += lanes) {
            const typename C::Vec f = C::vec(csr, q);
            add_vec<DP, kFmt>(s, e, neg);
            e = f;
        }
        add_vec<DP, kFmt>(s, e, neg);
    }
}

// Two whole rows walked by one lane as one list: the lanes of a warp then wait
// for the longest pair, not for the longest row twice (mean degree 19: 13
// vectors for two rows of 5 instead of 16).  An absent row has equal words.
template <class DP, int kFmt>
__device__ __forceinline__ void scatter_two(const ChainSmem& s, const CsrView& csr, const uint32_t lo[2],
                                            const uint32_t hi[2], const uint32_t neg[2]) {
    using C = Csr<kFmt>;
    if constexpr (C::kPlain) {
        scatter_row<DP, kFmt>(s, csr, lo[0], hi[0], neg[0], 0, 1);
        scatter_row<DP, kFmt>(s, csr, lo[1], hi[1], neg[1], 0, 1);
    } else {
        const uint32_t n0 = (hi[0] >> 2) - (lo[0] >> 2), n = n0 + (hi[1] >> 2) - (lo[1] >> 2);
        const uint32_t at0 = lo[0] >> 2, at1 = (lo[1] >> 2) - n0;
        if (n == 0) return;
        typename C::Vec e = C::vec(csr, n0 ? at0 : at1);
        uint32_t ng = n0 ? neg[0] : neg[1];
        for (uint32_t i = 1; i < n; ++i) {
            const typename C::Vec f = C::vec(csr, i + (i < n0 ? at0 : at1));
            add_vec<DP, kFmt>(s, e, ng);
            e = f;
            ng = i < n0 ? neg[0] : neg[1];
        }
        add_vec<DP, kFmt>(s, e, ng);
    }
}

// What a walk of row `lo` adds to the row's own vertex through the padding:
// nothing but for 16-bit entries, whose padding weighs +1 (2 s_v to the field;
// to the gain, 2 s_v s_v).
template <class DP, int kFmt>
__device__ __forceinline__ int32_t own_padding(uint32_t lo, uint32_t neg) {
    if constexpr (Csr<kFmt>::kUnit) return static_cast<int32_t>(lo & 3u) * (DP::kField && neg ? -2 : 2);
    else return 0;
}

// Winner v (gain d, mask byte m before) flips: its stored value, its spin.
template <class DP>
__device__ __forceinline__ void flip_vertex(const ChainSmem& s, int v, int32_t d, uint32_t m) {
    DP::flip(s.D, v, d, m);
    atomicXor(&s.bits[v >> 5], 1u << (v & 31));
    s.sb[v] = static_cast<unsigned char>(m ^ 0xFFu);
}

// The best of a wider chain's 2, 4, 8 or 16 partials of one group, four loads in
// flight together.
__device__ __forceinline__ unsigned long long best_partial(const unsigned char* part, int warps) {
    unsigned long long best = 0;
    for (int w0 = 0; w0 < warps; w0 += 4) {
        unsigned long long p[4];
#pragma unroll
        for (int w = 0; w < 4; ++w)
            p[w] = w0 + w < warps ? *reinterpret_cast<const unsigned long long*>(part + (w0 + w) * kWarpScratch) : 0ull;
#pragma unroll
        for (int d = 1; d < 4; d *= 2) {
#pragma unroll
            for (int w = 0; w < 4; w += 2 * d) p[w] = p[w + d] > p[w] ? p[w + d] : p[w];
        }
        best = p[0] > best ? p[0] : best;
    }
    return best;
}

// FLIP on kPathWarp.  Row r = (t >> laneShift) + q T of the P winners is
// flipped by its first lane and walked by all 2^laneShift of them; v[q] comes
// from SELECT's registers (one-warp chains) or the warps' partials.  Returns
// this thread's part of sum(D before) - sum(D after), which is twice the cut
// gain once summed over the chain.  settle() (see run_chain) is called before
// the first flip, behind the loads that lead to it.
//
// With int8 gains nothing a row's walk reads is changed by another row (a
// flip adds +-1 to its own byte, a walk +-2w to its neighbours': they commute
// as 32-bit adds, whatever the bytes pass through on the way), so after the
// gains are read there is one barrier, at the end.  With int32 gains a walk
// reads its neighbours' new spins, so the flips are fenced off from the walks.
template <bool kOne, int kRows, class DP, int kFmt, class Loc, class Settle>
__device__ __forceinline__ Loc flip_rows(const ChainSmem& s, const CsrView& csr, const PhaseCfg& pc, int t, int T,
                                         int grp, int32_t v[4], Settle settle) {
    const int sub = t & ((1 << pc.laneShift) - 1);
    uint32_t lo[kRows], hi[kRows], neg[kRows];
    int32_t d[kRows];
    Loc loc = 0;
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
        lo[q] = hi[q] = neg[q] = 0;
        const int r = (t >> pc.laneShift) + q * T;
        if constexpr (kOne) {
            if (kRows == 1) {
                v[0] = __shfl_sync(0xFFFFFFFFu, v[0], r);
                if (r >= pc.P) v[0] = -1;
            } else if (q >= pc.rows) {
                v[q] = -1;
            }
        } else {
            unsigned long long p = 0;
            v[q] = -1;
            if (r < pc.P) {
                p = best_partial(reinterpret_cast<const unsigned char*>(s.slots) + 8 * r, T >> 5);
                const uint32_t low = static_cast<uint32_t>(p);
                if constexpr (DP::kField) {
                    v[q] = p ? static_cast<int32_t>(~(low >> 9) & 0x7FFFFFu) : -1;
                    neg[q] = ((low >> 8) & 1u) ^ 1u;
                    d[q] = static_cast<int32_t>(low & 0xFFu) - 128;
                } else {
                    v[q] = p ? static_cast<int32_t>(~low) : -1;
                }
            }
        }
        if (v[q] >= 0) {
            if (kOne || !DP::kField) {
                neg[q] = (s.sb[v[q]] & 1u) ^ 1u;
                d[q] = DP::get(s.D, s.sb, v[q]);
            }
            Csr<kFmt>::row(csr, v[q], lo[q], hi[q]);
            if (sub == 0) loc += d[q];
        }
    }
    settle();
    if (kOne || !DP::kField) __syncwarp();
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
        if (v[q] >= 0 && sub == 0) {
            if constexpr (DP::kField) {
                // q' = q - 1 (+1 -> -1) or q + 1: an add, as a neighbour's
                // walk may be adding to this byte.
                DP::add(s.D, v[q], (neg[q] ? -1 : 1) - own_padding<DP, kFmt>(lo[q], neg[q]));
                atomicXor(&s.bits[v[q] >> 5], 1u << (v[q] & 31));
                s.sb[v[q]] = neg[q] ? 0xFFu : 0u;
            } else {
                flip_vertex<DP>(s, v[q], d[q] + own_padding<DP, kFmt>(lo[q], neg[q]), neg[q] ? 0u : 0xFFu);
            }
        }
    }
    if (!DP::kField) group_sync(grp, T);
    if constexpr (kRows == 1) {
        scatter_row<DP, kFmt>(s, csr, lo[0], hi[0], neg[0], sub, 1 << pc.laneShift);
    } else {
#pragma unroll
        for (int q = 0; q < kRows; q += 2) scatter_two<DP, kFmt>(s, csr, lo + q, hi + q, neg + q);
    }
    group_sync(grp, T);
    if (kRows == 1 && pc.P == 1) return 2 * loc;   // a lone winner's gain just changes sign
#pragma unroll
    for (int q = 0; q < kRows; ++q)
        if (v[q] >= 0 && sub == 0) loc -= DP::get_as(s.D, neg[q], v[q]);
    return loc;
}

// P <= 128 over at least 32 (one-warp chains) or 64 threads: one to four rows,
// or one or two, a thread.
template <bool kOne, class DP, int kFmt, class Loc, class Settle>
__device__ __forceinline__ Loc flip_warp(const ChainSmem& s, const CsrView& csr, const PhaseCfg& pc, int t, int T,
                                         int grp, int32_t v[4], Settle settle) {
    if (pc.rows == 1) return flip_rows<kOne, 1, DP, kFmt, Loc>(s, csr, pc, t, T, grp, v, settle);
    if (!kOne || pc.rows == 2) return flip_rows<kOne, 2, DP, kFmt, Loc>(s, csr, pc, t, T, grp, v, settle);
    return flip_rows<kOne, 4, DP, kFmt, Loc>(s, csr, pc, t, T, grp, v, settle);
}


// FLIP of winners in the group slots (other paths, int64 scores; a barrier
// since SELECT's atomics has passed): publish and flip them, walk the rows,
// read the gains again.
template <class DP, int kFmt, bool kS64, class Loc>
__device__ __forceinline__ Loc flip_slots(const ChainSmem& s, const CsrView& csr, const PhaseCfg& pc, int t, int T,
                                          int grp) {
    Loc loc = 0;
    for (int gi = t; gi < pc.P; gi += T) {
        int v;
        if constexpr (kS64) {
            const int32_t id = s.ids[gi];
            v = (id == INT32_MAX) ? -1 : id;
            s.scores[gi] = LLONG_MIN;
            s.ids[gi] = INT32_MAX;
        } else {
            const unsigned long long k = s.slots[gi];
            s.slots[gi] = 0ull;
            v = k ? key_vertex(k) : -1;
        }
        s.win[gi] = v;
        if (v >= 0) {
            const int32_t d = DP::get(s.D, s.sb, v);
            loc += d;
            flip_vertex<DP>(s, v, d, s.sb[v]);
        }
    }
    group_sync(grp, T);
    const int lanes = 1 << pc.laneShift;
    for (int gi = t >> pc.laneShift; gi < pc.P; gi += T >> pc.laneShift) {
        const int v = s.win[gi];
        if (v >= 0) {
            uint32_t lo, hi;
            Csr<kFmt>::row(csr, v, lo, hi);
            const uint32_t neg = s.sb[v] & 1u;
            const int sub = t & (lanes - 1);
            // Past the barrier only: the plain byte stores above do not mix
            // with an add that may carry through a neighbouring byte.
            if (sub == 0 && Csr<kFmt>::kUnit) DP::add(s.D, v, -own_padding<DP, kFmt>(lo, neg));
            scatter_row<DP, kFmt>(s, csr, lo, hi, neg, sub, lanes);
        }
    }
    group_sync(grp, T);
    for (int gi = t; gi < pc.P; gi += T) {
        const int v = s.win[gi];
        if (v >= 0) loc -= DP::get(s.D, s.sb, v);
    }
    return loc;
}

// ------------------------------------------------------------------ chain
// Pacing between the chains of one CTA.  The warp scheduler does not share
// issue slots evenly, so chains of one item drift apart within a window (by
// up to ~40% of it measured on GB300), and the CTA then runs its last chains
// with few warps while the others wait at the item barrier.  Every
// kPaceEvery sweeps a chain publishes its progress; one more than kPaceLead
// sweeps ahead of the slowest chain of its CTA yields its issue slots with
// short sleeps (bounded: at most kPaceSleeps of them per check).
constexpr int kPaceEvery = 32;
constexpr int kPaceLead = 64;
constexpr int kPaceSleeps = 32;

// The CTA header holds the pacing state: progress of each warp group at
// bytes 160..223, the number of running groups at 224.
__device__ __forceinline__ volatile int* pace_state() {
    extern __shared__ __align__(128) unsigned char smem[];
    return reinterpret_cast<volatile int*>(smem + 160);
}

__device__ __forceinline__ int slowest_chain(const volatile int* prog) {
    const int active = prog[16];
    int m = INT_MAX;
    for (int q = 0; q < active; ++q) m = min(m, prog[q]);
    return m;
}

template <bool kOne, class DP, int kFmt, bool kS64>
__device__ void run_chain(const DevLaunch& L, const ChainSmem& s, const CsrView& csr,
                          const int32_t* lut, int ci, int t, int threads, int grp) {
    const int T = kOne ? 32 : threads;
    volatile int* prog = pace_state();
    DevChain& ch = L.chains[ci];
    if (uniform(static_cast<int>(ch.sweepsDone >= ch.sweepsTotal && ch.cur != kUnsetCut))) {
        if (t == 0) prog[grp] = INT_MAX;
        return;
    }
    const DevGraph& g = L.graphs[uniform(ch.graph)];
    DevSchedule sch = L.scheds[uniform(ch.sched)];
    sch.phaseP = uniform(sch.phaseP);
    sch.phaseIters = uniform(sch.phaseIters);
    sch.nphases = uniform(sch.nphases);
    const int n = uniform(g.n);
    const int words = (n + 31) >> 5;

    // ---- state in: spin bits and best bits; empty group slots
    const bool fresh = uniform(static_cast<int>(ch.cur == kUnsetCut));
    for (int w = t; w < words; w += T) {
        const uint32_t sb = ch.spinBits[w];
        s.bits[w] = sb;
        s.best[w] = fresh ? sb : ch.bestBits[w];
    }
    if (L.layout != kLayoutMain) {
        for (int i = t; i < L.pmax; i += T) {
            s.slots[i] = kS64 ? static_cast<unsigned long long>(LLONG_MIN) : 0ull;
            s.ids[i] = INT32_MAX;
        }
    }
    group_sync(grp, T);
    const int nPad = (n + 7) & ~7;
    for (int v = t; v < nPad; v += T)
        s.sb[v] = (v < n && !spin_of(s.bits, v)) ? 0xFFu : 0u;
    group_sync(grp, T);

    // ---- D[v] = spin[v] * sum_u w(v,u) spin[u]; padding past n is 0
    int64_t dsum = 0;
    for (int v = t; v < nPad; v += T) {
        int32_t d = 0;
        if (v < n) {
            uint32_t lo, hi;
            Csr<kFmt>::entries(csr, v, lo, hi);
            int32_t acc = 0;
            for (uint32_t i = lo; i < hi; ++i) {
                int col, w;
                Csr<kFmt>::entry(csr, i, col, w);
                acc += s.sb[col] ? -w : w;
            }
            d = s.sb[v] ? -acc : acc;
            dsum += d;
        }
        DP::set(s.D, s.sb, v, d);
    }
    // cut = (sum over directed entries of w - sum_v D[v]) / 4, exactly.
    const int64_t cutD = (g.wsum2 - group_sum(dsum, s, t, T, grp)) / 4;
    int64_t cur = uniform(ch.cur);
    int64_t best = uniform(ch.best);
    if (fresh) {
        cur = best = uniform(cutD);
    } else if (cur != cutD) {
        if (t == 0) raise_error(L, kDevCutMismatch, ci);
    }

    // ---- window, beta cursor (first run with end > s0), phase cursor
    const uint64_t s0 = uniform(ch.sweepsDone);
    const uint64_t sEnd = uniform(ch.sweepsTotal);
    const uint64_t s1 = (sEnd - s0 > L.window) ? s0 + L.window : sEnd;
    int64_t run = 0;
    {
        int64_t lo = 0, hi = ch.betaRuns;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (static_cast<uint64_t>(ch.betaEnd[mid]) > s0) hi = mid; else lo = mid + 1;
        }
        run = uniform(lo);
    }
    if (s1 > s0 && (run >= ch.betaRuns ||
                    static_cast<uint64_t>(ch.betaEnd[ch.betaRuns - 1]) < s1)) {
        if (t == 0) {
            raise_error(L, kDevBetaTable, ci);
            prog[grp] = INT_MAX;
        }
        return;
    }
    int p = 0;
    uint64_t phaseEnd = 0;
    int P = 1;
    {
        uint64_t acc = 0;
        for (p = 0; p < sch.nphases; ++p) {
            if (uniform(sch.phaseP[p]) == 0) continue;
            const uint64_t iters = uniform(sch.phaseIters[p]);
            if (acc + iters > s0) break;
            acc += iters;
        }
        if (p < sch.nphases) {
            phaseEnd = acc + uniform(sch.phaseIters[p]);
            P = static_cast<int>(umin(uniform(sch.phaseP[p]), static_cast<uint32_t>(n)));
        }
    }
    // The last beta run holds the schedule's largest beta.
    const int kbMax = kS64 ? 31 : uniform(key_room(__ldg(ch.betaVal + ch.betaRuns - 1), g.B));
    const bool slotsOnly = kS64 || L.layout == kLayoutSlots;
    const bool table = L.layout != kLayoutMain;
    PhaseCfg pc = phase_cfg(P, n, t, T, kOne, kbMax, slotsOnly);
    KeyCfg kc = key_cfg(n, pc.S, t, lut);
    if (!table && (pc.path != kPathWarp || pc.shares != 0)) {
        // The host plans a table for every schedule that needs one.
        if (t == 0) {
            raise_error(L, kDevBadItem, ci);
            prog[grp] = INT_MAX;
        }
        return;
    }

    const ChainKeys keys = make_keys(ch.solverSeed);
    // Beta cursor: lane l holds run `run` + l of the table (the last runs' ends
    // are past the window), loaded a segment of sweeps ahead.
    const int lane = t & 31;
    const int64_t* __restrict__ bEnd = uniform(ch.betaEnd);
    const int32_t* __restrict__ bVal = uniform(ch.betaVal);
    const int64_t nRuns = uniform(ch.betaRuns);
    uint64_t runEnd = ~uint64_t(0);
    int32_t runVal = 0;
    auto load_runs = [&]() {
        runEnd = ~uint64_t(0);
        if (run + lane < nRuns) {
            runEnd = static_cast<uint64_t>(__ldg(bEnd + run + lane));
            runVal = __ldg(bVal + run + lane);
        }
    };
    load_runs();
    uint64_t improved = 0;
    using Loc = typename std::conditional<DP::kField, int32_t, int64_t>::type;
    // The last sweep's gain is settled when the next one is about to flip (or
    // at the window's end): the loads and the warp sum behind it overlap
    // SELECT, and wider chains pass the warps' sums through s.red under
    // SELECT's own barrier instead of one more.
    Loc loc = 0;
    // The cut as its distance below the best, in a gain's type.  With int8 gains no
    // two cuts of a graph are n B / 2 apart, below 2^23 (B <= 127, and a chain's
    // shared memory holds fewer than 2^17 vertices), so that it is exact in int32;
    // a best further off than 2^30 cannot be one, and is never reached.
    constexpr int64_t kFar = DP::kField ? int64_t(1) << 30 : INT64_MAX / 2;
    Loc behind = static_cast<Loc>(best < cur - kFar ? -kFar : best > cur + kFar ? kFar : best - cur);
    int64_t top = cur + behind;
    auto settle = [&]() {
        Loc gain;
        if constexpr (kOne) gain = warp_sum(loc);
        else gain = warp_sum(static_cast<Loc>((t & 31) < (T >> 5) ? s.red[t & 31] : 0));
        behind -= gain >> 1;
        if (behind < 0) {
            top -= behind;
            behind = 0;
            ++improved;
            for (int w = t; w < words; w += T) s.best[w] = s.bits[w];
            group_sync(grp, T);
        }
    };
    group_sync(grp, T);   // s.red is read
    if (t < (T >> 5)) s.red[t] = 0;
    group_sync(grp, T);

    uint64_t sw = s0;
    SweepConst sc = make_sweep(s0 + 1, keys);   // the sweep id is 1-based
    while (sw < s1) {
        if (sw >= phaseEnd) {
            while (sw >= phaseEnd) {
                ++p;
                if (p >= sch.nphases) break;
                if (uniform(sch.phaseP[p]) == 0) continue;
                phaseEnd += uniform(sch.phaseIters[p]);
                P = static_cast<int>(umin(uniform(sch.phaseP[p]), static_cast<uint32_t>(n)));
            }
            const bool warp = pc.path == kPathWarp;
            pc = phase_cfg(P, n, t, T, kOne, kbMax, slotsOnly);
            kc = key_cfg(n, pc.S, t, lut);
            if (!table && (pc.path != kPathWarp || pc.shares != 0)) {
                if (t == 0) raise_error(L, kDevBadItem, ci);
                break;
            }
            if (warp && pc.path != kPathWarp) {
                // The slots held scratch and partials: empty them (all their
                // readers are past the last sweep's barrier).
                for (int i = t; i < L.pmax; i += T) s.slots[i] = 0ull;
                group_sync(grp, T);
            }
        }
        const uint32_t paced = static_cast<uint32_t>(sw - s0) & (kPaceEvery - 1);
        if (paced == 0) {
            const int mine = static_cast<int>(sw - s0);
            if (t == 0) prog[grp] = mine;
            int lead = mine - slowest_chain(prog);
            for (int q = 0; q < kPaceSleeps && lead > kPaceLead; ++q) {
                __nanosleep(2000);
                lead = mine - slowest_chain(prog);
            }
        }
        // Sweeps up to the next pacing point, end of phase or of the window.
        uint32_t left = kPaceEvery - paced;
        if (phaseEnd > sw && phaseEnd - sw < left) left = static_cast<uint32_t>(phaseEnd - sw);
        if (s1 - sw < left) left = static_cast<uint32_t>(s1 - sw);
        // Their betas, one to a lane: sweep sw + l takes the first run that ends
        // past it (runs are never empty, so that is one of the 32 at hand).
        // A beta lasts one sweep for most of a schedule (t0 = 35: until sweep
        // 30,000).  Against a cursor that moved with the sweeps (two loads, three
        // warp reductions and 64-bit compares a run), GB300, us per sweep at P =
        // 1: 32 chains of ER n = 800 1.165 / 1.081, four one-warp chains of ER n =
        // 256 0.858 / 0.782, 1024 of ER n = 2000 2.09 / 1.98; 80 of the 100x200
        // torus 2.91 / 2.76.
        int32_t betas;
        {
            const uint64_t room = runEnd - sw;
            const uint32_t ends = room < 64 ? static_cast<uint32_t>(room) : 64u;
            int at = 0;
#pragma unroll
            for (int step = 16; step; step >>= 1)
                if (__shfl_sync(0xFFFFFFFFu, ends, at + step - 1) <= static_cast<uint32_t>(lane)) at += step;
            betas = __shfl_sync(0xFFFFFFFFu, runVal, at);
            run += __popc(__ballot_sync(0xFFFFFFFFu, ends <= left));
            load_runs();
        }
        const uint32_t segment = left;
        do {
            const int32_t beta = __shfl_sync(0xFFFFFFFFu, betas, static_cast<int>(segment - left));
            int32_t v[4];
            if constexpr (kS64) select64<DP>(s, lut, n, pc, beta, sc, keys, t, T, grp);
            else select32<kOne, DP>(s, lut, kc, n, pc, beta, sc, keys, t, T, v);
            ++sw;
            sc = make_sweep(sw + 1, keys);
            const bool slots = kS64 || pc.path != kPathWarp;
            if (!kOne || slots) group_sync(grp, T);
            if (slots) {
                settle();
                loc = flip_slots<DP, kFmt, kS64, Loc>(s, csr, pc, t, T, grp);
            } else {
                loc = flip_warp<kOne, DP, kFmt, Loc>(s, csr, pc, t, T, grp, v, settle);
            }
            if (!kOne) {
                loc = warp_sum(loc);
                if ((t & 31) == 0) s.red[t >> 5] = loc;
            }
        } while (--left);
    }
    if (!kOne) group_sync(grp, T);
    settle();
    if (t == 0) prog[grp] = INT_MAX;
    group_sync(grp, T);

    // ---- state out
    for (int w = t; w < words; w += T) {
        ch.spinBits[w] = s.bits[w];
        ch.bestBits[w] = s.best[w];
    }
    if (t == 0) {
        ch.cur = top - behind;
        ch.best = best > top ? best : top;
        ch.sweepsDone = s1;
        ch.improvedSweeps += improved;
    }
}

// ------------------------------------------------------------ bulk copy
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* mbar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* mbar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(mbar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* mbar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(mbar))
        : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* mbar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_addr(mbar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Stage graph g's row words and compact entries (kUnit: 16 bits, else 32) into
// shared memory: thread 0 arms the mbarrier with the byte count and issues the
// bulk copies (<= 64 KB each); every thread waits on the phase with a bounded
// poll.  Returns this thread's outcome (false: its polls ran out); the caller
// makes it CTA-uniform and advances the phase.
template <bool kUnit>
__device__ bool stage_csr(const DevGraph& g, unsigned char* dst, uint64_t* mbar, uint32_t phase) {
    const uint32_t entBytes = kUnit ? g.u16Bytes : g.p32Bytes;
    const uint32_t total = g.rowBytes + entBytes;
    if (threadIdx.x == 0) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(mbar, total);
        const unsigned char* srcs[2] = {reinterpret_cast<const unsigned char*>(g.rows),
                                        kUnit ? reinterpret_cast<const unsigned char*>(g.u16)
                                              : reinterpret_cast<const unsigned char*>(g.p32)};
        const uint32_t sizes[2] = {g.rowBytes, entBytes};
        uint32_t o = 0;
        for (int k = 0; k < 2; ++k) {
            for (uint32_t c = 0; c < sizes[k]; c += 65536u) {
                const uint32_t len = (sizes[k] - c < 65536u) ? (sizes[k] - c) : 65536u;
                bulk_g2s(dst + o + c, srcs[k] + c, len, mbar);
            }
            o += sizes[k];
        }
    }
    bool ok = false;
    for (int i = 0; i < kMaxCopyPolls && !ok; ++i) ok = mbar_try_wait(mbar, phase);
    return ok;
}

// kDBytes: 1 -> D8, 4 -> D32.  kOne: chains of one warp, whose barriers are
// __syncwarp and whose winners stay in registers; a kernel of its own, as both
// forms in one do not fit 128 registers (they spill ~200 bytes).  The int64
// score path is one kernel for every width.
template <int kDBytes, int kFmt, bool kS64, bool kOne>
__global__ void __launch_bounds__(512, 1) rfmf_anneal_kernel(const DevLaunch L) {
    using DP = typename std::conditional<kDBytes == 1, D8, D32>::type;
    extern __shared__ __align__(128) unsigned char smem[];
    int32_t* lut = reinterpret_cast<int32_t*>(smem);                 // 64 B
    uint64_t* mbar = reinterpret_cast<uint64_t*>(smem + 128);        // 8 B
    int* sItem = reinterpret_cast<int*>(smem + 144);
    volatile int* sProg = pace_state();   // 16 progress words + running-group count
    unsigned char* csrBase = smem + kSmemHeader;
    unsigned char* chainBase = csrBase + L.csrBytes;

    const int T = kOne ? 32 : 32 * L.warpsPerChain;
    const int grp = uniform(static_cast<int>(threadIdx.x) / T);
    const int t = threadIdx.x - grp * T;
    const ChainSmem cs = carve_chain(chainBase + static_cast<size_t>(grp) * L.chainBytes, L, kDBytes);

    if (threadIdx.x < 16) lut[threadIdx.x] = L.lut[threadIdx.x];
    if (!csr_in_hbm(kFmt) && threadIdx.x == 0) mbar_init(mbar);
    __syncthreads();

    uint32_t phase = 0;
    int loaded = -1;
    for (;;) {
        if (threadIdx.x == 0) *sItem = atomicAdd(L.queue, 1);
        __syncthreads();
        const int it = uniform(*sItem);
        if (it >= L.nitems) break;
        DevItem item = L.items[it];
        item.graph = uniform(item.graph);
        item.first = uniform(item.first);
        item.count = uniform(item.count);
        if (item.graph < 0 || item.graph >= L.ngraphs) {
            if (threadIdx.x == 0) raise_error(L, kDevBadItem, it);
            __syncthreads();
            continue;
        }
        uint64_t t0 = 0;
        if (threadIdx.x == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
        const DevGraph& g = L.graphs[item.graph];
        CsrView csr;
        if constexpr (csr_in_hbm(kFmt)) {
            csr.off = (kFmt == kCsrGlobal) ? g.offsets : g.rows;
            csr.ent = (kFmt == kCsrGlobal)    ? static_cast<const void*>(g.edges)
                      : Csr<kFmt>::kUnit ? static_cast<const void*>(g.u16)
                                         : static_cast<const void*>(g.p32);
        } else {
            if (item.graph != loaded) {
                // All threads agree on the outcome, so that a chain's
                // barriers never see part of its warp group leave.
                if (!__syncthreads_and(stage_csr<Csr<kFmt>::kUnit>(g, csrBase, mbar, phase))) {
                    // The copy may still be in flight.  Report it, then stay
                    // resident for a second, longer bounded wait: a CTA that
                    // retired with a copy outstanding would leave its target
                    // shared memory to whatever CTA the SM runs next.  The
                    // CTA then takes no more work; the host reports the error
                    // and the context is not to be reused.
                    if (threadIdx.x == 0) raise_error(L, kDevCopyTimeout, it);
                    bool landed = false;
                    for (int i = 0; i < 4 * kMaxCopyPolls && !landed; ++i) landed = mbar_try_wait(mbar, phase);
                    __syncthreads();
                    break;
                }
                phase ^= 1u;
                loaded = item.graph;
            }
            csr.off = reinterpret_cast<const uint32_t*>(csrBase);
            csr.ent = csrBase + g.rowBytes;
        }
        const int active = (item.count < L.chainsPerCta) ? item.count : L.chainsPerCta;
        if (threadIdx.x < 16) sProg[threadIdx.x] = (static_cast<int>(threadIdx.x) < active) ? 0 : INT_MAX;
        if (threadIdx.x == 0) sProg[16] = active;
        __syncthreads();
        if (grp < active) {
            const int ci = uniform(L.order[item.first + grp]);
            run_chain<kOne, DP, kFmt, kS64>(L, cs, csr, lut, ci, t, T, grp);
        }
        __syncthreads();
        if (threadIdx.x == 0 && L.itemNs) {
            uint64_t t1;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
            L.itemNs[it] = t1 - t0;
        }
    }
}

}  // namespace

// ------------------------------------------------------------ host hooks
// Kernel variants: D width {1, 4} x CSR format {unit16, packed32, HBM 8-byte,
// HBM 16-bit, HBM 32-bit} x {int32 scores one-warp, int32 scores wider, int64
// scores}.  The two D widths compile as two translation units (this file, and
// rfmf_anneal_i32.cu, which includes it), side by side.
namespace {
template <int DB, bool S, bool One>
const void* kernel_for_format(int fmt) {
    switch (fmt) {
        case kCsrUnit16: return reinterpret_cast<const void*>(&rfmf_anneal_kernel<DB, kCsrUnit16, S, One>);
        case kCsrPacked32: return reinterpret_cast<const void*>(&rfmf_anneal_kernel<DB, kCsrPacked32, S, One>);
        case kCsrGlobal16: return reinterpret_cast<const void*>(&rfmf_anneal_kernel<DB, kCsrGlobal16, S, One>);
        case kCsrGlobal32: return reinterpret_cast<const void*>(&rfmf_anneal_kernel<DB, kCsrGlobal32, S, One>);
        default: return reinterpret_cast<const void*>(&rfmf_anneal_kernel<DB, kCsrGlobal, S, One>);
    }
}

template <int DB>
const void* kernel_for(int fmt, bool s64, int warps) {
    if (s64) return kernel_for_format<DB, true, false>(fmt);
    return warps == 1 ? kernel_for_format<DB, false, true>(fmt) : kernel_for_format<DB, false, false>(fmt);
}
}  // namespace

#if RFMF_GAIN_BYTES == 4
const void* kernel_ptr_i32(int fmt, bool s64, int warps) { return kernel_for<4>(fmt, s64, warps); }
#else
const void* kernel_ptr_i32(int fmt, bool s64, int warps);

const void* kernel_ptr(int dbytes, int fmt, bool s64, int warps) {
    return dbytes == 1 ? kernel_for<1>(fmt, s64, warps) : kernel_ptr_i32(fmt, s64, warps);
}

// Rows walked in HBM pass through the L1 that the SM's chains leave: a launch
// that has the GPU to itself (sms > 0) asks for no more shared memory than its
// resident CTAs hold, as otherwise 28 KB of L1 are left whatever they hold.
// GB300, 28 KB / as asked: 150 chains of a planar graph n = 3000 in 8-byte pairs
// 17.0 / 16.1 ms, 16 graphs n 807..14,000 x 48 44.7 / 42.0, 80 of the 100x200
// torus 52.8 / 52.1; ER n = 5000 x 256 at P = 128 2.88 / 2.40 us per sweep, full
// SMs the same.
cudaError_t launch_anneal(const DevLaunch& L, int dbytes, int fmt, bool s64, int grid,
                          int threads, size_t smem, cudaStream_t stream, int sms) {
    void* args[] = {const_cast<DevLaunch*>(&L)};
    cudaLaunchAttribute split{};
    split.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    if (sms > 0 && csr_in_hbm(fmt)) {
        constexpr size_t kSmBytes = 228 << 10, kCtaBytes = 1 << 10;   // shared memory of an SM; a CTA's own part
        const size_t held = static_cast<size_t>((grid + sms - 1) / sms) * (smem + kCtaBytes);
        split.val.sharedMemCarveout = static_cast<unsigned>(held < kSmBytes ? (100 * held + kSmBytes - 1) / kSmBytes : 100);
        cfg.attrs = &split;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelExC(&cfg, kernel_ptr(dbytes, fmt, s64, L.warpsPerChain), args);
}
#endif

}  // namespace rfmf
