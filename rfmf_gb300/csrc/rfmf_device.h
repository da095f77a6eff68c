// rfmf_device.h -- structures shared by the host driver and the sm_103a
// kernels.  Plain C++ (no CUDA headers) so the host .cpp can include it.
#ifndef RFMF_DEVICE_H
#define RFMF_DEVICE_H

#include <climits>
#include <cstdint>

namespace rfmf {

// One directed CSR entry: neighbour id and weight, loaded as one 8-byte word.
struct alignas(8) Edge {
    int32_t col;
    int32_t w;
};

// How a launch reads the CSR.  The compact formats are copied once per CTA
// into shared memory (bulk async copy) and walked there; the HBM formats walk
// the graph's own arrays through L1/L2 (graphs too large for shared memory
// beside their chains), with the most compact entries the graph allows.
enum CsrFormat : int32_t {
    kCsrUnit16 = 0,    // uint16 entry = col | (w < 0) << 15; |w| == 1, n <= 32768
    kCsrPacked32 = 1,  // uint32 entry = (w << 16) | col;  |w| < 2^15, n <= 65536
    kCsrGlobal = 2,    // Edge {col, w} in HBM
    kCsrGlobal16 = 3,  // the unit16 entries, in HBM
    kCsrGlobal32 = 4,  // the packed32 entries, in HBM
};

#if defined(__CUDACC__)
#define RFMF_CHD __host__ __device__ constexpr
#else
#define RFMF_CHD constexpr
#endif
// Formats walked in HBM (no shared-memory copy of the CSR).
RFMF_CHD bool csr_in_hbm(int fmt) { return fmt == kCsrGlobal || fmt == kCsrGlobal16 || fmt == kCsrGlobal32; }

// The compact formats keep every row at a multiple of four entries, so that a
// row is read as aligned vectors of four: row word r of vertex v holds its
// first entry (a multiple of four) and, in the low two bits, how many of its
// last vector's entries are padding (0..3); its vectors end where row v + 1's
// begin.  Padding entries name vertex v itself, with weight +1 (16-bit) or 0
// (32-bit).
//
// One CSR graph in HBM, read-only, shared by every chain that anneals it.
// Rows are sorted ascending by neighbour (the reference's AnnealCsr order,
// src/immutable_graph.hpp:83-101); each undirected edge is stored twice.
struct DevGraph {
    const uint32_t* offsets;   // n + 1 (padded to 16 B)
    const Edge*     edges;     // 2m  {col, weight}
    const uint32_t* rows;      // n + 1 row words of the compact entries (padded to 16 B)
    const uint16_t* u16;       // compact entries by width, rows padded to four (16 B in all); null: the
    const uint32_t* p32;       //   graph has none.  A record serves every format, as launches of several
                               //   formats may share it
    int32_t         n;
    int32_t         words;     // ceil(n / 32): spin bit-words per chain
    int64_t         B;         // max weighted degree: no gain exceeds it
    int64_t         wsum2;     // sum of weight over directed entries (2 * sum over edges)
    uint32_t        rowBytes;  // bytes of rows, multiple of 16
    uint32_t        u16Bytes;  // bytes of u16 and of p32, multiples of 16
    uint32_t        p32Bytes;
};

// One schedule: phases (group counts P) and sweeps per phase, shared by the
// chains that reference it.  Phases with P == 0 are skipped without
// advancing the sweep counter (src/anneal_kernels.cu:272).
struct DevSchedule {
    const uint32_t* phaseP;
    const uint64_t* phaseIters;
    int32_t         nphases;
    int32_t         pad;
};

// One chain.  Its state (spin bits, best-spin bits, current and best cut,
// progress) lives in HBM between launches and in shared memory while a
// warp group runs it.
struct DevChain {
    int32_t         graph;        // index into the graph table
    int32_t         sched;        // index into the schedule table
    uint64_t        solverSeed;   // Philox key (seed + kSolverSeedOffset)
    const int64_t*  betaEnd;      // run-length beta table, 0-based exclusive ends
    const int32_t*  betaVal;      //   (one table per distinct t0)
    int64_t         betaRuns;
    uint32_t*       spinBits;     // words(graph) words, bit v = (spin[v] > 0)
    uint32_t*       bestBits;     // words(graph) words
    int64_t         cur;          // in/out: cut value of spinBits
    int64_t         best;         // in/out: cut value of bestBits
    uint64_t        sweepsDone;   // executed sweeps so far (in/out)
    uint64_t        sweepsTotal;  // executed sweeps of the whole schedule
    uint64_t        improvedSweeps;  // sweeps that raised the best cut (statistic)
};

// One work item of the persistent kernel: up to K chains of ONE graph, run
// side by side by the K warp groups of a CTA on one shared-memory copy of
// the graph.  The chains are order[first .. first + count).
struct DevItem {
    int32_t graph;
    int32_t first;
    int32_t count;
    int32_t pad;
};

// Error word written by the kernel (0 = ok).  The kernel never traps: it
// records the first problem it sees and lets the CTA finish.
enum DevError : int32_t {
    kDevOk = 0,
    kDevCutMismatch = 1,     // carried cut value disagrees with the spins
    kDevBetaTable = 2,       // beta table shorter than the window
    kDevBadItem = 3,         // graph/schedule index out of range
    kDevCopyTimeout = 4,     // bulk copy of the CSR did not complete in time
    kDevBadInput = 5,        // a caller's device CSR failed the on-device check
};

// Launch-wide parameters.
struct DevLaunch {
    const DevGraph*    graphs;
    const DevSchedule* scheds;
    DevChain*          chains;
    const DevItem*     items;
    const int32_t*     order;       // chain indices grouped by item
    int32_t            nitems;
    int32_t            ngraphs;
    int32_t            nscheds;
    int32_t            warpsPerChain;   // W: threads per chain = 32 W
    int32_t            chainsPerCta;    // K: warp groups per CTA
    int32_t            maxN;            // largest n (sizes the per-chain gain array)
    int32_t            maxWords;        // largest spin word count
    int32_t            pmax;            // group slots per chain: min(max P, max n)
    uint32_t           csrBytes;        // shared-memory CSR region (0 for kCsrGlobal)
    uint32_t           chainBytes;      // shared-memory bytes per chain
    int32_t            layout;          // which per-chain arrays there are (LayoutKind)
    int32_t*           queue;       // work-queue head (zeroed before the launch)
    int32_t*           error;       // first device error (DevError)
    int32_t*           errorItem;   // chain/item that raised it
    uint64_t*          itemNs;      // per item: device time the CTA spent on it (ns)
    uint64_t           window;      // sweeps each chain advances in this launch
    int32_t            lut[16];     // Q20 Gumbel quantile table
};

// cur == kUnsetCut on input: the kernel derives the cut of spinBits itself
// and starts bestBits/best from it (a fresh chain).
constexpr int64_t kUnsetCut = INT64_MIN;

// Shared-memory header in front of the CSR region: Gumbel table (64 B),
// bulk-copy mbarrier, work-item slot, chain pacing state (bytes 160..227).
constexpr uint32_t kSmemHeader = 256;

#if defined(__CUDACC__)
#define RFMF_HD __host__ __device__ __forceinline__
#else
#define RFMF_HD inline
#endif

RFMF_HD uint32_t align16(uint32_t x) { return (x + 15u) & ~15u; }

// Per-chain shared-memory region, in order: gains D (nPad * dbytes), spin
// bits, best-spin bits, spins as mask bytes (0x00 / 0xFF), group key slots
// (8 B per group, or the warps' argmax scratch and partials), ids (4 B),
// winners (4 B), reduction partials (8 B per warp).
// Host and kernel both carve with this.
struct ChainLayout {
    uint32_t d, bits, best, sb, slots, ids, win, red, total;
};

// Argmax scratch of one warp: 256 keys in two halves 16 banks apart, reused
// for up to 128 partials of 8 bytes.
constexpr uint32_t kWarpScratch = (144 + 128) * 4;

// What a chain's region holds besides its state.  The group table (slots
// aside: ids and winners) serves the phases off the kernel's main path; the
// argmax scratch the int32 score path.
enum LayoutKind : int32_t {
    kLayoutMain = 0,    // scratch only: every phase has 256 % P == 0, P <= 128
    kLayoutAny = 1,     // scratch and table
    kLayoutSlots = 2,   // table only: int64 scores, and chains that fit a CTA only so;
                        // every phase goes through the group slots
};

// Whether a phase of P groups (clamped to n) runs on the main path.
RFMF_HD bool main_phase(uint32_t P, int n) {
    const uint32_t p = P < static_cast<uint32_t>(n) ? P : static_cast<uint32_t>(n);
    return p == 0 || (p <= 128 && 256 % p == 0);
}

RFMF_HD ChainLayout chain_layout(int maxN, int maxWords, int pmax, int warps, int dbytes, int kind) {
    ChainLayout c;
    const uint32_t nPad = (static_cast<uint32_t>(maxN) + 7u) & ~7u;
    uint32_t o = 0;
    c.d = o;     o = align16(o + nPad * static_cast<uint32_t>(dbytes));
    c.bits = o;  o = align16(o + static_cast<uint32_t>(maxWords) * 4u);
    c.best = o;  o = align16(o + static_cast<uint32_t>(maxWords) * 4u);
    c.sb = o;    o = align16(o + nPad);
    const uint32_t scratch = kind == kLayoutSlots ? 0u : static_cast<uint32_t>(warps) * kWarpScratch;
    const uint32_t groups = kind == kLayoutMain ? 0u : static_cast<uint32_t>(pmax), slots = groups * 8u;
    c.slots = o; o = align16(o + (slots > scratch ? slots : scratch));
    c.ids = o;   o = align16(o + groups * 4u);
    c.win = o;   o = align16(o + groups * 4u);
    c.red = o;   o = align16(o + static_cast<uint32_t>(warps) * 8u);
    c.total = o;
    return c;
}

}  // namespace rfmf

#endif  // RFMF_DEVICE_H
