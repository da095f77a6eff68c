// rfmf_ingest.cu -- graph ingest and output path of librfmf.so.
//
// Ingest (reference: src/read_gset.cpp:61-201 parseAndScale +
// read_instance_from_stream, src/graph.cpp addEdge, src/immutable_graph.hpp:
// 44-120 ImmutableGraph::build):
//   * rfmf_gset_header / rfmf_gset_parse: native parser of Gset/MQLib text
//     with the reference's rules (comment and blank lines skipped, header
//     "N M", M edge lines "u v w", power-of-ten scaling when a weight is
//     fractional, zero weights dropped after rounding);
//   * rfmf_graph_from_edges: the CSR built ON THE DEVICE from an edge list --
//     undirected duplicates keep their first weight, vertices are the
//     endpoints of the surviving edges renumbered densely in ascending
//     original id, every row sorted ascending -- then the compact shared-memory
//     entry formats, B and the weight sum, all without a host CSR.
//     Steps: one pass checks the edges and finds the largest id; endpoint
//     presence marks and an exclusive scan give the dense ids; a degree
//     histogram and scan give row starts; every edge puts one 8-byte key
//     (neighbour, input index) in each of its two rows; a warp sorts each row
//     by counting ranks (rows above 2048 entries: tiles, merged), so the first
//     occurrence of a duplicate leads its run;
//     the first of each run is emitted in every entry format.
// Output (reference: src/max_cut.cpp:5-15 cutValueCsr and the
// Solution-*-partition: lines of src/host_common.cpp:412-422):
//   * rfmf_batch_cuts: every chain's cut recomputed on the device from its
//     end or best spins;
//   * rfmf_batch_partitions: the '0'/'1' partition strings of every chain
//     expanded on the device.
#include <cuda_runtime.h>

#include <algorithm>
#include <cerrno>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <memory>
#include <new>
#include <utility>
#include <vector>

#include "rfmf_host.h"

using namespace rfmf;

// ======================================================================
// Gset / MQLib text parser (host)
// ======================================================================
// The text format and the weight rule this parser implements (the loader
// behaviour of src/read_gset.cpp:61-170, restated):
//   * lines end at '\n'; a line that is empty after leading spaces, tabs and
//     CRs, or whose first such character is '#', carries no data;
//   * the first data line holds N and M (integers >= 0), the next M data
//     lines one edge each: two integer ids and a real weight, any further
//     text on the line ignored;
//   * weights that are all integral (w == floor(w), |w| < 2^53) are used
//     as they are.  Otherwise every weight is multiplied by one power of
//     ten s = 10^k, k in 12..-12, the largest for which A s + D / 2 stays
//     within a budget and W s within (2^31 - 1) / 2, where W is the largest
//     |w|, and over the ids of the edge lines, A the largest sum of |w| of
//     an id's lines and D the largest number of line ends at one id.  The
//     budget is (2^31 - 1) / 4, or (2^63 - 1) / 8 when no k meets the first;
//     no k at all, or W s < 1/2 (every weight would round to zero), is an
//     error.  Scaled weights are rounded to the nearest integer, halves away
//     from zero;
//   * edges whose integer weight is 0 are dropped and counted; the others
//     are returned in file order, duplicates included.
// A forced scale s > 0 replaces the choice and its two checks.
namespace {

// Data lines of the text as [begin, end) spans, in order.
std::vector<std::pair<const char*, const char*>> data_lines(const char* text, size_t len) {
    std::vector<std::pair<const char*, const char*>> out;
    const char* const stop = text + len;
    for (const char* cur = text; cur < stop;) {
        const char* nl = static_cast<const char*>(std::memchr(cur, '\n', static_cast<size_t>(stop - cur)));
        const char* lineEnd = nl ? nl : stop;
        const char* first = cur;
        while (first < lineEnd && (*first == ' ' || *first == '\t' || *first == '\r')) ++first;
        if (first < lineEnd && *first != '#') out.emplace_back(cur, lineEnd);
        cur = nl ? nl + 1 : stop;
    }
    return out;
}

// Reads numbers off one line (a NUL-terminated copy, so the C library
// conversions stop at its end).
class LineScanner {
public:
    LineScanner(const char* b, const char* e) : text_(b, e) { text_.push_back('\0'); at_ = text_.data(); }
    bool integer(long long& x) {
        char* after = nullptr;
        x = std::strtoll(at_, &after, 10);
        return advance(after);
    }
    bool real(double& x) {
        char* after = nullptr;
        x = std::strtod(at_, &after);
        return advance(after);
    }

private:
    bool advance(char* after) {
        if (after == at_) return false;
        at_ = after;
        return true;
    }
    std::vector<char> text_;
    const char* at_;
};

struct EdgeLine {
    int64_t a, b;
    double w;
};

bool whole_number(double w) { return w == std::floor(w) && std::fabs(w) < 9007199254740992.0; }

// W, A and D of the weight rule over the edge lines.  Each line contributes
// (id, |w|) for both of its ends; a stable sort by id keeps every id's
// contributions in file order, so each per-id sum is accumulated in line
// order.
struct WeightBounds {
    double maxAbs = 0.0, maxIdSum = 0.0, maxIdEnds = 0.0;
};

WeightBounds weight_bounds(const std::vector<EdgeLine>& lines) {
    WeightBounds wb;
    std::vector<std::pair<int64_t, double>> ends;
    ends.reserve(2 * lines.size());
    for (const EdgeLine& l : lines) {
        const double mag = std::fabs(l.w);
        wb.maxAbs = std::max(wb.maxAbs, mag);
        ends.emplace_back(l.a, mag);
        ends.emplace_back(l.b, mag);
    }
    std::stable_sort(ends.begin(), ends.end(),
                     [](const std::pair<int64_t, double>& x, const std::pair<int64_t, double>& y) {
                         return x.first < y.first;
                     });
    for (size_t lo = 0; lo < ends.size();) {
        size_t hi = lo;
        double sum = 0.0;
        for (; hi < ends.size() && ends[hi].first == ends[lo].first; ++hi) sum += ends[hi].second;
        wb.maxIdSum = std::max(wb.maxIdSum, sum);
        wb.maxIdEnds = std::max(wb.maxIdEnds, static_cast<double>(hi - lo));
        lo = hi;
    }
    return wb;
}

// The power of ten of the weight rule, or 0 when none qualifies.
double power_of_ten_scale(const WeightBounds& wb) {
    static const double kPow10[25] = {1e12, 1e11, 1e10, 1e9,  1e8,   1e7,   1e6,   1e5,  1e4,
                                      1e3,  1e2,  1e1,  1e0,  1e-1,  1e-2,  1e-3,  1e-4, 1e-5,
                                      1e-6, 1e-7, 1e-8, 1e-9, 1e-10, 1e-11, 1e-12};
    const double weightCap = static_cast<double>(std::numeric_limits<int32_t>::max()) / 2;
    const double sumCaps[2] = {static_cast<double>(std::numeric_limits<int32_t>::max()) / 4,
                               static_cast<double>(std::numeric_limits<int64_t>::max()) / 8};
    for (double cap : sumCaps)
        for (double s : kPow10)
            if (wb.maxIdSum * s + wb.maxIdEnds / 2 <= cap && wb.maxAbs * s <= weightCap) return s;
    return 0.0;
}

}  // namespace

extern "C" int rfmf_gset_header(const char* text, size_t len, int64_t* n, int64_t* m) {
    if (!text || !n || !m) return fail(RFMF_ERR_INVALID, "text/n/m is NULL");
    const auto lines = data_lines(text, len);
    long long N = -1, M = -1;
    if (lines.empty()) return fail(RFMF_ERR_INVALID, "no data line: the first must hold the vertex and edge counts");
    LineScanner sc(lines[0].first, lines[0].second);
    if (!sc.integer(N) || !sc.integer(M) || N < 0 || M < 0)
        return fail(RFMF_ERR_INVALID, "the first data line must hold two counts >= 0 (vertices, edges)");
    *n = N;
    *m = M;
    return RFMF_OK;
}

static int rfmf_gset_parse_impl(const char* text, size_t len, double forced_scale, int64_t cap,
                               int64_t* u, int64_t* v, int64_t* w, int64_t* nedges,
                               double* scale_out, int64_t* zero_dropped) {
    if (!text || !u || !v || !w || !nedges) return fail(RFMF_ERR_INVALID, "NULL argument");
    host_alloc_point();
    int64_t N = 0, M = 0;
    if (int rc = rfmf_gset_header(text, len, &N, &M)) return rc;
    if (cap < M) return fail(RFMF_ERR_CAPACITY, "cap %lld < %lld edges", (long long)cap, (long long)M);
    const auto lines = data_lines(text, len);
    if (static_cast<int64_t>(lines.size()) - 1 < M)
        return fail(RFMF_ERR_INVALID, "header announces %lld edges, the text has %lld edge lines",
                    (long long)M, (long long)(lines.size() - 1));
    std::vector<EdgeLine> edges(static_cast<size_t>(M));
    bool allWhole = true;
    for (int64_t i = 0; i < M; ++i) {
        LineScanner sc(lines[i + 1].first, lines[i + 1].second);
        long long a = 0, b = 0;
        double x = 0.0;
        if (!sc.integer(a) || !sc.integer(b) || !sc.real(x))
            return fail(RFMF_ERR_INVALID, "edge line %lld: expected two ids and a weight", (long long)i);
        edges[i] = EdgeLine{a, b, x};
        allWhole = allWhole && whole_number(x);
    }
    double s = 1.0;
    if (forced_scale > 0.0) {
        s = forced_scale;
    } else if (!allWhole) {
        const WeightBounds wb = weight_bounds(edges);
        s = power_of_ten_scale(wb);
        if (s == 0.0)
            return fail(RFMF_ERR_INVALID, "weights too large for any power-of-ten scale (max |w| %g, max id |w| sum %g)",
                        wb.maxAbs, wb.maxIdSum);
        if (wb.maxAbs * s < 0.5)
            return fail(RFMF_ERR_INVALID, "at scale %g every weight rounds to zero (max |w| %g)", s, wb.maxAbs);
    }
    int64_t kept = 0, zeros = 0;
    for (const EdgeLine& l : edges) {
        const int64_t iw = (s == 1.0 && whole_number(l.w)) ? static_cast<int64_t>(l.w) : std::llround(l.w * s);
        if (iw == 0) {
            ++zeros;
            continue;
        }
        u[kept] = l.a;
        v[kept] = l.b;
        w[kept] = iw;
        ++kept;
    }
    *nedges = kept;
    if (scale_out) *scale_out = s;
    if (zero_dropped) *zero_dropped = zeros;
    return RFMF_OK;
}

// ======================================================================
// CSR build on the device
// ======================================================================
namespace {

constexpr int kScanBlock = 1024;     // threads per scan block
constexpr int kScanItems = 4;        // items per thread
constexpr int kScanTile = kScanBlock * kScanItems;

// Exclusive scan of one tile per block; the block total goes to sums[block].
template <class T>
__global__ void scan_tiles(const T* in, T* out, T* sums, int64_t n) {
    __shared__ T warpTot[kScanBlock / 32];
    const int64_t base = static_cast<int64_t>(blockIdx.x) * kScanTile + threadIdx.x * kScanItems;
    T v[kScanItems];
    T run = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = (base + k < n) ? in[base + k] : T(0);
        const T x = v[k];
        v[k] = run;
        run += x;
    }
    // inclusive warp scan of the thread totals
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    T incl = run;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T o = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += o;
    }
    if (lane == 31) warpTot[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        T t = (lane < kScanBlock / 32) ? warpTot[lane] : T(0);
        T ti = t;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const T o = __shfl_up_sync(0xFFFFFFFFu, ti, d);
            if (lane >= d) ti += o;
        }
        if (lane < kScanBlock / 32) warpTot[lane] = ti - t;   // exclusive
        if (lane == kScanBlock / 32 - 1 && sums) sums[blockIdx.x] = ti;
    }
    __syncthreads();
    const T off = warpTot[wid] + (incl - run);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
        if (base + k < n) out[base + k] = v[k] + off;
}

template <class T>
__global__ void add_tile_offsets(T* out, const T* offs, int64_t n) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * kScanTile + threadIdx.x;
    const T o = offs[blockIdx.x];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int64_t j = i + static_cast<int64_t>(k) * kScanBlock;
        if (j < n) out[j] += o;
    }
}

// Elements of scan scratch for n values: the tile sums of every level.
int64_t scan_scratch(int64_t n) {
    int64_t total = 0;
    while (n > 1) {
        n = (n + kScanTile - 1) / kScanTile;
        total += n + 1;
    }
    return total + 1;
}

// Exclusive scan of n values (out may equal in), recursive over tiles;
// `sums` holds scan_scratch(n) elements.  Asynchronous on st.
template <class T>
int exclusive_scan(const T* in, T* out, int64_t n, T* sums, cudaStream_t st) {
    if (n <= 0) return RFMF_OK;
    const int64_t tiles = (n + kScanTile - 1) / kScanTile;
    scan_tiles<T><<<static_cast<unsigned>(tiles), kScanBlock, 0, st>>>(in, out, sums, n);
    CU(cudaGetLastError());
    if (tiles > 1) {
        if (int rc = exclusive_scan<T>(sums, sums, tiles, sums + tiles + 1, st)) return rc;
        add_tile_offsets<T><<<static_cast<unsigned>(tiles), kScanBlock, 0, st>>>(out, sums, n);
        CU(cudaGetLastError());
    }
    return RFMF_OK;
}

// What one pass over the edge lines finds (zero weights count for the id
// check only: the parser's rule drops them).
struct EdgeFacts {
    unsigned long long firstNegative;   // first edge with a negative id (~0: none)
    unsigned long long firstBig;        // first edge whose weight does not fit int32
    long long maxId;                    // largest id of the kept edges
    unsigned long long kept;
    int selfLoop;
    int pad;
};

// Facts of the surviving entries.
struct RowFacts {
    unsigned long long B;
    long long wsum2;
    int notUnit;
    int notSmall;
    int hubs;     // rows in the hub list
    int longest;  // entries of the longest
};

constexpr int kIngestBlock = 256;

// HBM bound: 24 bytes an edge read once.
__global__ void check_edges(const int64_t* u, const int64_t* v, const int64_t* w, int64_t E, EdgeFacts* f) {
    long long maxId = 0;
    unsigned long long kept = 0;
    bool loop = false;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < E;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t a = u[i], b = v[i], x = w[i];
        if (a < 0 || b < 0) {
            atomicMin(&f->firstNegative, static_cast<unsigned long long>(i));
            continue;
        }
        if (x == 0) continue;
        if (x > INT32_MAX || x < -static_cast<int64_t>(INT32_MAX)) {
            atomicMin(&f->firstBig, static_cast<unsigned long long>(i));
            continue;
        }
        ++kept;
        maxId = max(maxId, static_cast<long long>(a > b ? a : b));
        loop = loop || a == b;
    }
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
        maxId = max(maxId, __shfl_xor_sync(0xFFFFFFFFu, maxId, m));
        kept += __shfl_xor_sync(0xFFFFFFFFu, kept, m);
    }
    const bool any = __any_sync(0xFFFFFFFFu, loop);
    if ((threadIdx.x & 31) == 0) {
        if (kept) {
            atomicMax(&f->maxId, maxId);
            atomicAdd(&f->kept, kept);
        }
        if (any) atomicOr(&f->selfLoop, 1);
    }
}

__global__ void mark_endpoints(const int64_t* u, const int64_t* v, const int64_t* w, int64_t E, int32_t* present) {
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < E;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        if (w[i] == 0) continue;
        present[u[i]] = 1;
        present[v[i]] = 1;
    }
}

__global__ void count_degrees(const int64_t* u, const int64_t* v, const int64_t* w, int64_t E, const int32_t* dense,
                              int32_t* deg) {
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < E;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        if (w[i] == 0) continue;
        atomicAdd(&deg[dense[u[i]]], 1);
        atomicAdd(&deg[dense[v[i]]], 1);
    }
}

// Directed entry: neighbour in the high half, input edge index in the low one
// (fewer than 2^32 edge lines); ascending keys are the row's order.
__device__ __forceinline__ unsigned long long entry_key(int32_t col, int64_t idx) {
    return (static_cast<unsigned long long>(static_cast<uint32_t>(col)) << 32) | static_cast<uint32_t>(idx);
}

// cursor[r] starts at row r's first entry.
__global__ void scatter_entries(const int64_t* u, const int64_t* v, const int64_t* w, int64_t E,
                                const int32_t* dense, int32_t* cursor, unsigned long long* ent) {
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < E;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        if (w[i] == 0) continue;
        const int32_t a = dense[u[i]], b = dense[v[i]];
        ent[atomicAdd(&cursor[a], 1)] = entry_key(b, i);
        ent[atomicAdd(&cursor[b], 1)] = entry_key(a, i);
    }
}

// Rows above this are sorted as tiles of this length and merged (sort_tiles).
constexpr int kHubRow = 2048;

// Rank of `key` among the d keys of a row.
__device__ __forceinline__ int rank_in(const unsigned long long* row, int d, unsigned long long key) {
    int rank = 0;
#pragma unroll 4
    for (int j = 0; j < d; ++j) rank += row[j] < key;
    return rank;
}

// The surviving entries (first key of each neighbour) of a sorted row: counts
// them for this thread's stride and folds their weights into the facts.
struct RowSum {
    int kept = 0;
    long long abs = 0, sum = 0;
    bool notUnit = false, notSmall = false;
    __device__ __forceinline__ void add(const unsigned long long* row, int i, const int64_t* w) {
        const unsigned long long k = row[i];
        if (i > 0 && (row[i - 1] >> 32) == (k >> 32)) return;
        const int32_t x = static_cast<int32_t>(w[static_cast<uint32_t>(k)]);
        ++kept;
        abs += x < 0 ? -static_cast<long long>(x) : x;
        sum += x;
        notUnit = notUnit || (x != 1 && x != -1);
        notSmall = notSmall || x < -32767 || x > 32767;
    }
    __device__ __forceinline__ void warp() {
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) {
            kept += __shfl_xor_sync(0xFFFFFFFFu, kept, m);
            abs += __shfl_xor_sync(0xFFFFFFFFu, abs, m);
        }
    }
};

// Count of survivors and, in the high half, padded to four (both are scanned
// together).
__device__ __forceinline__ uint64_t kept_word(int k) {
    return (static_cast<uint64_t>((k + 3) & ~3) << 32) | static_cast<uint32_t>(k);
}

// One warp a row: every lane ranks its keys against the whole row (d^2 / 32
// comparisons on broadcast loads, no moves) and writes them in order, then the
// row's survivors are counted.  (One thread's insertion sort of 16-byte
// entries, d^2 / 4 moves through memory, took most of a 481,000-edge build.)
__global__ void __launch_bounds__(kIngestBlock) sort_rows(const unsigned long long* ent, const int32_t* rowStart,
                                                          const int32_t* nPtr, const int64_t* w,
                                                          unsigned long long* out, uint64_t* keep, RowFacts* f,
                                                          int32_t* hubList) {
    const int n = *nPtr, lane = threadIdx.x & 31;
    const int warps = (gridDim.x * kIngestBlock) >> 5;
    unsigned long long maxB = 0;
    long long wsum = 0;
    bool notUnit = false, notSmall = false;
    for (int r = (blockIdx.x * kIngestBlock + threadIdx.x) >> 5; r < n; r += warps) {
        const int lo = rowStart[r], d = rowStart[r + 1] - lo;
        if (d > kHubRow) {
            if (lane == 0) {
                hubList[atomicAdd(&f->hubs, 1)] = r;
                atomicMax(&f->longest, d);
            }
            continue;
        }
        for (int i = lane; i < d; i += 32) {
            const unsigned long long k = ent[lo + i];
            out[lo + rank_in(ent + lo, d, k)] = k;
        }
        __syncwarp();
        RowSum s;
        for (int i = lane; i < d; i += 32) s.add(out + lo, i, w);
        s.warp();
        if (lane == 0) keep[r] = kept_word(s.kept);
        maxB = maxB > static_cast<unsigned long long>(s.abs) ? maxB : static_cast<unsigned long long>(s.abs);
        wsum += s.sum;
        notUnit = notUnit || s.notUnit;
        notSmall = notSmall || s.notSmall;
    }
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) wsum += __shfl_xor_sync(0xFFFFFFFFu, wsum, m);
    notUnit = __any_sync(0xFFFFFFFFu, notUnit);
    notSmall = __any_sync(0xFFFFFFFFu, notSmall);
    if (lane == 0) {
        if (maxB) atomicMax(&f->B, maxB);
        if (wsum) atomicAdd(reinterpret_cast<unsigned long long*>(&f->wsum2), static_cast<unsigned long long>(wsum));
        if (notUnit) atomicOr(&f->notUnit, 1);
        if (notSmall) atomicOr(&f->notSmall, 1);
    }
}

// The rows of the hub list, sorted in d log d: tiles of kHubRow keys by rank
// counts in shared memory, in place in `ent` or into `out`; then runs merged
// pairwise (merge_runs), every key finding its place in the other run by
// bisection.  Each row's tiles are spread over the blocks, the first one's block
// rotating with the row.  GB300, a whole call on a star of 20,000 leaves 0.8 ms
// (13.3 when a block ranked every key of a hub row against the row), of 300,000
// 5.2, of 1,000,000 16.
__global__ void __launch_bounds__(1024) sort_tiles(const unsigned long long* ent, const int32_t* rowStart,
                                                   const RowFacts* f, const int32_t* hubList,
                                                   unsigned long long* out) {
    __shared__ unsigned long long tile[kHubRow];
    const int hubs = f->hubs;
    for (int h = 0; h < hubs; ++h) {
        const int r = hubList[h], lo = rowStart[r], d = rowStart[r + 1] - lo;
        for (int64_t at = static_cast<int64_t>((blockIdx.x + h) % gridDim.x) * kHubRow; at < d;
             at += static_cast<int64_t>(gridDim.x) * kHubRow) {
            const int len = static_cast<int>(min(static_cast<int64_t>(kHubRow), d - at));
            for (int i = threadIdx.x; i < len; i += blockDim.x) tile[i] = ent[lo + at + i];
            __syncthreads();
            for (int i = threadIdx.x; i < len; i += blockDim.x) out[lo + at + rank_in(tile, len, tile[i])] = tile[i];
            __syncthreads();
        }
    }
}

__global__ void __launch_bounds__(kIngestBlock) merge_runs(const unsigned long long* in, const int32_t* rowStart,
                                                           const RowFacts* f, const int32_t* hubList, int64_t run,
                                                           unsigned long long* out) {
    const int hubs = f->hubs;
    for (int h = 0; h < hubs; ++h) {
        const int r = hubList[h], lo = rowStart[r], d = rowStart[r + 1] - lo;
        for (int64_t i = static_cast<int64_t>((blockIdx.x + h) % gridDim.x) * kIngestBlock + threadIdx.x; i < d;
             i += static_cast<int64_t>(gridDim.x) * kIngestBlock) {
            const unsigned long long key = in[lo + i];
            const int64_t pair = i / (2 * run) * (2 * run), mid = min(pair + run, static_cast<int64_t>(d));
            const int64_t end = min(mid + run, static_cast<int64_t>(d));
            int64_t a = i < mid ? mid : pair, b = i < mid ? end : mid;   // the other run
            while (a < b) {
                const int64_t m = (a + b) >> 1;
                if (in[lo + m] < key) a = m + 1;
                else b = m;
            }
            out[lo + i + a - mid] = key;   // pair + the smaller keys of both runs, whichever run it is from
        }
    }
}

// Survivors and weight facts of the sorted hub rows, a block each.
__global__ void __launch_bounds__(1024) count_hubs(const unsigned long long* out, const int32_t* rowStart,
                                                   const int64_t* w, uint64_t* keep, RowFacts* f,
                                                   const int32_t* hubList) {
    __shared__ int kept[32];
    __shared__ long long abs[32];
    const int hubs = f->hubs, lane = threadIdx.x & 31;
    for (int h = blockIdx.x; h < hubs; h += gridDim.x) {
        const int r = hubList[h], lo = rowStart[r], d = rowStart[r + 1] - lo;
        RowSum s;
        for (int i = threadIdx.x; i < d; i += blockDim.x) s.add(out + lo, i, w);
        if (s.sum) atomicAdd(reinterpret_cast<unsigned long long*>(&f->wsum2), static_cast<unsigned long long>(s.sum));
        if (s.notUnit) atomicOr(&f->notUnit, 1);
        if (s.notSmall) atomicOr(&f->notSmall, 1);
        s.warp();
        if (lane == 0) {
            kept[threadIdx.x >> 5] = s.kept;
            abs[threadIdx.x >> 5] = s.abs;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int k = 0;
            long long b = 0;
            for (int q = 0; q < static_cast<int>(blockDim.x >> 5); ++q) {
                k += kept[q];
                b += abs[q];
            }
            keep[r] = kept_word(k);
            atomicMax(&f->B, static_cast<unsigned long long>(b));
        }
        __syncthreads();
    }
}

// The survivors of every sorted row, one warp a row, in all the formats given:
// {col, w} pairs with their offsets and their two halves, and the compact rows (start[r]: kept
// entries before row r, padded entries in the high half) with their row words
// and padding (the vertex itself, weight +1 or 0).  offsets and rows are
// filled up to `words`.
__global__ void __launch_bounds__(kIngestBlock) emit_rows(const unsigned long long* ent, const int32_t* rowStart,
                                                          const uint64_t* start, int n, int words, const int64_t* w,
                                                          uint32_t* offsets, Edge* edges, int32_t* cols,
                                                          int32_t* weights, uint32_t* rows, uint16_t* u16,
                                                          uint32_t* p32) {
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * kIngestBlock) >> 5;
    for (int r = (blockIdx.x * kIngestBlock + threadIdx.x) >> 5; r < n; r += warps) {
        const int lo = rowStart[r], d = rowStart[r + 1] - lo;
        const uint32_t o = static_cast<uint32_t>(start[r]), c = static_cast<uint32_t>(start[r] >> 32);
        uint32_t k = 0;   // survivors so far
        for (int i0 = 0; i0 < d; i0 += 32) {
            const int i = i0 + lane;
            bool take = false;
            unsigned long long key = 0;
            if (i < d) {
                key = ent[lo + i];
                take = i == 0 || (ent[lo + i - 1] >> 32) != (key >> 32);
            }
            const uint32_t vote = __ballot_sync(0xFFFFFFFFu, take);
            if (take) {
                const uint32_t at = k + __popc(vote & ((1u << lane) - 1u));
                const int32_t col = static_cast<int32_t>(key >> 32);
                const int32_t x = static_cast<int32_t>(w[static_cast<uint32_t>(key)]);
                edges[o + at] = Edge{col, x};
                cols[o + at] = col;
                weights[o + at] = x;
                if (u16) u16[c + at] = static_cast<uint16_t>(col | (x < 0 ? 0x8000 : 0));
                if (p32) p32[c + at] = (static_cast<uint32_t>(x) << 16) | static_cast<uint32_t>(col);
            }
            k += __popc(vote);
        }
        const uint32_t pad = (0u - k) & 3u;
        if (static_cast<uint32_t>(lane) < pad) {
            if (u16) u16[c + k + lane] = static_cast<uint16_t>(r);
            if (p32) p32[c + k + lane] = static_cast<uint32_t>(r);
        }
        if (lane == 0) {
            offsets[r] = o;
            if (rows) rows[r] = c | pad;
        }
    }
    if (blockIdx.x == 0) {
        for (int r = n + threadIdx.x; r < words; r += kIngestBlock) {
            offsets[r] = static_cast<uint32_t>(start[n]);
            if (rows) rows[r] = static_cast<uint32_t>(start[n] >> 32);
        }
    }
}

__global__ void orig_ids(const int32_t* present, const int32_t* dense, int64_t maxId, int64_t* out) {
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i <= maxId;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        if (present[i]) out[dense[i]] = i;
}

unsigned grid_for(int64_t n) {
    return static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 4096)));
}

}  // namespace

// Parts of one scratch allocation, each 256-byte aligned.
class Arena {
public:
    template <class T>
    size_t add(int64_t count) {
        const size_t at = bytes_;
        bytes_ += (static_cast<size_t>(count) * sizeof(T) + 255) & ~size_t(255);
        return at;
    }
    int alloc(const rfmf_context* ctx) { return buf_.alloc(ctx, bytes_); }
    template <class T>
    T* at(size_t off) const { return reinterpret_cast<T*>(static_cast<char*>(buf_.p) + off); }

private:
    Scratch buf_;
    size_t bytes_ = 0;
};

static int rfmf_graph_from_edges_impl(rfmf_context* ctx, int64_t nedges, const int64_t* u,
                                     const int64_t* v, const int64_t* w, rfmf_graph** out,
                                     int64_t* n_out) {
    if (!ctx || !out || nedges < 0 || (nedges > 0 && (!u || !v || !w)))
        return fail(RFMF_ERR_INVALID, "bad arguments");
    *out = nullptr;
    const int64_t E = nedges;
    // More lines than a graph can keep (below 2^30): those of weight zero do not
    // get device memory, nor a number in the entries' 32 bits.
    if (E >= (int64_t(1) << 30)) {
        std::vector<int64_t> keep[3];
        int64_t largest = 0, kept = 0;
        for (int64_t i = 0; i < E; ++i) {
            if (u[i] < 0 || v[i] < 0) return fail(RFMF_ERR_INVALID, "negative vertex id at edge %lld", (long long)i);
            if (w[i] == 0) continue;
            if (w[i] > INT32_MAX || w[i] < -static_cast<int64_t>(INT32_MAX))
                return fail(RFMF_ERR_CAPACITY, "weight at edge %lld does not fit int32", (long long)i);
            largest = std::max(largest, std::max(u[i], v[i]));
            if (++kept >= (int64_t(1) << 30)) continue;
            keep[0].push_back(u[i]);
            keep[1].push_back(v[i]);
            keep[2].push_back(w[i]);
        }
        if (largest < (int64_t(1) << 28) && kept >= (int64_t(1) << 30)) return fail(RFMF_ERR_CAPACITY, "too many edges");
        return rfmf_graph_from_edges_impl(ctx, static_cast<int64_t>(keep[0].size()), keep[0].data(), keep[1].data(),
                                          keep[2].data(), out, n_out);
    }
    CU(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    int rc;
    // The edge lines as they are; ids and weights are checked on the device.
    Arena in;
    const size_t oU = in.add<int64_t>(E), oV = in.add<int64_t>(E), oW = in.add<int64_t>(E), oF = in.add<EdgeFacts>(1);
    if ((rc = in.alloc(ctx))) return rc;
    const int64_t *dU = in.at<int64_t>(oU), *dV = in.at<int64_t>(oV), *dW = in.at<int64_t>(oW);
    EdgeFacts ef{~0ull, ~0ull, 0, 0, 0, 0};
    CU(cudaMemcpyAsync(in.at<EdgeFacts>(oF), &ef, sizeof ef, cudaMemcpyHostToDevice, st));
    if (E) {
        CU(cudaMemcpyAsync(in.at<int64_t>(oU), u, E * 8, cudaMemcpyHostToDevice, st));
        CU(cudaMemcpyAsync(in.at<int64_t>(oV), v, E * 8, cudaMemcpyHostToDevice, st));
        CU(cudaMemcpyAsync(in.at<int64_t>(oW), w, E * 8, cudaMemcpyHostToDevice, st));
        check_edges<<<grid_for(E), kIngestBlock, 0, st>>>(dU, dV, dW, E, in.at<EdgeFacts>(oF));
        CU(cudaGetLastError());
    }
    CU(cudaMemcpyAsync(&ef, in.at<EdgeFacts>(oF), sizeof ef, cudaMemcpyDeviceToHost, st));
    CU(cudaStreamSynchronize(st));
    if (ef.firstNegative != ~0ull && ef.firstNegative <= ef.firstBig)
        return fail(RFMF_ERR_INVALID, "negative vertex id at edge %lld", (long long)ef.firstNegative);
    if (ef.firstBig != ~0ull)
        return fail(RFMF_ERR_CAPACITY, "weight at edge %lld does not fit int32", (long long)ef.firstBig);
    const int64_t maxId = ef.maxId, kept = static_cast<int64_t>(ef.kept);
    if (maxId >= (int64_t(1) << 28))
        return fail(RFMF_ERR_CAPACITY, "vertex ids up to %lld: the device build takes ids below 2^28",
                    (long long)maxId);
    if (ef.selfLoop) return fail(RFMF_ERR_INVALID, "self loop in the edge list");

    // Scratch, rows at most one per id and per line end.
    const int64_t ids = maxId + 1, rowsMax = std::min<int64_t>(ids, 2 * kept) + 1;
    Arena sc;
    const size_t oPresent = sc.add<int32_t>(ids + 1), oDeg = sc.add<int32_t>(rowsMax), oKeep = sc.add<uint64_t>(rowsMax),
                 oRf = sc.add<RowFacts>(1), zeroBytes = sc.add<char>(0), oDense = sc.add<int32_t>(ids + 1),
                 oRow = sc.add<int32_t>(rowsMax), oCursor = sc.add<int32_t>(rowsMax), oStart = sc.add<uint64_t>(rowsMax),
                 oEnt = sc.add<unsigned long long>(2 * kept), oSorted = sc.add<unsigned long long>(2 * kept),
                 oHubs = sc.add<int32_t>(2 * kept / kHubRow + 1), oIds = sc.add<int64_t>(rowsMax),
                 oSums = sc.add<uint64_t>(scan_scratch(std::max(ids + 1, rowsMax)));
    if ((rc = sc.alloc(ctx))) return rc;
    int32_t *present = sc.at<int32_t>(oPresent), *dense = sc.at<int32_t>(oDense), *deg = sc.at<int32_t>(oDeg);
    int32_t *row = sc.at<int32_t>(oRow), *cursor = sc.at<int32_t>(oCursor), *hubs = sc.at<int32_t>(oHubs);
    uint64_t *keep = sc.at<uint64_t>(oKeep), *start = sc.at<uint64_t>(oStart);
    unsigned long long *ent = sc.at<unsigned long long>(oEnt), *sorted = sc.at<unsigned long long>(oSorted);
    RowFacts* rf = sc.at<RowFacts>(oRf);
    int32_t* sums32 = sc.at<int32_t>(oSums);
    CU(cudaMemsetAsync(present, 0, zeroBytes, st));   // presence, degrees, kept counts, facts
    if (E) mark_endpoints<<<grid_for(E), kIngestBlock, 0, st>>>(dU, dV, dW, E, present);
    // dense ids: exclusive scan of presence over ids + 1 slots; n = last value
    if ((rc = exclusive_scan<int32_t>(present, dense, ids + 1, sums32, st))) return rc;
    if (E) count_degrees<<<grid_for(E), kIngestBlock, 0, st>>>(dU, dV, dW, E, dense, deg);
    // row starts (slots past the last row hold 2 * kept)
    if ((rc = exclusive_scan<int32_t>(deg, row, rowsMax, sums32, st))) return rc;
    CU(cudaMemcpyAsync(cursor, row, rowsMax * 4, cudaMemcpyDeviceToDevice, st));
    if (E) scatter_entries<<<grid_for(E), kIngestBlock, 0, st>>>(dU, dV, dW, E, dense, cursor, ent);
    if (kept) {
        const unsigned blocks = static_cast<unsigned>(std::min<int64_t>((rowsMax + 7) / 8, 8 * ctx->sms));
        sort_rows<<<blocks, kIngestBlock, 0, st>>>(ent, row, dense + ids, dW, sorted, keep, rf, hubs);
    }
    CU(cudaGetLastError());
    RowFacts hf{};
    int32_t n = 0;
    uint64_t total = 0;
    auto facts = [&]() -> int {
        if (int rc2 = exclusive_scan<uint64_t>(keep, start, rowsMax, sc.at<uint64_t>(oSums), st)) return rc2;
        CU(cudaMemcpyAsync(&hf, rf, sizeof hf, cudaMemcpyDeviceToHost, st));
        CU(cudaMemcpyAsync(&n, dense + ids, 4, cudaMemcpyDeviceToHost, st));
        CU(cudaMemcpyAsync(&total, start + rowsMax - 1, 8, cudaMemcpyDeviceToHost, st));
        CU(cudaStreamSynchronize(st));
        return RFMF_OK;
    };
    if ((rc = facts())) return rc;
    if (hf.hubs) {   // their rows sorted and counted, then the facts again
        int passes = 0;
        while ((static_cast<int64_t>(kHubRow) << passes) < hf.longest) ++passes;
        unsigned long long *from = (passes & 1) ? ent : sorted, *to = (passes & 1) ? sorted : ent;
        sort_tiles<<<2 * ctx->sms, 1024, 0, st>>>(ent, row, rf, hubs, from);
        for (int p = 0; p < passes; ++p, std::swap(from, to))
            merge_runs<<<8 * ctx->sms, kIngestBlock, 0, st>>>(from, row, rf, hubs, static_cast<int64_t>(kHubRow) << p, to);
        count_hubs<<<2 * ctx->sms, 1024, 0, st>>>(sorted, row, dW, keep, rf, hubs);
        CU(cudaGetLastError());
        if ((rc = facts())) return rc;
    }
    const int32_t m2 = static_cast<int32_t>(total);
    const uint32_t mPad = static_cast<uint32_t>(total >> 32);   // entries of the padded compact rows

    auto g = std::unique_ptr<rfmf_graph>(new (std::nothrow) rfmf_graph());
    if (!g) return fail(RFMF_ERR_NOMEM, "host allocation failed");
    g->ctxHold.set(ctx);
    g->ctx = ctx;
    g->n = n;
    g->m = m2 / 2;
    g->B = static_cast<int64_t>(hf.B);
    g->wsum2 = hf.wsum2;
    if (g->B > std::numeric_limits<int32_t>::max())
        return fail(RFMF_ERR_CAPACITY, "max weighted degree %lld exceeds int32", (long long)g->B);
    const uint64_t ob = (static_cast<uint64_t>(n + 1) * 4u + 15u) & ~uint64_t(15);
    g->halves = true;
    if ((rc = g->edges.alloc(static_cast<size_t>(m2) * (sizeof(Edge) + 8)))) return rc;
    g->unit16 = !hf.notUnit && n <= 32768;
    g->packed32 = !hf.notSmall && n <= 65536 && mPad < (1u << 30);
    if (g->unit16 || g->packed32) g->rowBytes = static_cast<uint32_t>(ob);
    if ((rc = g->offsets.alloc(ob + g->rowBytes))) return rc;
    if (g->unit16) {
        g->u16Bytes = align16(mPad * 2u);
        if ((rc = g->u16.alloc(g->u16Bytes))) return rc;
        CU(cudaMemsetAsync(static_cast<char*>(g->u16.p) + (g->u16.bytes - 16), 0, 16, st));   // the last vector's rest
    }
    if (g->packed32) {
        g->p32Bytes = align16(mPad * 4u);
        if ((rc = g->p32.alloc(g->p32Bytes))) return rc;
    }
    const unsigned blocks = static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>((n + 7) / 8, 8 * ctx->sms)));
    emit_rows<<<blocks, kIngestBlock, 0, st>>>(sorted, row, start, n, static_cast<int>(ob / 4), dW,
                                               g->offsets.as<uint32_t>(), g->edges.as<Edge>(), g->cols(), g->weights(),
                                               g->row_words(),
                                               g->unit16 ? g->u16.as<uint16_t>() : nullptr,
                                               g->packed32 ? g->p32.as<uint32_t>() : nullptr);
    CU(cudaGetLastError());
    // dense id -> original id, kept on the host with the graph
    g->origIds.resize(static_cast<size_t>(n));
    if (n) {
        orig_ids<<<grid_for(ids), kIngestBlock, 0, st>>>(present, dense, maxId, sc.at<int64_t>(oIds));
        CU(cudaGetLastError());
        CU(cudaMemcpyAsync(g->origIds.data(), sc.at<int64_t>(oIds), n * 8, cudaMemcpyDeviceToHost, st));
    }
    CU(cudaStreamSynchronize(st));
    if (n_out) *n_out = n;
    *out = g.release();
    return RFMF_OK;
}

static int rfmf_graph_orig_ids_impl(const rfmf_graph* g, int64_t* out) {
    if (!g || !out) return fail(RFMF_ERR_INVALID, "graph/out is NULL");
    if (static_cast<int64_t>(g->origIds.size()) != g->n)
        return fail(RFMF_ERR_INVALID, "graph was not built from an edge list");
    std::copy(g->origIds.begin(), g->origIds.end(), out);
    return RFMF_OK;
}

static int rfmf_graph_csr_impl(const rfmf_graph* g, uint32_t* offsets, int32_t* col, int32_t* weight) {
    if (!g) return fail(RFMF_ERR_INVALID, "graph is NULL");
    CU(cudaSetDevice(g->ctx->device));
    const int64_t m2 = 2 * g->m;
    if (offsets) CU(cudaMemcpy(offsets, g->offsets.p, (g->n + 1) * 4, cudaMemcpyDeviceToHost));
    // Plain copies: they need no device memory and wait for no launch.
    if (g->halves) {
        if (col && m2) CU(cudaMemcpy(col, g->cols(), m2 * 4, cudaMemcpyDeviceToHost));
        if (weight && m2) CU(cudaMemcpy(weight, g->weights(), m2 * 4, cudaMemcpyDeviceToHost));
        return RFMF_OK;
    }
    if (!col && !weight) return RFMF_OK;
    constexpr int64_t kPart = int64_t(1) << 16;   // split a cache-sized part at a time
    const std::unique_ptr<Edge[]> part(new Edge[static_cast<size_t>(std::min(m2, kPart))]);
    for (int64_t at = 0; at < m2; at += kPart) {
        const int64_t cnt = std::min(kPart, m2 - at);
        CU(cudaMemcpy(part.get(), g->edges.as<Edge>() + at, static_cast<size_t>(cnt) * sizeof(Edge),
                      cudaMemcpyDeviceToHost));
        if (col)
            for (int64_t i = 0; i < cnt; ++i) col[at + i] = part[i].col;
        if (weight)
            for (int64_t i = 0; i < cnt; ++i) weight[at + i] = part[i].w;
    }
    return RFMF_OK;
}

// ======================================================================
// Output path (device)
// ======================================================================
namespace {

__device__ __forceinline__ int bit_of(const uint32_t* bits, int v) {
    return (bits[v >> 5] >> (v & 31)) & 1;
}

// The transpose of the warp's 32 x 32 bits: bit c of lane l's word becomes bit l
// of lane c's.
__device__ __forceinline__ uint32_t transpose_bits(uint32_t x, int lane) {
    uint32_t m = 0x0000FFFFu;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1, m ^= m << s) {
        const uint32_t y = __shfl_xor_sync(0xFFFFFFFFu, x, s);
        x = (lane & s) ? (x & ~m) | ((y >> s) & m) : (x & m) | ((y << s) & ~m);
    }
    return x;
}

// cutValueCsr of up to 32 chains of one graph per CTA (end spins: which 0, best:
// 1): lane c sums chain c.  The chains' spin bits are transposed into one word
// per vertex (bit c: chain c) in shared memory.  A warp takes 32 rows at a time and
// loads their entries 32 together; the words of which chains each entry
// crosses, transposed, give every lane its chain's entries as a bit mask, and
// its sum of weights is a population count per bit of the weights (one for
// +-1).  So 32 entries cost 32 chains about 60 instructions.  Graphs above tableN
// vertices read the chains' bits directly.  GB300, 1024 chains each of the 50x60
// torus and ER n = 2000 d = 19: 25 us; one CTA per chain walking all its entries
// took 87.  (Every slice builds the whole vertex table: slices are kept to 256
// rows at least.)
constexpr int kCutWarps = 8;
__global__ void __launch_bounds__(32 * kCutWarps) chain_cuts_kernel(const DevChain* chains, const DevGraph* graphs,
                                                                    const CutItem* items, const int32_t* order,
                                                                    int tableN, int which, int64_t* out,
                                                                    const int32_t* ctl, int ctlWords,
                                                                    int32_t* ctlOut) {
    extern __shared__ uint32_t spins[];
    __shared__ long long part[kCutWarps][32];
    if (ctl && blockIdx.x == 0)
        for (int w = threadIdx.x; w < ctlWords; w += 32 * kCutWarps) ctlOut[w] = ctl[w];
    const CutItem group = items[blockIdx.x];
    const DevGraph& g = graphs[group.graph];
    const int n = g.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t* offsets = g.offsets;
    const Edge* edges = g.edges;
    int c = -1;
    const uint32_t* bits = nullptr;
    if (lane < group.count) {
        c = order[group.first + lane];
        bits = which ? chains[c].bestBits : chains[c].spinBits;
    }
    const bool table = n <= tableN;
    if (table) {
#pragma unroll 4
        for (int w = warp; w < g.words; w += kCutWarps) {
            const uint32_t x = bits ? bits[w] : 0u;
            const uint32_t mine = transpose_bits(x, lane);
            if (32 * w + lane < n) spins[32 * w + lane] = mine;
        }
        __syncthreads();
    }
    const int v0 = static_cast<int>(static_cast<int64_t>(n) * group.slice / group.slices);
    const int v1 = static_cast<int>(static_cast<int64_t>(n) * (group.slice + 1) / group.slices);
    long long acc = 0;
    for (int base = v0 + 32 * warp; base < v1; base += 32 * kCutWarps) {
        const int rows = min(32, v1 - base);
        const uint32_t off = offsets[base + min(lane, rows)];
        const uint32_t e1 = rows < 32 ? __shfl_sync(0xFFFFFFFFu, off, rows) : offsets[base + 32];
        const uint32_t e0 = __shfl_sync(0xFFFFFFFFu, off, 0);
        for (uint32_t k = 0; k < e1 - e0; k += 32) {   // (e0 + k may pass 2^32 with the last 32)
            const uint32_t i = e0 + k + lane;
            const Edge e = k + lane < e1 - e0 ? edges[i] : Edge{-1, 0};
            int r = 0;   // the entry's row: the last one that starts at or before it
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const uint32_t o = __shfl_sync(0xFFFFFFFFu, off, (r + step) & 31);
                if (r + step < rows && o <= i) r += step;
            }
            const int v = base + r;
            const bool up = e.col > v;
            if (table) {
                const uint32_t mine = transpose_bits(up ? spins[v] ^ spins[e.col] : 0u, lane);
                const uint32_t neg = __ballot_sync(0xFFFFFFFFu, e.w < 0);
                const uint32_t mag = static_cast<uint32_t>(abs(e.w));
                uint32_t planes = __reduce_or_sync(0xFFFFFFFFu, up ? mag : 0u);
                for (; planes; planes &= planes - 1) {
                    const int k = __ffs(planes) - 1;
                    const uint32_t has = mine & __ballot_sync(0xFFFFFFFFu, (mag >> k) & 1u);
                    acc += static_cast<long long>(__popc(has & ~neg) - __popc(has & neg)) << k;
                }
            } else {
                for (uint32_t left = __ballot_sync(0xFFFFFFFFu, up); left; left &= left - 1) {
                    const int j = __ffs(left) - 1;
                    const int w = __shfl_sync(0xFFFFFFFFu, e.w, j);
                    const int vj = __shfl_sync(0xFFFFFFFFu, v, j), uj = __shfl_sync(0xFFFFFFFFu, e.col, j);
                    if (bits && bit_of(bits, vj) != bit_of(bits, uj)) acc += w;
                }
            }
        }
    }
    part[warp][lane] = acc;
    __syncthreads();
    if (warp == 0 && c >= 0) {
        long long t = 0;
#pragma unroll
        for (int w = 0; w < kCutWarps; ++w) t += part[w][lane];
        if (group.slices == 1) out[c] = t;
        else if (t) atomicAdd(reinterpret_cast<unsigned long long*>(out + c), static_cast<unsigned long long>(t));
    }
}

// '0'/'1' per vertex, 16 characters a thread (6.1 MB: 9 us, one character a
// thread 23): bit k of a nibble moves to byte k of 0x30303030 by one multiply.  The rows are one flat array (a thread's 16
// bytes are aligned whatever the stride); bytes past n are 0.
__global__ void chain_partitions_kernel(const DevChain* chains, const DevGraph* graphs, int c0, int count, int which,
                                        char* out, int64_t stride, int64_t total) {
    for (int64_t at = 16 * (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x); at < total;
         at += 16 * static_cast<int64_t>(gridDim.x) * blockDim.x) {
        int r = static_cast<int>(at / stride);
        int64_t v = at - r * stride;
        const DevChain* ch = chains + c0 + r;
        int n = graphs[ch->graph].n;
        const uint32_t* bits = which ? ch->bestBits : ch->spinBits;
        if (v + 16 <= n) {
            const uint32_t lo = bits[v >> 5], hi = (v & 31) > 16 ? bits[(v >> 5) + 1] : 0u;
            const uint32_t x = __funnelshift_r(lo, hi, static_cast<uint32_t>(v) & 31u);
            uint4 q;
            q.x = (((x & 15u) * 0x00204081u) & 0x01010101u) + 0x30303030u;
            q.y = ((((x >> 4) & 15u) * 0x00204081u) & 0x01010101u) + 0x30303030u;
            q.z = ((((x >> 8) & 15u) * 0x00204081u) & 0x01010101u) + 0x30303030u;
            q.w = ((((x >> 12) & 15u) * 0x00204081u) & 0x01010101u) + 0x30303030u;
            *reinterpret_cast<uint4*>(out + at) = q;
        } else {
            for (int k = 0; k < 16 && at + k < total; ++k) {
                out[at + k] = v < n ? (bit_of(bits, static_cast<int>(v)) ? '1' : '0') : '\0';
                if (++v == stride && at + k + 1 < total) {
                    v = 0;
                    ++ch;
                    n = graphs[ch->graph].n;
                    bits = which ? ch->bestBits : ch->spinBits;
                }
            }
        }
    }
}

__global__ void lift_best_kernel(DevChain* chains, int64_t count, int64_t* own) {
    for (int64_t c = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; c < count;
         c += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        DevChain& ch = chains[c];
        const bool low = ch.best < ch.cur && ch.sweepsDone < ch.sweepsTotal;
        own[c] = low ? ch.best : kUnsetCut;
        if (low) ch.best = ch.cur;
    }
}

// A warp a chain.  (A best that the sweep did raise is right as it is.)
__global__ void settle_best_kernel(DevChain* chains, const DevGraph* graphs, int64_t count, const int64_t* own) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = static_cast<int64_t>(gridDim.x) * blockDim.x >> 5;
    for (int64_t c = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5; c < count; c += warps) {
        const int64_t best = own[c];
        DevChain& ch = chains[c];
        if (best == kUnsetCut || ch.improvedSweeps != 0) continue;
        const bool better = ch.cur > best;
        if (better)
            for (int w = lane; w < graphs[ch.graph].words; w += 32) ch.bestBits[w] = ch.spinBits[w];
        __syncwarp();
        if (lane == 0) {
            ch.best = better ? ch.cur : best;
            ch.improvedSweeps = better;
        }
    }
}

}  // namespace

namespace rfmf {

cudaError_t lift_best(DevChain* chains, int64_t count, int64_t* own, cudaStream_t st) {
    lift_best_kernel<<<grid_for(count), 256, 0, st>>>(chains, count, own);
    return cudaGetLastError();
}

cudaError_t settle_best(DevChain* chains, const DevGraph* graphs, int64_t count, const int64_t* own, cudaStream_t st) {
    settle_best_kernel<<<grid_for(32 * count), 256, 0, st>>>(chains, graphs, count, own);
    return cudaGetLastError();
}

cudaError_t launch_chain_cuts(const DevChain* chains, const DevGraph* graphs, const CutItem* items, int nsmall,
                              int nitems, const int32_t* order, int64_t maxN, int smemOptin, int which, int64_t* out,
                              const int32_t* ctl, int words, int32_t* ctlOut, cudaStream_t st) {
    const cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(&chain_cuts_kernel),
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, smemOptin - 4096);
    if (e != cudaSuccess) return e;
    auto launch = [&](const CutItem* from, int count, int64_t largest) {
        if (count <= 0) return;
        const int tableN = static_cast<int>(std::min<int64_t>(largest, (smemOptin - 4096) / 4));
        chain_cuts_kernel<<<static_cast<unsigned>(count), 32 * kCutWarps, 4 * tableN, st>>>(
            chains, graphs, from, order, tableN, which, out, ctl, words, ctlOut);
        ctl = nullptr;
    };
    launch(items, nsmall, std::min(maxN, kCutSmallN));
    launch(items + nsmall, nitems - nsmall, maxN);
    return cudaGetLastError();
}

cudaError_t launch_chain_partitions(const DevChain* chains, const DevGraph* graphs, int c0, int count, int which,
                                    char* out, int64_t stride, cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
    const int64_t total = static_cast<int64_t>(count) * stride;
    const int64_t blocks = std::min<int64_t>((total + 16 * 256 - 1) / (16 * 256), 1 << 16);
    chain_partitions_kernel<<<static_cast<unsigned>(blocks), 256, 0, st>>>(chains, graphs, c0, count, which, out,
                                                                           stride, total);
    return cudaGetLastError();
}

}  // namespace rfmf

// C ABI entry points: no C++ exception crosses the boundary.
extern "C" int rfmf_gset_parse(const char* text, size_t len, double forced_scale, int64_t cap,
                               int64_t* u, int64_t* v, int64_t* w, int64_t* nedges,
                               double* scale_out, int64_t* zero_dropped) {
    try {
        return rfmf_gset_parse_impl(text, len, forced_scale, cap, u, v, w, nedges, scale_out, zero_dropped);
    } catch (const std::bad_alloc&) {
        return rfmf::fail(RFMF_ERR_NOMEM, "host allocation failed in rfmf_gset_parse");
    } catch (...) {
        return rfmf::fail(RFMF_ERR_INVALID, "unexpected host exception in rfmf_gset_parse");
    }
}

extern "C" int rfmf_graph_from_edges(rfmf_context* ctx, int64_t nedges, const int64_t* u,
                                     const int64_t* v, const int64_t* w, rfmf_graph** out,
                                     int64_t* n_out) {
    try {
        return rfmf_graph_from_edges_impl(ctx, nedges, u, v, w, out, n_out);
    } catch (const std::bad_alloc&) {
        return rfmf::fail(RFMF_ERR_NOMEM, "host allocation failed in rfmf_graph_from_edges");
    } catch (...) {
        return rfmf::fail(RFMF_ERR_INVALID, "unexpected host exception in rfmf_graph_from_edges");
    }
}

extern "C" int rfmf_graph_csr(const rfmf_graph* g, uint32_t* offsets, int32_t* col, int32_t* weight) {
    try {
        return rfmf_graph_csr_impl(g, offsets, col, weight);
    } catch (const std::bad_alloc&) {
        return rfmf::fail(RFMF_ERR_NOMEM, "host allocation failed in rfmf_graph_csr");
    } catch (...) {
        return rfmf::fail(RFMF_ERR_INVALID, "unexpected host exception in rfmf_graph_csr");
    }
}

extern "C" int rfmf_graph_orig_ids(const rfmf_graph* g, int64_t* out) {
    try {
        return rfmf_graph_orig_ids_impl(g, out);
    } catch (const std::bad_alloc&) {
        return rfmf::fail(RFMF_ERR_NOMEM, "host allocation failed in rfmf_graph_orig_ids");
    } catch (...) {
        return rfmf::fail(RFMF_ERR_INVALID, "unexpected host exception in rfmf_graph_orig_ids");
    }
}
