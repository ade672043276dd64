// Products of the sphere Hamiltonians by splitting the Fock word (ed_split.cu).
#pragma once

#include <thread>
#include <tuple>

#include "ed_internal.h"

namespace edgb {

// What a split product needs of the Hamiltonian, kept by a built matrix.
struct SplitSource {
    int levels = 1;
    int N = 0;
    int norb0 = 0, norb1 = 0;       // one level: norb0 orbitals; two: the levels'
    int64_t sector_sum = 0;         // sum of the occupied orbitals' weights (ed_basis)
    HopTables hop0, hop1;           // hop weights of each level
};

inline SplitSource split_source(const ed_basis& b, const ed_terms& t)   // one level
{
    return SplitSource{1, b.N, b.norb, 0, b.sector_sum, t.hop, {}};
}

// One pass's lists (see ed_split.cu): per primary word the segment base, the
// class and, per gamma, the alpha entries (row base, weight's limb pair);
// per class and gamma the secondary entries.
struct SplitSide {
    int ntasks = 0, gammas = 1, nseg = 1, rows = 0, moves = 0, sbits = 0;
    DevBuf<int2> task;
    DevBuf<int> pbase, pcls, ssize, astart, lstart;
    DevBuf<int4> alpha;
    DevBuf<uint32_t> list;
    // moves of one secondary particle by each distance: segment bases and
    // weight rows per primary word, entries per class
    DevBuf<int> mstart, mbase, mlstart;
    DevBuf<int64_t> mweight;
    DevBuf<uint32_t> mlist;
};

struct SplitPlan {
    int64_t n = 0;
    int ea = 1;                     // exponent bound of the weights and the diagonal
    SplitSide native, trans;
    DevBuf<int> perm;               // native row -> transposed row
    DevBuf<int64_t> diag;           // the diagonal's limb pairs
    DevBuf<double> values;          // the diagonal, where a matrix-free product keeps it
    struct Scratch {
        DevBuf<int64_t> x, xt;      // x in fixed point, both orders
        DevBuf<int> part;           // per-block exponent maxima and the bound
        DevBuf<ulonglong2> acct;    // the transposed pass's exact sums
    };
    // a stream: the device, the handle and, for the per-thread default stream
    // (one handle, as many streams as threads), the thread
    using StreamKey = std::tuple<int, cudaStream_t, std::thread::id>;
    std::mutex mu;
    std::map<StreamKey, std::unique_ptr<Scratch>> scratch;
    // Held over all launches of a product, the kernel gated on x's bound
    // included: several operators share a plan through their terms, and two
    // threads may enqueue their products on one stream, whose scratch holds
    // one x at a time.
    std::mutex order;
};

struct SplitArgs {
    const int2* task;
    const int* pbase;
    const int* pcls;
    const int* ssize;
    const int* astart;
    const int4* alpha;
    const int* lstart;
    const uint32_t* list;
    const int* mstart;
    const int* mbase;
    const int2* mweight;
    const int* mlstart;
    const uint32_t* mlist;
    int gammas, nseg, rows, moves, sbits;
    const int2* x;
    const int* xexp;
    ulonglong2* acct;
    const int* perm;
    const int2* diag;
    double* y;
    int ea;
    bool gated;     // another kernel answers for a bound of 2047
};

// The plan of a Hamiltonian with the given diagonal (device, n entries), or
// null where it does not apply.  max_row bounds the elements of a row (0: not
// known).  Allocates and waits: not in a capture.
std::unique_ptr<SplitPlan> split_build(const SplitSource& s, const double* diag, int64_t n, int max_row, cudaStream_t st);
// The plan of a stored matrix: its own diagonal, its source's weights.
std::unique_ptr<SplitPlan> split_build_crs(const ed_crs& a, cudaStream_t st);
// The stream's scratch, made outside a capture where it takes at most half of
// the free device memory; false when it is missing.
bool split_ready(SplitPlan& p, cudaStream_t st);
// y = H x on a stream that split_ready accepted, p.order held; returns the device word with
// x's exponent bound (2047: a non-finite entry, y is all NaN; with mark also
// where an entry is lost in fixed point, and y is left to the caller's kernel).
const int* split_product(SplitPlan& p, const double* x, double* y, bool mark, cudaStream_t st);
// Gives back the stream's scratch (before a solver's stream is destroyed).
void split_release(SplitPlan& p, cudaStream_t st);

}  // namespace edgb
