// y = H x on the 5th-generation tensor cores: H of the Sz sector written as products of
// small matrices (tensor.cu), its FP64 operands split into exact bf16 digits.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <functional>
#include <vector>

namespace ae {

constexpr int kTcVecDigits = 7;  // base-512 digits of a vector element (63 bits below the vector's scale)
constexpr int kTcMatDigits = 7;  // base-512 digits of a matrix element (63 bits below the matrix's scale)

// Launch shape and device tables of one integral Hamiltonian (or of one per instance),
// and the workspace of the product.  Pointers belong to the engine's allocators.
struct TcProduct {
    bool ok = false;
    int N = 0, P = 0, Pp = 0, nch = 0, Kp = 0;  // orbitals, orbital pairs p <= q, padded columns, 32-column chunks, padded rows
    int nA = 0, nB = 0, mtA = 0, mtB = 0;       // strings, 128-string tiles
    int nkB = 0, nnB = 0, nkA = 0, nnA = 0;     // same-spin blocks: row chunks, column blocks
    int slots = 0, vbufs = 0;                   // shared-memory buffers of one digit's tile, of a unit's columns
    size_t smem = 0;
    bool row_sums = false;                      // a beta string's row of y is summed in shared memory
    int sm_count = 0;
    bool shared = true;                         // one Hamiltonian for every instance
    bool square = false;                        // as many alpha as beta electrons

    // tables that depend on the strings only
    const int32_t *rows = nullptr;    // [nB][Kp] beta string read by row k (nB: the zero row)
    const int32_t *code = nullptr;    // [nB][Kp] its row of vt: the orbital pair (P: zero), + P + 1 where the sign is -
    const uint16_t *tgt = nullptr;    // [mtA][Pp / 8][128][8] alpha target << 2 | 1 valid | 0x8000 negative
    const int *min_target = nullptr;  // [mtA][nch] smallest target of a tile's chunk
    const uint32_t *flip_cost = nullptr;  // [nB * mtA + 1] cost of the steps before each, spin-flip symmetric vectors
    // integrals, per instance unless shared
    const uint16_t *vt = nullptr;     // [2 (P + 1)][chunk][digit][width] digits of (pq|rs), of -(pq|rs)
    const uint16_t *hsB = nullptr, *hsA = nullptr;  // [block][chunk][Kp / 8][digit * width / 8][8][8] same-spin digits
    const double *diag = nullptr;     // diagonal of H
    const double *scale = nullptr;    // per Hamiltonian: matrix scales S_V, S_H and the vector scale's norm factor
    size_t vt_inst = 0, hsB_inst = 0, hsA_inst = 0;

    // workspace of `chunk` instances
    int chunk = 0, W = 1;
    uint16_t *G1 = nullptr, *G2 = nullptr;
    size_t g1_vec = 0, g2_vec = 0;    // 16-byte pieces per vector
    unsigned long long *sig = nullptr, *Pb = nullptr, *Pa = nullptr;
    void *head = nullptr;
    double *part = nullptr;
    int ngx = 0;                      // energy partial sums per instance
    int scan_grid = 0;                // CTAs per instance of the vector scan
};

struct TcBasis {
    int N, na, nb;
    const std::vector<uint32_t> *strA, *strB;
    const std::vector<int32_t> *rankA, *rankB;
    const uint32_t *dA, *dB;  // strings on the device
};

using TcAlloc = std::function<void *(size_t bytes)>;

// Whether the shapes fit the kernel (shared memory, table widths) and pay.
bool tc_shape(TcProduct &t, const TcBasis &B, int sm_count, int smem_optin);
// Workspace bytes of one instance.
size_t tc_workspace(const TcProduct &t, int W);
// Whether the integrals g2s of ntab Hamiltonians are finite and have the symmetry (pq|rs) = (qp|rs) = (pq|sr).
bool tc_symmetric(int N, const double *g2s, int ntab);
// String tables, digit tables of ntab Hamiltonians (host h1s/g2s, device copies d_h1/d_g2),
// of integrals that tc_symmetric takes.  False (t.ok cleared): the digits' exactness bound does not
// hold, a same-spin element is not finite, or an allocation failed.  Values only (same shape):
// tables are rewritten in place.
bool tc_build(TcProduct &t, const TcBasis &B, const double *h1s, const double *g2s, const double *d_h1,
              const double *d_g2, const double *diag, int ntab, const TcAlloc &alloc, bool values_only, cudaStream_t s);
bool tc_alloc_workspace(TcProduct &t, int W, int max_inst, const TcAlloc &alloc, cudaStream_t s);
// y = H x of ninst vectors of D * W doubles.  bad[b] != 0 after the stream reached this
// point: instance b was left to the caller's other product (a value that is not finite
// or out of the digits' range, or, with elements -- y goes to a caller who may look at single
// elements -- a vector of too wide a range).  epart: ngx partial sums of <x|y> per instance
// (nullable).  flip_tol2 < 0: do not use psi(a,b) = psi(b,a); flip_sums: its test's two
// sums per instance, for the caller's other product (nullable).  Returns kernel launches.
int tc_apply(const TcProduct &t, const double *x, double *y, int ninst, const int *active, bool elements, double flip_tol2,
             int *flip_used, double *flip_sums, int *bad, double *epart, cudaStream_t s);

}  // namespace ae
