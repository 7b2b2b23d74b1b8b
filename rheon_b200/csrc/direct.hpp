// Fast diagonalisation of the sealed box, the preconditioner of the
// mixed-precision pressure method on the grids it covers (new; the reference
// has no direct solve).
//
// The 7-point sealed-box operator on a uniform grid is a sum of one-axis
// operators, each diagonal in the orthonormal cosine basis
// c_q(i) = s_q cos(pi q (2i + 1) / 2n) with eigenvalue 4 w sin^2(pi q / 2n)
// (Lynch, Rice and Thomas, "Direct solution of partial difference equations by
// tensor product methods", 1964). z = K^+ r is therefore three forward
// transforms, one division by the sum of the eigenvalues (the constant mode is
// set to 0) and three inverse transforms, all in FP32. The outer iteration is
// FP64 iterative refinement: p += z - z[0], r = b - K p, accepted on that true
// residual. The FP32 rounding leaves about 1e-5 of a smooth residual and 1e-6
// of a rough one, so a solve takes two iterations to 1e-8 and three to 1e-12,
// where flexible CG with the V-cycle takes 7 and 10.
//
// The transforms are dense products with the basis (a contraction of length
// n, at most 512), halved by the basis' symmetry: with e_i = x_i + x_{n-1-i}
// and o_i = x_i - x_{n-1-i}, the even coefficients need only e and the odd
// ones only o. Coefficients are stored even ones first.
#pragma once

#include <vector>

#include "internal.hpp"

namespace rb200 {

struct SolveState;

constexpr int kDctMaxAxis = 512;
constexpr size_t kDctSmemMax = 200 * 1024;  // of a transform's block

// One axis' transform: tables are k-major ([k][m], rows of mP floats, padded
// with zeros) so that a thread's outputs are consecutive in a row.
struct DctAxis {
    int n, ne, no;        // length, even and odd coefficients
    int neP, noP;         // ne and no rounded up to 4 (the contraction lengths)
    int mP;               // outputs rounded up to 4 RM MB
    int RM, MB;           // outputs per thread, warps along the outputs
    const float *fe, *fo; // forward: [i][q]
    const float *ie, *io; // inverse: [q][i]
    const float* lam;     // eigenvalues in stored order
};

// One transform pass over a grid's lines along one axis.
struct DctJob {
    DctAxis A;
    int inner;            // stride of a line's elements (1: rows along x)
    int lines;            // n-element lines
    int nb;               // a tile has 32 nb lines
    int tiles;
    int n0;               // row length (the eigenvalues of a z line)
    const float* src;
    const double* src64;  // the FP64 right-hand side read by a cold solve's first pass, or nullptr
    float* dst;
    const float *lam0, *lam1;
};

// The three axes' tables of a grid, in one device allocation.
class DctTables {
public:
    DctTables() = default;
    ~DctTables();
    DctTables(const DctTables&) = delete;
    DctTables& operator=(const DctTables&) = delete;
    int init(const GridDev& g, cudaStream_t s);
    DctAxis axis[3];
    size_t bytes() const { return bytes_; }

private:
    float* data_ = nullptr;
    size_t bytes_ = 0;
};

// Whether the direct preconditioner covers a grid: more than 8 cells along
// some axis (smaller boxes are solved densely in FP64), at most 512 along each
// (the tile shapes), and a condition below 10^9.
bool direct_supported(const GridDev& g);

// The passes of one application, in order: x, y forward, z forward, division
// and inverse, y, x inverse. r32 -> z through `z` in place; b is read instead
// of r32 by the first pass of a cold solve. `alone`: the grid has the chip to
// itself (an instance of a batch does not).
void direct_jobs(const DctTables& T, const GridDev& g, const double* b, const float* r32, float* z, bool alone,
                 DctJob (&jobs)[5]);
size_t direct_job_smem(const DctJob& J);

class DirectSolver {
public:
    DirectSolver() = default;
    ~DirectSolver();
    DirectSolver(const DirectSolver&) = delete;
    DirectSolver& operator=(const DirectSolver&) = delete;

    int init(const GridDev& g, cudaStream_t s);
    // A seeded solve's first residual: r32 = f32(b - K p), accepted or not.
    int enqueue_seed(const GridDev& g, SolveState* st, const double* b, double* p, double* p2, Partials part,
                     cudaStream_t s) const;
    // One refinement iteration; p alternates between the two buffers (the
    // state's dsel tells which holds it). Returns the number of launches.
    int enqueue_iteration(const GridDev& g, SolveState* st, const double* b, double* p, double* p2, Partials part,
                          rb200_trace* trace, cudaStream_t s) const;
    // Copies a finished iterate from p2 to p where it ended there; p = 0 where
    // the solve ended before its first iteration.
    int enqueue_settle(const GridDev& g, SolveState* st, double* p, const double* p2, cudaStream_t s) const;
    size_t bytes() const { return bytes_; }

private:
    DctTables tables_;
    float* r32_ = nullptr;
    float* z_ = nullptr;
    size_t bytes_ = 0;
};

}  // namespace rb200
