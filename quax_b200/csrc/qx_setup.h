// qx_setup.h -- host-side set-up shared by every entry point that builds the
// device tables of a basis (qx_initialize and qx_compute_2e_int_noalloc):
// shell validation and Libint-convention normalisation, the primitive-pair and
// shell-pair records, and the Boys-function table.
#pragma once
#include <string>
#include <vector>

#include "qx_device.cuh"

namespace qx {

struct ShellTables {
    std::vector<int> l, nprim, atom, poff, bf;
    std::vector<double> alpha, coef;  // normalised contraction coefficients
    int nbf = 0;
};

// Validates the shells (l in [0, lmax], 1..64 primitives, atom index, positive
// finite exponents, finite coefficients, non-degenerate contraction) and
// normalises the contractions so that the x^l component of each contracted shell
// has unit norm (Libint's convention).  Returns QX_OK, or QX_E_INVALID /
// QX_E_UNSUPPORTED with `err` set (prefixed by `who`).
int normalize_shells(const char* who, int natom, int nshell, const int* shell_l, const int* shell_nprim,
                     const int* shell_atom, const double* exps, const double* coefs, int lmax, ShellTables& t,
                     std::string& err);

// Shell pairs s1 >= s2 in the reference's order, each in canonical orientation
// (higher angular momentum first), with their primitive-pair records; pcls is the
// pair class l1 (l1 + 1) / 2 + l2 of each, and nfull (if not null) the pair's number of
// primitive pairs before the negligible ones are dropped.
//
// A primitive pair is dropped when a bound on sqrt((ab|ab)) of it, raised by a factor
// for four nuclear derivatives, is below 1e-18 min(tol, 1e-10), tol being the Schwarz
// threshold, and below 1e-18 of the pair's largest: a quartet that passes the screening
// has a bound of at least tol, so what is left out lies two decades below the rounding
// of its integrals.  On the synthetic workloads (exponents 0.08 to 5e3, atoms 2 to 20
// bohr apart) half of the primitive pairs, and three quarters of the primitive quartets,
// carry an exp(-mu R^2) below that.
//
// all (if not null) receives every primitive pair of the s and p pairs, in order, and
// all_off its range per pair: the second-derivative programs of those classes sum
// weights of (2 alpha)^2 that cancel, and any other grouping of that sum is visible.
void build_pairs(const ShellTables& t, const double* coords, double tol, std::vector<PrimPair>& prims,
                 std::vector<PairInfo>& pairs, std::vector<int>& pcls, std::vector<int>* nfull = nullptr,
                 std::vector<PrimPair>* all = nullptr, std::vector<int>* all_off = nullptr);

// Boys table F_m(T_g) (BOYS_NG x BOYS_NM, row-major [g][m]); built once per
// process on first use.
const std::vector<double>& boys_table();

}  // namespace qx
