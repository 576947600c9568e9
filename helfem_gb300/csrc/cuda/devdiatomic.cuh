// Device-resident diatomic context shared by the diatomic Fock-build kernels.
//
// Radial layout: element e owns an nn x nn primitive tile; primitive p is the
// global function g(e,p) = e*(nn-1) + p, valid for g < nrad. Dummy AO index
// = iang*nrad + irad (nd = nang*nrad); the pure index of (s, g) is
// poff[s] + g - pstart[s] for g >= pstart[s] (m != 0 shells drop g = 0).
// Matrices are column-major FP64.
#pragma once

#include "side_stream.hpp"

#include <cuda_runtime.h>

namespace hfg {

struct DevDiatomic {
  int nn, nel, nrad, nang, nd, nlm, rmax, Lmax, mmax, nM, nbf;
  const int* poff;       // [nang] pure index of (s, pstart[s])
  const int* pstart;     // [nang] first radial function of shell s in the pure basis
  // per (ilm, e) padded nn x nn tiles
  const double* p0;
  const double* p2;
  const double* q0;
  const double* q2;
  const double* cdB;     // [(ilm*nel+e)*2nn^2*rmax]
  const double* cds;     // [(ilm*nel+e)*rmax]
  const int* cdrank;     // [ilm*nel+e]
  const double* tx;      // [((ilm*nel+e)*4 + ab)*(nn^2)^2] exchange-ordered in-element kernel
  const double* lmfac;   // [ilm] 4 pi Rhalf^5 (L-|M|)!/(L+|M|)! (sign (-1)^M applied at use)
  // angular coupling table: (a, L, M) -> (b, c0 = cos^2 coupling, c2 = Gaunt)
  const int* al_ptr;
  const int* al_b;
  const double* al_c0;
  const double* al_c2;
  // Coulomb channels and bra lists
  int nchan;
  const int* ch_L;
  const int* ch_M;
  const int* ch_ilm;
  const double* ch_fac;
  const int* jbra_ptr;
  const int* jbra_chan;
  const double* jbra_c0;
  const double* jbra_c2;
  // exchange entries
  int nent;
  const int* kjk_ptr;    // [nang^2+1]
  const int* kent_L;
  const int* kent_Ma;
  const int* kent_ilm;
  const int* kent_jk;    // [nent] owning output block
  // shells ordered by m (ascending within an m): those of m are
  // msh[msh_ptr[m + mmax] .. msh_ptr[m + mmax + 1]); groups of at most 16 (and
  // of at most 8) consecutive shells of one m are msh[grp_ptr[g] ..), and
  // (L, |M|) of each multipole
  const int* mval;
  const int* msh;
  const int* msh_ptr;
  int ngrp, gmax;
  const int* grp_ptr;
  int ngrp8;
  const int* grp8_ptr;
  const int* lmL;
  const int* lmM;
  // element pairs: off-diagonal ordered pairs (a != b) and a < b pairs
  const int2* pairs_all;
  int npairs_all;
  const int2* pairs_sym;
  int npairs_sym;
  // split-precision copies: each FP64 value v as float2 (hi, lo), hi = fl32(v)
  const float2* p0s = nullptr;
  const float2* p2s = nullptr;
  const float2* q0s = nullptr;
  const float2* q2s = nullptr;
  const float2* al_c0s = nullptr;
  const float2* al_c2s = nullptr;
  const float2* lmfacs = nullptr;
  // P_L^|M| grows as e^{L mu} and Q_L^|M| decays as e^{-(L+1) mu}: beyond the
  // FP32 range at large L and mu. The split tables hold P * 2^-k and
  // Q * 2^+k with k = kexp[ilm*nel+e] (the exponent of the element's largest
  // P entry); an element pair (inner a, outer b) restores 2^(k_a - k_b) <= 1.
  const int* kexp = nullptr;
};

// In-element tiles of the split exchange on the tensor cores (dk_tc.cu): digit
// planes of the exchange-ordered kernel, and the scratch of one call
#define DTC_XDIGITS 6  // of a recoupled float-pair tile; one of FP64 has as many as the table
#define DTC_TDIGITS 7
#define DTC_TT 64
#define DTC_WAIT (1u << 20)  // polls of a completion wait before it gives up
struct DevDiaTC {
  int ksteps = 0, ntt = 0;            // K steps of 16 over 4 nn^2 columns, tiles of DTC_TT rows
  const unsigned char* tx = nullptr;  // [ilm][e][tile][K step][digit][DTC_TT x 16]
  const int* txexp = nullptr;         // [ilm][e][tile][DTC_TT] row exponents
  const int* cexp = nullptr;          // [ilm][e][4 nn^2] column exponents
  int cap = 0, lparts = 1;            // units of digits held at a time, parts of the multipole sum
  unsigned char* x = nullptr;         // [unit][ilm][K step][digit][128 x 16]
  int* xexp = nullptr;                // [unit][ilm][128]
  double* part = nullptr;             // [part][unit][tile][DTC_TT][128]
  int* err = nullptr;                 // set when a completion wait ran out
  unsigned wait = DTC_WAIT;
};

// Scratch of the in-element tiles of the FP64 exchange (dk_share.cu): units
// are (element, 8 output blocks)
struct DevDia64 {
  int cap = 0, lparts = 1;       // units of recoupled tiles held at a time, parts of the multipole sum
  int rsplit = 1, vsplit = 1;    // parts of the tile rows, threads that share a row
  double* x = nullptr;           // [unit][ilm][4 nn^2][8]
  unsigned int* xact = nullptr;  // [unit][ilm] rows with an entry (bits)
  double* part = nullptr;        // [part][unit][8][nn^2]
};

struct DevDiatomicScratch {
  double* jin;            // [nchan*nel*2*nn^2] in-element channel tiles, then the full channel tiles
  double* jscal;          // [nchan*nel*4]
  double* khalo;          // [nel*nel*nang^2*(2nn-1)]
  double* bnorm;          // [nang^2*DNORM_SPLIT]
  unsigned char* act;     // [nang^2] density block above the screen
  unsigned char* ent_act; // [nent]
  unsigned char* jk_act;  // [nang^2]
  int* jk_list;           // [2*nang^2]: active output blocks, then those with j <= k
  int* jk_pos;            // [nang^2] position in the call's list of output blocks, or -1
  int* kg_list;           // active (k*ngrp + g), then (k*ngrp8 + g) of the in-element items
  // [0] active output blocks, [1] those with j <= k, [2] and [3] the lengths of
  // the two kg lists, [4] item counter
  int* counts;
  float2* pd2;            // [nd*nd] split copy of the density (split path)
  // off-diagonal pairs in parts of the multipole sum: part sums of each item's
  // tiles, [part][item][gmax][nn^2] (offparts > 1 only)
  int offparts;
  double* offsum;
};

#define DNORM_SPLIT 8

// pure-m DFT grid: nq mu points per element, na nu points, npair unordered
// pairs of shells (s <= t) of one m, those of m < 0 with their m > 0 mirrors
struct DevDiatomicXC {
  int nq = 0, na = 0, npair = 0;
  const int4* pair = nullptr;    // [npair] s, t and the mirror shells of -m (or -1)
  const double* mult = nullptr;  // 2 (s != t) or 1
  const double* W = nullptr;     // [k*na + a]: Y_s Y_t
  const double* Wt = nullptr;    //             Y_s' Y_t + Y_s Y_t'
  const double* WT = nullptr;    // [a*npair + k]: the same, transposed
  const double* WtT = nullptr;
  const double* R = nullptr;     // [(e*nq + q)*nn + p]
  const double* dR = nullptr;
  const double* w = nullptr;     // [(e*nq + q)*na + a]
  const double* hinv = nullptr;
};
struct DiatomicXcScratch {
  double* D;      // [nsd][nel][npair][nq]  mult * B^T P_st B (and the mirror's)
  double* Dr;     // same                   mult/2 * (dB^T P_st B + B^T P_st dB)
  double* F;      // [nout][3][nel][nq][na]
  double* U;      // [nout][3][nel][npair][nq]
  double* epart;  // [nel*blocks of points][2]
};
// blocks of grid points of one element
constexpr int DXC_POINTS = 32;  // one warp: the functional is a long serial chain, few points still fill the SMs
inline int dxc_blocks(int nq, int na) { return (nq * na + DXC_POINTS - 1) / DXC_POINTS; }
// Pb == nullptr: restricted (Pa is the total density, Ha the potential).
// Densities and potentials are in the pure basis (nbf x nbf, column-major);
// H is overwritten. energies (device, may be null) receives {Exc, Nel}.
cudaError_t launch_diatomic_xc(const DevDiatomic& D, const DevDiatomicXC& X, const DiatomicXcScratch& S, int xid,
                               int cid, const double* Pa, const double* Pb, double* Ha, double* Hb, double* energies,
                               double thr, cudaStream_t st);

// exchange tiles with the recoupling shared by the output blocks of one k
// (dk_share.cu): off-diagonal element pairs (FP64, or float pairs), and the
// in-element tiles in FP64
cudaError_t launch_dk_share_off(const DevDiatomic& D, const DevDiatomicScratch& S, const double* Pd, double* Kd,
                                bool symmetric, bool split, cudaStream_t st);
cudaError_t launch_dk_share_diag(const DevDiatomic& D, const DevDiatomicScratch& S, const DevDia64& T,
                                 const double* Pd, double* Kd, bool symmetric, cudaStream_t st);

cudaError_t launch_diatomic_expand(const double* P, int nbf, const int* pure, double* Pd, int nd, cudaStream_t st);
cudaError_t launch_diatomic_gather(const double* Fd, int nd, const int* pure, int nbf, double* F, cudaStream_t st);
cudaError_t launch_diatomic_tx(const DevDiatomic& D, double* tx, cudaStream_t st);
// J of a pure-basis density, written to the pure-basis J (overwritten)
cudaError_t launch_diatomic_coulomb(const DevDiatomic& D, const DevDiatomicScratch& S, const double* P, double* J,
                                    cudaStream_t st);
// one output block per item, FP64 (short elements)
cudaError_t launch_diatomic_exchange_items(const DevDiatomic& D, const DevDiatomicScratch& S, const double* Pd,
                                           double* Kd, bool symmetric, cudaStream_t st);
// tc: the in-element tiles on the tensor cores, or nullptr for the FP64 kernels (T)
cudaError_t launch_diatomic_exchange(const DevDiatomic& D, const DevDiatomicScratch& S, const DevDia64& T,
                                     const DevDiaTC* tc, const double* Pd, double* Kd, bool symmetric, cudaStream_t st,
                                     const SideStream& side);
cudaError_t launch_dk_tc_table(const DevDiatomic& D, const DevDiaTC& T, unsigned char* tx, int* txexp, int* cexp,
                               cudaStream_t st);
cudaError_t launch_dk_tc_diag(const DevDiatomic& D, const DevDiatomicScratch& S, const DevDiaTC& T, const double* Pd,
                              double* Kd, bool symmetric, bool itemwise, cudaStream_t st);
// split-precision exchange: off-diagonal element pairs in float pairs, the
// in-element tiles on the tensor cores; itemwise: their recoupled tiles one
// output block at a time (bitwise the same K)
cudaError_t launch_diatomic_exchange_split(const DevDiatomic& D, const DevDiatomicScratch& S, const DevDiaTC& T,
                                           const double* Pd, double* Kd, bool symmetric, cudaStream_t st,
                                           const SideStream& side, bool itemwise = false);

}  // namespace hfg
