// bin.hpp -- shell binning of half spectra (k_bin.cu): what one lattice shape
// keeps between spectra, and the spectra themselves.
#pragma once
#include <vector>

#include "engine.hpp"
#include "sizes.hpp"

namespace lat {

struct BinArgs {
  int nx, ny, nz;
  const void* F[6];     // half spectra [z][y][nx/2+1]: one, two (cross) or the six pi_ij
  const double2* wtab;  // two-bin weights by |n|^2
  const double* sins;   // sin(2 pi i / n): x (nx/2+1), y, z
  int nbins;
  double* partials;     // [grid][sums][nbins]
  double* out;          // [sums][nbins]
  unsigned int* counter;
};

// Tables, scratch and the data-free weight sums of a lattice shape, made with its handle.
struct BinPlan {
  int nx = 0, ny = 0, nz = 0, nsm = 0;
  double2* wtab = nullptr;  // start of the plan's allocation
  double* sins = nullptr;
  double* partials = nullptr;
  double* out = nullptr;
  unsigned int* counter = nullptr;
  std::vector<double> Ww, Wc;  // two-bin weight sums and integer counts per shell

  int make(int nx, int ny, int nz, int nsm, cudaStream_t s);
  void free();
  // S = sum / W per shell (the plain sum where W = 0) and W, on the host
  int power(const void* F, int mode, int precision, int nbins, double* S, double* W, cudaStream_t s);
  int cross(const void* F1, const void* F2, int precision, int nbins, double* S_re, double* S_im, cudaStream_t s);
  int gw(const void* const* F, int precision, int nbins, double* S, double* W, cudaStream_t s);

 private:
  int sums(int kind, const void* const* F, int nf, int precision, int nbins, std::vector<double>& o, cudaStream_t s);
};

}  // namespace lat
