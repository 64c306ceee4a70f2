// Position arithmetic of Distribution layers (plain C++ and CUDA).
//
// The SNPs that a layer owns for one prefix are every step-th one from a first;
// a tile of a tensor kernel goes on past the last of them, up to 127 positions,
// and drops what lies at or past n.  Requests may name any step up to 2^31 - 1,
// so a position is computed with the step capped at n: a step of n or more owns
// one SNP all the same, and with n < 2^21 no position leaves 32 bits (128 x 2^21).
#pragma once

#include <climits>

#ifdef __CUDACC__
#define FIU_POS __host__ __device__ __forceinline__
#else
#define FIU_POS inline
#endif

namespace fiu {

// The step as positions count it.
FIU_POS int layer_step(int step, int n) { return step < n ? step : n; }

// Position m of the owned SNPs from `first` (step: layer_step's); an SNP when below n.
FIU_POS int layer_snp(int first, int step, int m) { return first + step * m; }

// Row (SNP position) of SNP j in the bit rows ordered by residue mod step
// (SNPs r, r + step, .. for r = 0, 1, ..; residue r holds n / step + (r < n %
// step) SNPs; step: layer_step's).
FIU_POS int residue_row(int j, int step, int n) {
    const int r = j % step, more = n % step;
    return r * (n / step) + (r < more ? r : more) + j / step;
}
// Its inverse: the SNP in a row.
FIU_POS int residue_snp(int row, int step, int n) {
    const int q = n / step, more = n % step;  // residues of q + 1 SNPs, then those of q
    const int in = more * (q + 1);
    return row < in ? row / (q + 1) + step * (row % (q + 1)) : more + (row - in) / q + step * ((row - in) % q);
}

// The step of a sample of a scan's prefixes, every stride-th one of those owned (stride >= 1): the most
// whole strides that a step holds (a sample that then ends early is still one of owned prefixes).
FIU_POS int sample_step(int step, long long stride) {
    const long long most = INT_MAX / step;
    return step * (int)(stride < most ? stride : most);
}

}  // namespace fiu
