// Launcher of the frame form of the spin-pair gradient (gradient_frame.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace vbcore {

constexpr int kAdjointMaxParts = 148;  // CTAs of the table adjoint, one per SM

struct FrameAdjointArgs {
    int n, k, n_strings, R, r_pos;
    const uint64_t* occ;
    const double* S;
    const double* h;
    const double* lf;   // factor columns, lf[q * ld + m]
    int ld;
    const double* tables;  // frame tables of the evaluation (launch_spin_tables)
    const int* rlist;      // right strings of every left string, as SpinTableArgs
    const unsigned* rdesc;
    const int* ebound;
    const double* adj;     // record adjoints, even stride: [u (R), determinant, energy]
    long long adj_stride;
    // instead (weight not null): one determinant per string u, of weight weight[u] and with the opposite
    // string partner[u] in the same table, and a spin-flip symmetric list; the adjoint of (u, v) is then
    // 2 (1 + [u < v]) weight[u] weight[v] times [sigma u, H - lambda S, S] of the partners' record
    const double* weight;
    const int* partner;
    const double* records;
    long long rec_stride;
    double lambda;
    unsigned long long* task_counter;   // zero
    unsigned long long* careful_count;  // zero; pairs left to the exact kernel
    unsigned long long* careful_list;
    unsigned long long* unsound_count;  // zero; strings left to the pair-by-pair kernels (kFrameCondition2)
    int* unsound;                       // n_strings
    double* out;      // n_strings blocks of frame_adjoint_block_doubles
    double* partial;  // kAdjointMaxParts x (np R + 2 n^2)
    double* gL;       // [pair * ld + m], added to
    double* gS;       // n x n, added to
    double* gh;
};

size_t frame_adjoint_block_doubles(int n, int k, int R);
bool frame_adjoint_supported(int n, int k, int R);
cudaError_t launch_frame_adjoint(const FrameAdjointArgs& a, cudaStream_t s);

}  // namespace vbcore
