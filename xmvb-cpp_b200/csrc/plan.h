// The structure H/S plan object shared by the plan, gradient and solver translation units.
#pragma once

#include <cuda_runtime.h>

#include <utility>
#include <vector>

#include "internal.h"
#include "kernels.h"

using namespace vbcore;

// Term segments of the band reduction per row tile of every structure group (see BandReduceArgs).
struct BandSegments {
    int n_groups = 0, seg_max = 0;
    DeviceBuffer off, meta, coef, row;
    // tiles of every group (CSR: tile_off[g] .. tile_off[g + 1]), their first and last rows
    DeviceBuffer first_row, last_row, tile_off;
    // instead (groups not empty): rows of every group together, terms by structure in the groups' order
    DeviceBuffer groups, rows, order, term_row;
    int group_rows = 0;
};

// Blocks of (alpha strings) x (beta strings) the determinant list is ordered by (see BlockPairArgs).
struct PlanBlocks {
    int n = 0;
    int max_a = 0, max_b = 0, max_dets = 0;
    DeviceBuffer first, strings;
    std::vector<int> first_host;
};

// Pair lists of a covalent determinant list (CovalentArgs); empty where it is not one.
struct CovalentPlan {
    DeviceBuffer det, beta, list, desc, bounds, listed;
};

constexpr int kPlanCounters = 17;

struct vb_hs_plan {
    vb_context* ctx = nullptr;
    int n = 0, ka = 0, kb = 0, np = 0, gd = 0;
    int n_str = 0;
    long long n_det = 0;
    int Na = 0, Nb = 0;
    bool shared_tables = false;
    DeviceBuffer occ_a, occ_b, det_alpha, det_beta;
    DeviceBuffer rec_a, rec_b, tables_a, tables_b;
    int stride_a = 0, stride_b = 0;
    long long npairs_a = 0, npairs_b = 0;
    // counters: [0, 1] listed (exact-path) spin pairs alpha/beta, [4, 5] the frame kernel's task counters alpha/beta, [7] the band reduction's
    // timeout flag, [8, 9] pairs the frame kernel evaluated outside the certificate alpha/beta,
    // [10] listed covalent determinant pairs, [11 .. 13, 14 .. 16] the gradient's listed pairs, strings
    // outside the frame form and task counter alpha/beta
    DeviceBuffer counters, list_a, list_b;
    // right strings of each left string bucketed by hole set (see SpinTableArgs::rlist)
    DeviceBuffer rlist_a, rlist_b, rdesc_a, rdesc_b, ebound_a, ebound_b;
    int rec_stride_alloc = 0;  // record stride the spin-pair records are allocated for
    DeviceBuffer S_in, h_in, eri_in, gamma, kfull;
    // pair-kernel factorization: lf[q * np + m], scratch, signs, meta = {r_pos, r_neg} (+ host copy)
    DeviceBuffer lf, fwork, fcols, fsigns, fmeta;
    int* meta_host = nullptr;
    int R = 0, r_pos = 0;
    std::vector<long long> bands;  // determinant columns of the bands (they live in the context scratch)
    long long band_ld = 0;         // band row stride (a multiple of 32 elements)
    PlanBlocks blocks;
    DeviceBuffer Hout, Sout;
    DeviceBuffer str_off, str_det, str_coef;
    // structure incidence by determinant (CSR) and the gradient's adjoint scratch
    DeviceBuffer det_off, det_str, det_coef;
    DeviceBuffer adj_a, adj_b, grad_acc;
    // host inputs of the last host-pointer evaluation whose records are still resident
    std::vector<double> last_inputs;
    bool tables_current = false, records_current = false;
    BandSegments segments;
    CovalentPlan covalent;
    // spin-flip map of the determinant list (folds the determinant-pair work in half)
    DeviceBuffer flip;
    // determinants by alpha string (CSR: alpha_off[i] .. alpha_off[i + 1] index alpha_dets)
    DeviceBuffer alpha_off, alpha_dets;
    bool has_flip = false;
    bool single_determinants = false;  // (has_flip) no alpha string carries two determinants
    // internal position of each determinant of the caller's list when the plan reorders them
    // (empty: the caller's order), host copy and device copy
    std::vector<long long> det_position;
    DeviceBuffer det_position_dev;
    long long det_pair_evaluations = 0;  // unordered determinant pairs evaluated (orbit representatives)
    vb_hs_stats stats{};
    bool evaluated = false;
    // phase timing: per phase a pool of (start, stop) event pairs, `used` pairs this execute
    bool timing = false;
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> events[VB_PHASE_COUNT];
    int used[VB_PHASE_COUNT] = {};
    ~vb_hs_plan() {
        if (meta_host) cudaFreeHost(meta_host);
        for (auto& v : events)
            for (auto& e : v) {
                cudaEventDestroy(e.first);
                cudaEventDestroy(e.second);
            }
    }
};


namespace vbcore {

vb_status upload(vb_context* ctx, DeviceBuffer& buf, const void* src, size_t bytes);
int record_stride(int R);
SpinTableArgs table_args(vb_hs_plan* p, bool beta, const double* S, const double* h, const double* eri);
FullPairArgs full_args(vb_hs_plan* p);
// Uploads host inputs (mem == VB_MEM_HOST), builds the integral tables and the pair-kernel
// factorization, and evaluates every spin-pair record; *dS, *dh, *deri receive the device
// copies of the inputs.
// True when the resident inputs and frame tables are those of exactly these host inputs.
bool inputs_match(const vb_hs_plan* p, const double* S, const double* h, const double* eri, int mem);
vb_status prepare_spin_records(vb_hs_plan* p, const double* S, const double* h, const double* eri, int mem,
                               const double** dS, const double** dh, const double** deri, int* launches);
// The second half of it: the records, from the frame tables.
vb_status evaluate_spin_records(vb_hs_plan* p, const double* dS, const double* dh, const double* deri, int* launches);

}  // namespace vbcore
