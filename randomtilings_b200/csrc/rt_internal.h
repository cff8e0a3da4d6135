// rt_internal.h -- declarations shared by the C-ABI layer and the kernels.
#pragma once

#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "../../include/rt_b200.h"

namespace rtb {

struct WalkArgs;

enum Family : int {
    FAM_DOMINO = 0,      // dominokernel.cl, int8
    FAM_DOMINO_HB = 1,   // dominokernelCFTP.cl, int8
    FAM_LOZENGE8 = 2,    // lozengekernel.cl, int8
    FAM_QLOZENGE8 = 3,   // qlozengekernel.cl; int8 (the reference's int states are below 64)
    FAM_RECTTRI = 4,     // recttrianglekernel.cl, int32
    FAM_TRIDIMER = 5     // triangledimerkernel.cl, 8 int32 arrays
};

// The most colour steps one call may ask for, about 1.1e12: weeks of device
// time even on small lattices.  Every entry point that sizes a schedule or a
// phase list from a step or sweep count refuses larger counts first, so no
// size computed from a count can wrap.
constexpr int64_t kMaxColourSteps = int64_t(1) << 40;

// The largest tiling side a walk accepts: the kernels index a lattice with
// 32-bit integers, and a side of 32,767 keeps every index below 2^31.
constexpr int kMaxTilingSide = 32767;

struct WalkPlan {
    int items = 0;
    int block = 0;
    int rows_per_cta = 0;
    int ctas = 0;
    size_t smem = 0;
    int wpad = 0;    // shared-memory row stride (elements)
    int xwords = 0;  // exchange words per halo row
    int xslots = 1;  // arrays exchanged per phase
    int depth = 1;   // band kernels: phases per halo exchange
    int pwords = 0;  // bit-plane kernel: words per row
    bool cluster = false;     // the CTAs are one thread-block cluster (else a cooperative launch)
    bool merge_runs = false;  // the kernel takes a run of same-colour steps as one phase
    const void* fn = nullptr;
};

rt_status plan_walk(int family, int device, int nlat, int rows, int cols, int width, bool uniform, bool philox,
                    WalkPlan* plan, std::string* err);
// Lets kernel `fn` use `smem` bytes of dynamic shared memory; an error if a block
// cannot have them beside the kernel's static ones.  What is set is all there is:
// the limit is the function's, so a plan that set its own size would take it from
// the larger plan of another handle (or thread).
rt_status allow_shared(const void* fn, int device, size_t smem, std::string* err);
// Launch configuration of a one-cluster plan; `attr` outlives *cfg.
void walk_launch_config(const WalkPlan& plan, cudaLaunchConfig_t* cfg, cudaLaunchAttribute (&attr)[1]);
rt_status launch_walk(const WalkPlan& plan, WalkArgs& args, cudaStream_t stream, std::string* err);
// Word-parallel kernels of the int8 models: uniform TinyMT32J parameters or fast
// mode.  On bands with halo rows (plan_word_band) where they fit, else rt_word.cu.
// ctas_hint 0: a grid by size; < 0: so too, and rt_word.cu only.
bool word_family(int family);
// weighted: the instantiation that reads per-site thresholds (WalkArgs::wper > 0).
rt_status plan_word_walk(int family, int device, int nlat, int rows, int width, bool philox, int ctas_hint,
                         WalkPlan* plan, std::string* err, bool weighted = false);
// One word per thread, on bands with halo rows (rt_wordband.cu); an error if the
// bands do not fit it.
rt_status plan_word_band(int family, int device, int nlat, int rows, int width, bool philox, int ctas_hint, bool weighted,
                         WalkPlan* plan, std::string* err);
// Bit-plane kernel of a single triangle-dimer walk (rt_td.cu), for arrays whose
// values fit its planes, on one cluster of ctas_hint CTAs (<= 0: by size).
rt_status plan_td_walk(int device, int rows, int width, bool philox, int ctas_hint, WalkPlan* plan, std::string* err);
// Rectangle-triangle kernel (rt_recttri.cu), one site per thread: bands of up to
// 1,024 sites.  ctas_hint <= 0: by size.
rt_status plan_recttri_walk(int device, int rows, int width, bool philox, int ctas_hint, WalkPlan* plan,
                            std::string* err);
// Bit-plane kernels of the int8 models (RT_RNG_PLANES): rt_planeband.cu up to 2,048
// words a CTA, else rt_plane.cu.  ctas_hint / depth_hint <= 0: by size, a depth of up
// to 32 / one CTA per SM, up to 8.
rt_status plan_plane_walk(int family, int device, int nlat, int rows, int width, int ctas_hint, int depth_hint,
                          WalkPlan* plan, std::string* err);
// The kernel a walk runs on, as every walk entry point chooses it: the
// bit-plane kernels in RT_RNG_PLANES mode; otherwise the word kernels for the
// int8 models with uniform generator parameters (unless kernel_choice = 1),
// the triangle dimers' bit-plane kernel for arrays whose values fit it
// (td_fits), and the rectangle-triangle kernel; falling back to the generic walk
// kernel for every other case and for any band those kernels cannot hold
// (kernel_choice = 2 forbids the fallback).
rt_status choose_plan(int family, int device, int nlat, int rows, int cols, int width, bool uniform, bool fast,
                      bool planes, bool weighted, bool td_fits, int kernel_choice, int ctas_hint, int depth_hint,
                      WalkPlan* plan, std::string* err);
// kind: 0 domino, 1 lozenge, 2 rect-triangle, 3 triangle-dimer (merge only).
rt_status launch_split(bool merge, int elem_bytes, int kind, int ncol, int n, int32_t* tiling, void* const* arr,
                       cudaStream_t stream, std::string* err);

// Fast-mode schedules (rt_capi.cu).  kind: 0 domino, 1 lozenge,
// 2 rect-triangle, 3 triangle dimer.  fast_step_phases appends the phases of
// step s of an epoch; fast_phases appends a whole walk of `steps` steps
// (with the final Update of the colour models, or the triangle dimers' pending
// refreshes).
class TdSchedule;
int64_t fast_step_phases(int kind, int64_t s, uint32_t* ph, int64_t at, uint32_t* prev, TdSchedule* td);
// Appends a bit-exact colour step of a two- or three-colour model: a phase of
// its own, or (merge) one more step of the run that `ph` ends with, if that
// run began at or after index `first`, the epoch's first phase.
int64_t colour_step_phase(uint32_t colour, bool merge, int64_t first, uint32_t* ph, int64_t at, uint32_t* prev);
void fast_phases(int kind, int64_t steps, std::vector<uint32_t>& ph);
// Integer threshold K with (k * 2^-23 < x) <=> (k < K) for k in [0, 2^23).
uint32_t below_threshold(double x);
// Integer acceptance thresholds of a kernel family on the 23-bit draw.
void family_thresholds(int family, double q, int qcmp, uint32_t thr[4]);

// Faces M of a side of a domain of `dlen` entries (dominoes M x M, lozenges M
// x 2M), -1 if there is no such domain (rt_host.cpp).
int domain_side(int model, int64_t dlen);

// Vertex kinds and in-domain edge bits of a domino / lozenge domain
// (rt_host.cpp), the graph of the height plans.
bool lipschitz_graph(int model, const int32_t* d, int64_t dlen, int* n_out, std::vector<uint8_t>* kind,
                     std::vector<uint8_t>* edges);

// Boundary heights of a domino / lozenge domain (rt_host.cpp): the vertex
// indices reachable from the first boundary vertex along boundary edges and
// their heights (0 at the start), in visiting order; vertex side in *n_out.
bool boundary_walk(int model, const int32_t* d, int64_t dlen, int* n_out, std::vector<int64_t>* idx,
                   std::vector<int32_t>* h);

// Six-vertex height rows on the host (rt_host.cpp).  Narrowing saturates.
// sixv_row_ok: row i (and `above`, row i - 1, null for i = 0) of the heights of an
// n x n domain wall: boundary values, and edges that join heights differing by 1.
// Rows that all pass are exactly a domain-wall height function: every face then
// lies within n / 2 edges of the boundary's 0..n <= 32,000 and, modulo 2^16,
// between the extremal heights, which no saturated value is.
void sixv_narrow_row(const int32_t* from, int count, int16_t* to);
bool sixv_row_ok(const int16_t* row, const int16_t* above, int n, int i);
void sixv_widen(const int16_t* from, size_t count, int32_t* to);

// The eight arrays of a triangle-dimer tiling (device pointers; array c at
// arrays + c stride), and in *over whether some value does not fit a dimer
// cover's bits (cover) or the bit planes (rt_walk.cu).
rt_status launch_td_split(const int32_t* tiling, int n, bool cover, int32_t* arrays, size_t stride, uint32_t* over,
                          cudaStream_t stream, std::string* err);

// Counts differing 32-bit words of a and b (bytes must be a multiple of 4).
rt_status launch_count_diff(const void* a, const void* b, size_t bytes, unsigned long long* d_count,
                            cudaStream_t stream, std::string* err);

}  // namespace rtb
