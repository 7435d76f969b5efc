// Internal launch helpers shared between libxdem's translation units.
#pragma once

#include <cuda_runtime.h>

#include "xd_internal.cuh"

namespace xd {

// cell grid (xd_grid.cu)
unsigned key_bits_for(unsigned ncell);
size_t reorder_scratch_bytes(unsigned n);
struct HistTable;   // xd_physics64.cuh: tangential-spring history of a scene

int launch_hash(const Params& P, unsigned* hash, unsigned* index, const double* pos, unsigned n,
                unsigned sid, cudaStream_t s);
int launch_fill_cells(unsigned* cstart, unsigned* cend, unsigned ncell, cudaStream_t s, unsigned* err = nullptr);
// The cell ranges of n keys already sorted in hash (with their values in
// index): cstart/cend at the runs' ends, sorted_index = index; a key >= ncell
// is skipped and raises *err.  Cells without keys are left as they are.
int launch_cell_bounds_sorted(unsigned* hash, unsigned* index, unsigned* cstart, unsigned* cend,
                              unsigned* sorted_index, unsigned n, unsigned ncell, unsigned* err, cudaStream_t s);
// check: wait, and report a key >= ncell.  word (nullable): an error word in
// host memory that the call has to itself until then.
int reorder_and_find_cell_start(unsigned* hash, unsigned* index, unsigned* cstart, unsigned* cend,
                                unsigned* sorted_index, unsigned n, unsigned ncell, void* scratch,
                                cudaStream_t s, bool check, unsigned* word = nullptr);

// integrator (xd_integrate.cu)
int launch_vv_position(const Params& P, double* pos, const double* vel, const double* acc,
                       unsigned np, cudaStream_t s);
int launch_vv_velocity(const Params& P, double* vel, double* acc, double* omega, double* alpha,
                       double* force, double* moment, const double* mass, const double* inertia,
                       unsigned np, cudaStream_t s);
int launch_vv_velocity_position(const Params& P, double* pos, double* vel, double* acc,
                                double* omega, double* alpha, double* force, double* moment,
                                const double* mass, const double* inertia, unsigned np,
                                cudaStream_t s);

// FP64 contacts (xd_contact64.cu)
int launch_p2p(const Params& P, const double* pos, const double* vel, const double* omega,
               double* force, double* moment, const double* mass, const unsigned* sorted,
               const unsigned* cstart, const unsigned* cend, const xd_contact_property* cp,
               unsigned np, cudaStream_t s, const HistTable* ht = nullptr);
int launch_cylinder(const Params& P, const xd_cylinder_info* cyl, const xd_contact_property* cp,
                    const double* pos, const double* vel, const double* omega, double* force,
                    double* moment, const double* mass, unsigned np, const double* mpos, double* mf,
                    double* mm, cudaStream_t s);
int launch_planes(const Params& P, const xd_plane_info* planes, const xd_contact_property* cps,
                  unsigned cp_stride, unsigned nplanes, const double* pos, const double* vel,
                  const double* omega, double* force, double* moment, const double* mass,
                  unsigned np, cudaStream_t s, const HistTable* ht = nullptr);
size_t polygon_scratch_bytes(unsigned np, unsigned nbodies);
int launch_polygon(const Params& P, const xd_polygon_info* dpi, xd_polygon_mass_info* dpmi,
                   const double* pos, const double* vel, const double* omega, double* force,
                   double* moment, const double* mass, const unsigned* sidx,
                   const unsigned* cstart, const unsigned* cend, const xd_contact_property* cp,
                   unsigned nbodies, void* scratch, cudaStream_t s, const HistTable* ht = nullptr);
// The end of a graph step of the mixed form (its advance and, beside it, the
// mesh update): blocks of both that have to finish, and the words they share
// (nullptr: launched directly, nothing to gate).
//   words[kStepDone]  blocks done and, in the next word, those that raised the
//                     flag (one 8-byte word, reset by the last block: what it
//                     needs to know comes with its own atomic)
//   words[kStepFlag]  a re-binning is due (raised ahead of the call, and by
//                     direct launches)
//   words[kStepStop]  the flag as the last finished step left it: the steps
//                     that follow in the graph do nothing until it is cleared
//   words[kStepTodo]  contact passes left in the call
// first: the call's first advance (no contact pass precedes it).  tail: the
// graph ends with this step: rebin is set where a re-binning is due, more (if
// loop) where passes are left.
enum { kStepFlag = 0, kStepStop = 34, kStepTodo = 35, kStepDone = 36 };   // (stop and todo in one 8-byte word)
struct StepGate {
    unsigned* words = nullptr;
    unsigned blocks = 0;
    int first = 0, tail = 0, loop = 0;
    cudaGraphConditionalHandle rebin = 0, more = 0;
};
#ifdef __CUDACC__
// Passes left as a kernel of the step finds them (0: nothing to do); an
// advance moves something if step_moves.
__device__ __forceinline__ unsigned step_todo(const unsigned* words)
{
    const uint2 w = __ldcg(reinterpret_cast<const uint2*>(words + kStepStop));   // one load: the kernel waits for it
    return w.x ? 0u : w.y;
}
__device__ __forceinline__ bool step_moves(const StepGate& g, unsigned todo) { return todo >= (g.first ? 1u : 2u); }

__device__ __forceinline__ void step_set(const StepGate& g, unsigned flag, unsigned left)
{
    // (the value is set either way: a loop's body does not reset it)
    cudaGraphSetConditional(g.rebin, flag ? 1u : 0u);
    if (g.loop) cudaGraphSetConditional(g.more, left ? 1u : 0u);
}
// A step that does nothing (step_todo 0), by one thread of it, at a graph's end.
__device__ __forceinline__ void step_skip(const StepGate& g)
{
    if (g.tail) step_set(g, __ldcg(g.words + kStepStop), __ldcg(g.words + kStepTodo));
}
// One block of the step has finished (its thread 0): the last one closes the step.
__device__ __forceinline__ void step_end(const StepGate& g, unsigned todo, bool raised)
{
    unsigned long long* done = reinterpret_cast<unsigned long long*>(g.words + kStepDone);
    const unsigned long long old = atomicAdd(done, raised ? 0x100000001ull : 1ull);
    if ((unsigned)old != g.blocks - 1u) return;
    const unsigned flag = raised || (old >> 32) != 0ull || (g.first && __ldcg(g.words + kStepFlag)) ? 1u : 0u;
    const unsigned left = g.first ? todo : todo - 1u;
    *done = 0;
    *reinterpret_cast<uint2*>(g.words + kStepStop) = make_uint2(flag, left);
    if (g.tail) step_set(g, flag, left);
}
#endif
int launch_body_advance(xd_polygon_mass_info* pmi, unsigned nbodies, double dt, cudaStream_t s,
                        double* pose = nullptr, const StepGate& g = StepGate());
unsigned mesh_move_blocks(unsigned ntri);
int launch_update_polygon(const xd_polygon_mass_info* dpmi, const double* vlist, double* sphere,
                          xd_polygon_info* dpi, unsigned ntri, cudaStream_t s);
// The mesh update with the mixed form's moved check in one launch (see
// k_mesh_move): *flag raised when a vertex moved disp2 or more from ref; rec
// (nullable) receives the triangle records of the new pose.
struct TriRec;
int launch_mesh_move(xd_polygon_mass_info* dpmi, const double* pose, unsigned nbodies, const double* vlist,
                     double* sphere, xd_polygon_info* dpi,
                     unsigned ntri, const float* ref, const double wo[3], float disp2, unsigned* flag,
                     TriRec* rec, cudaStream_t s, const StepGate& g = StepGate());
// The mixed form's triangle records of a mesh as it stands.
int launch_tri_records(const xd_polygon_info* dpi, unsigned ntri, TriRec* rec, cudaStream_t s);
int reduction_d3(const double* in, unsigned n, double out[3], void* scratch, cudaStream_t s);
size_t reduction_scratch_bytes(unsigned n);
size_t pair_list_scratch_bytes(unsigned np);
int pair_list(const Params& P, const double* pos, const unsigned* sorted, const unsigned* cstart,
              const unsigned* cend, unsigned np, unsigned* counts, unsigned* pairs,
              unsigned long long cap, unsigned long long* total, void* scratch, cudaStream_t s);

}  // namespace xd
