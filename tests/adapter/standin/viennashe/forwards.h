// Stand-in for the reference's viennashe/forwards.h: the solver tags that the drop-in adapter overloads on
// (viennashe/forwards.h:200-217).  The stand-ins declare what the adapter and its harness use, under the
// reference's names, so that the harness builds where the reference's headers are absent.
#ifndef VSHE_STANDIN_FORWARDS_H
#define VSHE_STANDIN_FORWARDS_H
namespace viennashe {
namespace solvers {
struct gpu_parallel_linear_solver_tag {};
struct petsc_amgx_solver_tag {};
}  // namespace solvers
}  // namespace viennashe
#endif
