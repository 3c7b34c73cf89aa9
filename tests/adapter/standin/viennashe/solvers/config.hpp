// Stand-in for the reference's linear_solver_config (viennashe/solvers/config.hpp:56-232): the solver's name
// and the values the adapter reads.
#ifndef VSHE_STANDIN_CONFIG_HPP
#define VSHE_STANDIN_CONFIG_HPP
#include <cstddef>
#include <string>
#include <utility>
#include <vector>
namespace viennashe {
namespace solvers {
class linear_solver_config {
 public:
  enum { other_solver, gpu_parallel_linear_solver };
  typedef std::vector<std::pair<std::size_t, std::size_t> > block_preconditioner_boundaries_container;

  void set(std::string const &name) { id_ = name == "gpu_parallel_linear_solver" ? gpu_parallel_linear_solver : other_solver; }
  long id() const { return id_; }
  double tolerance() const { return tolerance_; }
  void tolerance(double v) { tolerance_ = v; }
  std::size_t max_iters() const { return max_iters_; }
  void max_iters(std::size_t v) { max_iters_ = v; }
  std::size_t ilut_entries() const { return 60; }
  double ilut_drop_tolerance() const { return 1e-4; }
  block_preconditioner_boundaries_container &block_preconditioner_boundaries() { return blocks_; }
  block_preconditioner_boundaries_container const &block_preconditioner_boundaries() const { return blocks_; }

 private:
  long id_ = other_solver;
  double tolerance_ = 1e-10;
  std::size_t max_iters_ = 1000;
  block_preconditioner_boundaries_container blocks_;
};
}  // namespace solvers
}  // namespace viennashe
#endif
