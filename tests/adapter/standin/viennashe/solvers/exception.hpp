// Stand-in for the reference's viennashe/solvers/exception.hpp.
#ifndef VSHE_STANDIN_SOLVERS_EXCEPTION_HPP
#define VSHE_STANDIN_SOLVERS_EXCEPTION_HPP
#include <stdexcept>
namespace viennashe {
namespace solvers {
struct invalid_linear_solver_exception : std::runtime_error {
  invalid_linear_solver_exception() : std::runtime_error("the solver is not available in this build") {}
};
}  // namespace solvers
}  // namespace viennashe
#endif
