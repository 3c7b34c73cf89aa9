// Stand-in for the reference's linear_solver_exception (viennashe/util/exception.hpp:38).
#ifndef VSHE_STANDIN_UTIL_EXCEPTION_HPP
#define VSHE_STANDIN_UTIL_EXCEPTION_HPP
#include <stdexcept>
#include <string>
namespace viennashe {
namespace util {
struct linear_solver_exception : std::runtime_error {
  explicit linear_solver_exception(std::string const &what) : std::runtime_error(what) {}
};
}  // namespace util
}  // namespace viennashe
#endif
