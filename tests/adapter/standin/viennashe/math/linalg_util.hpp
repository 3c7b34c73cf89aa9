// Stand-in for the reference's sparse_matrix (viennashe/math/linalg_util.hpp:68-196): rows as ordered maps
// from column to value, which is what the adapter walks.
#ifndef VSHE_STANDIN_LINALG_UTIL_HPP
#define VSHE_STANDIN_LINALG_UTIL_HPP
#include <cstddef>
#include <map>
#include <vector>
namespace viennashe {
namespace math {
template <typename T>
class sparse_matrix {
  typedef std::map<std::size_t, T> row_type;
  std::vector<row_type> rows;

 public:
  typedef typename row_type::const_iterator const_iterator2;
  sparse_matrix(std::size_t n, std::size_t) : rows(n) {}
  std::size_t size1() const { return rows.size(); }
  std::size_t nnz() const {
    std::size_t count = 0;
    for (std::size_t i = 0; i < rows.size(); ++i) count += rows[i].size();
    return count;
  }
  T &operator()(std::size_t i, std::size_t j) { return rows[i][j]; }
  row_type const &row(std::size_t i) const { return rows[i]; }
};
}  // namespace math
}  // namespace viennashe
#endif
