// Stand-in for the reference's viennashe/log/log.hpp: warnings go to an output stream.
#ifndef VSHE_STANDIN_LOG_HPP
#define VSHE_STANDIN_LOG_HPP
#include <iostream>
namespace viennashe {
namespace log {
inline std::ostream &warning() { return std::cerr; }
}  // namespace log
}  // namespace viennashe
#endif
