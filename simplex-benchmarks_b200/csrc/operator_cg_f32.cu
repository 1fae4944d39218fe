#include "operator_cg.cuh"

namespace sfem {
template std::unique_ptr<Operator> make_cg_operator<float>(const Mesh&, const OpConfig&);
template std::unique_ptr<Operator> make_cg_local_operator<float>(const Mesh&, const CGDofs&, const std::vector<uint8_t>*,
                                                           const OpConfig&);
}  // namespace sfem
