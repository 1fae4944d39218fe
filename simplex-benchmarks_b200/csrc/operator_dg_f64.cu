#include "operator_dg.cuh"

namespace sfem {
template std::unique_ptr<Operator> make_dg_operator<double>(const Mesh&, const OpConfig&);
template std::unique_ptr<Batch> make_dg_batch<double>(const std::vector<Operator*>&);
}  // namespace sfem
