// Factories of the operator classes, one translation unit per kind and number type.
#pragma once
#include <memory>
#include <vector>

#include "operator.hpp"

namespace sfem {

template <typename T>
std::unique_ptr<Operator> make_cg_operator(const Mesh& mesh, const OpConfig& cfg);
template <typename T>
std::unique_ptr<Operator> make_cg_local_operator(const Mesh& mesh, const CGDofs& dofs,
                                                 const std::vector<uint8_t>* identity, const OpConfig& cfg);
template <typename T>
std::unique_ptr<Operator> make_dg_operator(const Mesh& mesh, const OpConfig& cfg);
template <typename T>
std::unique_ptr<Batch> make_dg_batch(const std::vector<Operator*>& ops);

}  // namespace sfem
