// k_terms.cu -- item-kernel instantiation of the indicator terms on 168 registers: in a unit
// of its own, since the functions that the kernels of a unit share are compiled for the
// smallest register budget among them (see gbs_items.cuh).
#include "gbs_items.cuh"

namespace gbsb {
#define GBSB_LIST_TERMS(X) X(kBrTerms)
GBSB_DEFINE_GROUP(terms, GBSB_LIST_TERMS)
}  // namespace gbsb
