// sweep.h — gradients of circuits whose parameters sit in uncontrolled
// 1-qubit gates (sweep.cu), for one parameter vector or many.
#pragma once

#include <cstddef>
#include <vector>

#include "yao_internal.h"

namespace yao {

struct SweepPlan;
// The plan of a circuit on n qubits, or null when it does not apply: every
// parametric gate is an uncontrolled 1-qubit gate, and the others are unitary
// 1-qubit gates, (controlled) X, SWAP and sign gates such as CZ.
SweepPlan* sweep_plan_new(const Circuit* c, uint32_t n);
void sweep_plan_free(SweepPlan* p);

// The reverse sweep of one parameter vector: psi the forward state, lam = H
// psi (both are consumed).  grad receives 2 Re <lam | G psi> per parameter.
// Synchronises at the end; a set error word of the work queued before is
// reported.
int sweep_reverse(Ctx* ctx, const SweepPlan* p, void* psi, void* lam, const double* params, double* grad);
// Energies Re <psi|H|psi> and gradients of nsets parameter vectors (row-major
// nsets x parameters) from psi0.
int sweep_batch(Ctx* ctx, const SweepPlan* p, const std::vector<MonoTerm>& terms, const double* params, size_t nsets,
                const Reg* psi0, double* values, double* grads);

}  // namespace yao
