// zzx.cuh — the ZZ + X observable and its tiled kernels (zzx.cu), shared with adjoint.cu.
#pragma once

#include "internal.cuh"

namespace qgpu {

constexpr int MAX_HAM_QUBITS = 40;

// sum_i a[i] Z_i Z_{(i+1) mod n} + b[i] X_i on wires i (wire i = index bit n-1-i)
struct Ham {
    int n;
    double a[MAX_HAM_QUBITS];
    double b[MAX_HAM_QUBITS];
};

// Smallest register of the tiled form: below it the plain kernel's blocks fill more SMs than the
// tiles of 2^11 amplitudes (energy call, complex128: 16 qubits 34 us plain against 38 us tiled, 18
// qubits 71 against 48 us).
constexpr int ZZX_MIN_QUBITS = 17;

// Whether the tiled kernels take this register and observable: complex64 or the fast mode, and
// coefficients whose largest lies within 2^-40 .. 2^40 (the float pairs' exponent range).
bool zzx_tiled_supported(const qgpu_handle* h, const Ham& H);

// *energy = Re <psi|H|psi>. With lam: phi = psi and lam = H psi as well, in the layout of the
// adjoint sweep (complex128: resident float pairs). *ok is false when <psi|psi> is not a number
// within 2^-40 .. 2^40: the results may then have left the float range and the caller runs the
// plain kernel. Synchronises.
int zzx_tiled(qgpu_handle* h, const void* psi, void* phi, void* lam, const Ham& H, double* energy,
              bool* ok);

}  // namespace qgpu
