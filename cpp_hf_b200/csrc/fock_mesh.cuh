// Internal interface of the fused Fock build of many bands with a scalar V (fock_mesh.cu).
#pragma once

#include "common.cuh"

namespace cpphf {

struct MeshOut {
    const double2 *h, *P, *refP;  // refP may be null
    const double* w;
    const double* hd;   // may be null (no Hartree)
    const double2* SC;  // may be null (no contact terms)
    double2* Sigma;     // may be null
    double2* F;
    double2* Hdense;    // may be null
    double* energy;     // may be null
    double* part;       // kFockMaxPartials
    unsigned* counter;
};

// Hermitian channel packing with a scalar V, complex128, no superlattice terms, and a
// shape that pays (hcp_tiled)
bool fock_mesh_eligible(const cpphf_kernel* K);
// bytes of T (0 when not eligible)
size_t fock_mesh_bytes(const cpphf_kernel* K);
int build_fock_mesh(const cpphf_kernel* K, const MeshOut& o, void* T, cudaStream_t st);

}  // namespace cpphf
