// Factored gradients of isoparametric P2 tetrahedra, and the element kernels that use them.
//
// Every P2 basis gradient at a point is a combination of the four barycentric gradients
// G_k = grad(lambda_k) with coefficients that depend on the point of the rule only
// (vertices 0..3, then the edges 01, 12, 02, 13, 23, 03):
//     vertex i      (4 lambda_i - 1) G_i
//     edge (a, b)   4 (lambda_b G_a + lambda_a G_b)           G_0 = -(G_1 + G_2 + G_3)
// so nine doubles per point (G_1, G_2, G_3; they vary inside a curved element) and one small
// table carry what the 30 gradients of d_dphi do.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "mesh.h"

namespace sg {

// Largest rule of the factored kernels (the reference's P2 rule has 11 points).
constexpr int P2T_MAXQ = 16;

// Barycentric coordinates of the rule's points, a kernel parameter (constant bank).
struct P2TetRule {
    double lam[P2T_MAXQ][4];
};

// Fills m->d_gxi and m->rule when the mesh's gradients are those of isoparametric P2
// tetrahedra in the numbering above, to within a few roundings; leaves d_gxi null otherwise
// (every kernel then reads d_dphi).
int p2tet_factor(sg_mesh *m, const double *D1, const double *D2, const double *D3);

// The reference's rule, for which the factored kernels are compiled.
constexpr int P2T_REF_RULE = 11;

// The element's 55 upper node blocks (9 values each, element-major) from DS into Ke, for
// factored meshes with the reference's rule.
int p2tet_element_blocks(const sg_mesh *m, const double *DS, double *Ke, cudaStream_t st);

}  // namespace sg
