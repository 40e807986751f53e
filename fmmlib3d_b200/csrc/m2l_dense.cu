// Dense M2L operators of the mixed form, one per translation offset (p <= 16).
//
// For a list-2 offset D (source box minus target box, in box units) the
// rotate-shift-rotate M2L of FMMLIB3D (l3dmplocquad2_trunc0,
// src/l3dtrans.f:1260-1387, truncated to nterms_trunc = pt) is a fixed
// linear map T_D from the (pt+1)^2 source coefficients to the (pt+1)^2
// target coefficients; with box-scaled coefficients it does not depend on
// the level.  k_build_m2l_ops composes T_D column by column on the GPU from
// the same rotation matrices and z-shift coefficients as the structured
// kernel:  T_D[(j,m)][(n,mc)] = e^{-i m phi} sum_k D^j[m][k] Z(j,k,n) D^n[mc][k] e^{i mc phi},
// Z(j,k,n) = (-1)^(j+k) sqrt(C(n+j,n-k) C(n+j,n+k)) / rt^(n+j+1).
// The FP32 kernels (mixed.cu, tc_m2l.cu) multiply by their roundings.
#include "lap_kernels.cuh"
#include "m2l_dense.cuh"

namespace fmm {

__global__ void k_build_m2l_ops(int p, const M2LOp *ops, const double *rot, const double *dc, int lddc,
                                double2 *T)
{
    const M2LOp op = ops[blockIdx.x];  // one unique offset per block row
    const int pt = op.pt, R = (pt + 1) * (pt + 1);
    const int col = blockIdx.y;
    if (col >= R) return;
    int nc = 0;
    while ((nc + 1) * (nc + 1) <= col) nc++;
    const int mc = col - nc * nc - nc;
    const size_t csz = rot_class_size(p);
    const double *Rm = rot + csz * op.cls;
    const double *Dn = Rm + (size_t)nc * (4 * nc * nc - 1) / 3 + (size_t)(mc + nc) * (2 * nc + 1);  // row mc
    // e^{i mc phi}
    double2 e1 = cmk(op.ex, op.ey), em = cmk(1, 0);
    for (int i = 0; i < (mc < 0 ? -mc : mc); i++) em = cmul(em, e1);
    if (mc < 0) em = cconj(em);
    for (int row = threadIdx.x; row < R; row += blockDim.x) {
        int j = 0;
        while ((j + 1) * (j + 1) <= row) j++;
        int m = row - j * j - j;
        const double *Dj = Rm + (size_t)j * (4 * j * j - 1) / 3 + (size_t)(m + j) * (2 * j + 1);
        int kmax = j < nc ? j : nc;
        double s = 0;
        double ir = 1.0 / op.rt, pw = 1;
        for (int i = 0; i < nc + j + 1; i++) pw *= ir;
        for (int k = -kmax; k <= kmax; k++) {
            double z = (((j + k) & 1) ? -1.0 : 1.0) * pw * dc[(nc + j) * lddc + (nc - k)] * dc[(nc + j) * lddc + (nc + k)];
            s += Dj[k + j] * z * Dn[k + nc];
        }
        // times e^{i mc phi} e^{-i m phi}
        double2 ph = em;
        double2 en = cmk(1, 0);
        for (int i = 0; i < (m < 0 ? -m : m); i++) en = cmul(en, e1);
        ph = m >= 0 ? cmulc(ph, en) : cmul(ph, en);
        T[op.toff + (size_t)col * R + row] = cscal(s, ph);  // column-major
    }
}

void build_m2l_ops(int p, int nops, const M2LOp *d_ops, const double *rot, const double *dc, int lddc,
                   double2 *T, cudaStream_t s, Status &st)
{
    if (!st.ok() || nops == 0) return;
    dim3 g(nops, (p + 1) * (p + 1));
    k_build_m2l_ops<<<g, 128, 0, s>>>(p, d_ops, rot, dc, lddc, T); FMM_COUNT_LAUNCH();
    FMM_LAUNCH_CHECK(st);
}

}  // namespace fmm
