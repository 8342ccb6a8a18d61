// resident_f64.cu -- the on-chip CG in FP64 (resident.cuh): QED2D_PREC_F64.
#include "resident.cuh"

namespace qed2d {

int res_f64_clusters(const ResPlan& p) {
    return p.K == 1 ? res_clusters_k<double, 1>(p) : res_clusters_k<double, 2>(p);
}

int res_f64_launch(const ResP& P, const ResPlan& plan, cudaStream_t stream) {
    switch (plan.K * 2 + plan.cl) {
        case 2: return res_launch_k<double, 1, false>(P, plan, stream);
        case 3: return res_launch_k<double, 1, true>(P, plan, stream);
        case 4: return res_launch_k<double, 2, false>(P, plan, stream);
        default: return res_launch_k<double, 2, true>(P, plan, stream);
    }
}

}  // namespace qed2d
