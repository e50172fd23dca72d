// The coupled time loop on the host side: map, fused step and DEM sub-steps of
// many steps issued from one call.  A step of a small lattice takes the GPU
// less time than a Python driver needs to issue it (one settling sphere: 45 us
// of kernels, 56 us a step).
#include "common.cuh"

using namespace lbdem;

extern "C" int lbdem_psc_run(const lbdem_lattice *L, lbdem_psc *P, const lbdem_grains *G, lbdem_dem *D,
                             void *dem_work, int32_t nsteps, int32_t nsub, int32_t src, int32_t gather,
                             int32_t moving, int32_t *done, int32_t *launches, void *stream) {
    if (!L || !P || !G || !D || !done || !launches || nsteps < 0 || src < 0 || src > 1 || G->n <= 0) {
        set_error("psc_run: bad arguments");
        return LBDEM_ERR_ARG;
    }
    if (P->eps || P->disp_limit > 0.0 || L->stress) {
        set_error("psc_run: the exact map only, without pipelined stepping and fused stress output");
        return LBDEM_ERR_UNSUPPORTED;
    }
    cudaStream_t st = (cudaStream_t)stream;
    *done = *launches = 0;
    const int boundary = (L->bnd_na > 0) + (L->bnd_nb > 0);
    for (int k = 0; k < nsteps; ++k) {
        // Where particles move, the keys of all steps but the last are cleared by
        // the step that reads them: the next map then starts on clear keys and
        // is one launch.  The last step's stay for lbdem_psc_decode.
        const bool clear_keys = moving && boundary == 0 && k + 1 < nsteps;
        *launches += 1 + (P->have_prev != 0);
        int rc = lbdem_psc_map(L, P, G, stream);
        if (rc) return rc;
        P->map_reuse = 1;   // (no cell type changes within the call)
        if (P->hydro_out &&
            cudaMemsetAsync(P->hydro_out, 0, sizeof(float) * 3 * (size_t)L->nx * L->ny * L->nz, st) != cudaSuccess)
            return check_launch("psc_run");
        rc = psc_step(L, P, G, src, gather, clear_keys, st);
        if (rc) return rc;
        *launches += 1 + boundary;
        if (clear_keys) P->have_prev = 0;
        src = 1 - src;
        gather = 1;
        *done = k + 1;
        if (nsub > 0) {
            rc = lbdem_dem_substeps_flow(D, nsub, dem_work, stream);
            if (rc) return rc;
            *launches += lbdem_dem_launches_last();
        }
    }
    return LBDEM_OK;
}
