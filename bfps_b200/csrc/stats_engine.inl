// Engine<T, N>::stats — field::compute_stats (bfps/cpp/field.cpp:984-1040)
// for one complex 3-vector field in the state layout: co-spectrum, then the
// unnormalised C2R into scratch and the real-space moments and histograms.
// The scratch is v2: between steps nothing in v1 and v2 is needed.  A step writes
// and reads them inside the region that the passes keep (passes.cuh, modes
// outside kM) and nowhere else, so what is left here stays in v2 outside it: a
// pass that reads v1 or v2 has to leave the same modes out (PRUNE_IN).
// Included by bfps_b200.cu after the Engine definition.

template <typename T, int N>
int Engine<T, N>::stats(bfg_ctx* c, int cfield, double max_est, int nbins, double* spec,
                        double* mom, int64_t* hist) {
    const size_t spec_n = (size_t)c->nshells * 9;
    // spectrum: SPEC_BLOCKS partials of spec_n doubles, then the result
    int spec_warps = SPEC_WARPS_MAX;
    const size_t spec_q = (size_t)c->nshells * SPEC_NQ;  // values per warp
    while (spec_warps > 1 && (size_t)spec_warps * spec_q * 8 > (size_t)c->smem_optin) --spec_warps;
    if (spec_n * 8 > (size_t)c->smem_optin)
        return fail(c, BFG_EUNSUP, "%d shells do not fit the spectrum kernel's shared memory",
                    c->nshells);
    const size_t need = spec_n * 8 + (size_t)SPEC_BLOCKS * spec_n * 8 +
                        (size_t)STATS_BLOCKS * NQ * 8 + NQ * 8 + (size_t)nbins * 4 * 8;
    if (c->stats_ws_bytes < need) {
        if (c->stats_ws) cudaFree(c->stats_ws);
        c->stats_ws = nullptr;
        c->stats_ws_bytes = 0;
        CU(cudaMalloc(&c->stats_ws, need));
        c->stats_ws_bytes = need;
    }
    double* d_spec = (double*)c->stats_ws;
    double* d_spart = d_spec + spec_n;
    double* d_part = d_spart + (size_t)SPEC_BLOCKS * spec_n;
    double* d_mom = d_part + (size_t)STATS_BLOCKS * NQ;
    unsigned long long* d_hist = (unsigned long long*)(d_mom + NQ);
    CU(cudaMemsetAsync(d_hist, 0, (size_t)nbins * 4 * 8, c->stream));
    const KParams kp = kparams(c, 0.0);
    Prof pr0(c, K_STATS);
    const void* cptr = cfield == B_W0 ? c->w0 : (cfield == B_V1 ? c->v1 : c->wa);
    const size_t spec_smem = (size_t)spec_warps * spec_q * 8;
    CU(ensure_smem(spectrum_kernel<T, N>, spec_smem, c->device));
    spectrum_kernel<T, N><<<SPEC_BLOCKS, spec_warps * 32, spec_smem, c->stream>>>(
        kp, (const C*)cptr, c->nshells, c->dk, d_spart);
    int rc = after_launch(c, "spectrum");
    if (rc) return rc;
    spectrum_final<<<(unsigned)((spec_q + 31) / 32), 32 * SPEC_FINAL_GROUPS, 0, c->stream>>>(
        d_spart, SPEC_BLOCKS, (int)spec_q, d_spec);
    if ((rc = after_launch(c, "spectrum_final"))) return rc;
    // real-space field into v2 (as [z][y][x][3] reals)
    // (the velocity is zero outside kM, the state where it is known to be)
    const int prune = cfield == B_WA || (cfield == B_W0 && !c->w0_full) ? PRUNE_IN : 0;
    if ((rc = col<CM_IZ_PLAIN>(c, self(c), 1, pruned(roles(cfield, B_NONE, B_WB, B_NONE), prune))))
        return rc;
    if ((rc = rspace(c, B_WB, B_V2, prune))) return rc;
    const double me3 = max_est * std::sqrt(3.0);
    const size_t npts = (size_t)N * N * N;
    CU(ensure_smem(moments_kernel<T>, (size_t)nbins * 4 * 4, c->device));
    Prof pr1(c, K_STATS);
    const int mom_blocks = stats_blocks(npts);
    moments_kernel<T><<<mom_blocks, STATS_THREADS, (size_t)nbins * 4 * 4, c->stream>>>(
        (const T*)c->v2, N, N, npts, hist_range(max_est, me3, nbins), d_part, d_hist);
    if ((rc = after_launch(c, "moments"))) return rc;
    moments_final<<<NQ, MOM_FINAL_THREADS, 0, c->stream>>>(d_part, mom_blocks, 1.0 / (double)npts, d_mom);
    if ((rc = after_launch(c, "moments_final"))) return rc;
    if (spec) CU(cudaMemcpyAsync(spec, d_spec, spec_n * 8, cudaMemcpyDeviceToHost, c->stream));
    if (mom) CU(cudaMemcpyAsync(mom, d_mom, NQ * 8, cudaMemcpyDeviceToHost, c->stream));
    if (hist) CU(cudaMemcpyAsync(hist, d_hist, (size_t)nbins * 4 * 8, cudaMemcpyDeviceToHost, c->stream));
    return finish_call(c);
}
