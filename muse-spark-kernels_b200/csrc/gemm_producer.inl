// Role body of moe_gemm_kernel (included inside the kernel): weight producer, warp 0.
// One lane streams the two packed tiles of every K stage of every piece of this CTA into the
// shared-memory ring, one contiguous copy (layout.cuh) per stage that completes on the stage's mbarrier. With both
// phases in one launch the stream runs on from the last gate/up stage into the first down stage.
//
// The ring is the only look-ahead. Asking L2 for stages further ahead (cp.async.bulk.prefetch.L2 from
// this lane, 4 to 32 stages in front of the ring) was built and measured: every few-token point got
// slower (one token 46 -> 48 us at 8 stages, 64 tokens 262 -> 274 us), because the main loop does not
// wait for memory (with the weight copies left out altogether the steps take the same time) and each
// prefetch occupies the copy engine of the SM for as long as the copy it anticipates.
    if (lane == 0) {
      const uint64_t pol = p.evict_first ? policy_evict_first() : policy_evict_last();
      uint32_t it = 0;
      int tri = 0;
      bool ok = true;
      MSK_PHASES {
        MSK_PHASE_SETUP;
        while (ok && pieces.next(base, ks0, ks1)) {
          const UnitInfo ui = decode_unit(base, tile_start, pp.n_pairs, p.nloc, N);
          const uint8_t* wsrc = pp.w + static_cast<size_t>(ui.expert * pp.n_pairs + ui.pair) * nst_total * STAGE_W_BYTES;
          for (int ks = ks0; ks < ks1; ++ks, ++it) {
            const uint32_t slot = it % NST, par = (it / NST) & 1u;
#ifdef MSK_TRACE_DETAIL
            if (!mbar_test(&ctl.raw_empty[slot], par ^ 1u)) MSK_TRD(2, tri, 2);   // ring slot still being read
#endif
            if (!MSK_WAIT(&ctl.raw_empty[slot], par ^ 1u, abortw)) { ok = false; break; }
            uint8_t* dst = ring + slot * C::STAGE_BYTES;
            mbar_arrive_expect_tx(&ctl.raw_full[slot], STAGE_W_BYTES);
            bulk_g2s(dst, wsrc + static_cast<size_t>(ks) * STAGE_W_BYTES, STAGE_W_BYTES, &ctl.raw_full[slot], pol);
            if (it == 0) MSK_TR(TR_FIRST_BULK);
            MSK_TRD(2, tri, 1);
          }
        }
        if (!ok) break;
      }
      if (MODE == 0 && ok && p.ph[1].w != nullptr) {
        // This CTA's own weight stream has been issued. The down GEMM that follows is dealt the same way
        // over the same token tiles, so its CTA of this index will start on the stages named below: pull
        // the first ring-full of them into L2 now, while the pipeline here drains and the next kernel sets
        // up (the reference lets its last gate/up refills fetch the first down units,
        // muse_moe_w4a16/cuda/moe.cu:615-617, 2307-2318).
        const PhaseParams& nx = p.ph[1];
        const int nst2 = nx.K / KS;
        PieceIter pi = make_piece_iter(iter_mode, ctl.n_tiles * nx.n_pairs, nst2, static_cast<int>(blockIdx.x),
                                       static_cast<int>(n_ctas));
        int left = NST + 1, b2, k0, k1;
        while (left > 0 && pi.next(b2, k0, k1)) {
          const UnitInfo u2 = decode_unit(b2, tile_start, nx.n_pairs, p.nloc, N);
          const uint8_t* src = nx.w + (static_cast<size_t>(u2.expert * nx.n_pairs + u2.pair) * nst2 + k0) * STAGE_W_BYTES;
          const int take = min(left, k1 - k0);
          bulk_prefetch_l2(src, static_cast<uint32_t>(take) * STAGE_W_BYTES);
          left -= take;
        }
      }
    }
