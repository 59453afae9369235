// Role body of moe_gemm_kernel (included inside the kernel): MMA issuers, warps 1 and 3, one per
// tile of the pair (a single issuing warp, sharing its scheduler with four dequant warps, took
// ~29 cycles per MMA and became the limiter of the narrow-tile main loop).
// One A slot (128 K, 64 TMEM columns per tile) is consumed by eight K=16 MMAs per tile and
// handed back with a tcgen05.commit, so several dequant -> MMA -> release hand-offs are in
// flight at once. The accumulators of consecutive pieces alternate between NDBUF buffers.
// One thread of the warp walks the whole loop, waits included: electing a lane for every slot and meeting again behind it, beside
// the dequant warps that leave few issue slots, made an MMA 80 cycles where it needs 16 to 32 (256 tokens 325 -> 310 us a step in a
// row of them, 512 tokens 370 -> 360).
    constexpr uint32_t idesc = idesc_f16(FMT_F16, FMT_F16, 128, N);
    const int mg = warp == 1 ? 0 : 1;  // warp 1 issues for tile 0, warp 3 for tile 1
    uint32_t it = 0, unit_i = 0, sc = 0;
    uint32_t as = 0, apar = 0;  // A ring position and its phase parity
    int tri = 0;
    (void)tri;
    bool ok = true;
    if (elect_one())
    MSK_PHASES {
      MSK_PHASE_SETUP;
      for (; ok && pieces.next(base, ks0, ks1); ++unit_i) {
        const UnitInfo ui = decode_unit(base, tile_start, pp.n_pairs, p.nloc, N);
        const uint32_t db = unit_i % NDBUF, duse = unit_i / NDBUF;
        if (!MSK_WAIT(&ctl.d_empty[db], (duse & 1u) ^ 1u, abortw)) { ok = false; break; }
        tc_fence_after();
        if (mg == 0) MSK_TRD(1, tri, 3);
        const uint32_t d_tmem = tmem + db * (2 * N) + mg * N;
        // a ragged last token tile of an expert only pays for the columns it has (MMA N in steps of 16)
        const uint32_t idesc_u = N >= 64 ? idesc_f16(FMT_F16, FMT_F16, 128, static_cast<uint32_t>((ui.rows + 15) & ~15)) : idesc;
        const uint32_t bsub = ui.rows <= 16 ? 2048u : ui.rows <= 32 ? 4096u : 8192u;   // bytes between 64 K of the rows
        const uint32_t a_base = tmem + C::A_BASE + mg * C::A_GROUP_COLS;
        for (int ks = ks0; ks < ks1 && ok; ++ks, ++it) {
          const uint32_t slot = it % NST, par = (it / NST) & 1u;
#ifdef MSK_TRACE_DETAIL
          if (mg == 0 && !mbar_test(&ctl.b_full[slot], par)) MSK_TRD(1, tri, 4);   // B tile not there yet
#endif
          if (!MSK_WAIT(&ctl.b_full[slot], par, abortw)) { ok = false; break; }
          if (mg == 0) MSK_TRD(1, tri, 1);
          const uint32_t b_addr = smem_u32(ring + slot * C::STAGE_BYTES + 2 * TILE_BYTES);
#pragma unroll
          for (int sl = 0; sl < 2; ++sl, ++sc) {
#ifdef MSK_TRACE_DETAIL
            if (mg == 0 && !mbar_test(&ctl.a_full[mg][as], apar)) MSK_TRD(1, tri, 5);   // A slot not there yet
#endif
            if (!MSK_WAIT(&ctl.a_full[mg][as], apar, abortw)) { ok = false; break; }
            if (mg == 0) MSK_TRD(1, tri, 6);
            tc_fence_after();
            if (sc == 0 && mg == 0) MSK_TR(TR_FIRST_MMA);
            const uint32_t acc = (ks > ks0 || sl > 0) ? 1u : 0u;
            if (TMA_B) mma_slot_ts<2>(d_tmem, a_base + as * C::SLOT_COLS, smem_desc_kmajor_sw128(b_addr + sl * 2 * bsub), idesc_u, acc, bsub >> 4);
            else mma_slot_ts<16>(d_tmem, a_base + as * C::SLOT_COLS, smem_desc_kmajor_noswz(b_addr + sl * 2048, B_LBO, B_SBO), idesc_u, acc, 64u);
            tc_commit(&ctl.a_empty[mg][as]);
            if (++as == NSLOT) { as = 0; apar ^= 1u; }
          }
          if (!ok) break;
          tc_commit(&ctl.b_empty[slot]);
        }
        if (ok) tc_commit(&ctl.d_full[db]);
        if (mg == 0) MSK_TRD(1, tri, 2);
      }
      if (!ok) break;
    }
