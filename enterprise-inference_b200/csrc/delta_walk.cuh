// The body of the walk (delta.cu), which its kernel and the block kernel's short portions share as text: as a function in both the kernel's registers
// fell differently (64 decode rows 40 -> 45 us).  From its surroundings: NP, DELTA, CHAN, the arguments a, sequence s, head h,
// first value column jb, shared memory `stage`, DS_SYNC().
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int start = a.seq_start[s], n_rows = a.seq_start[s + 1] - start;
  if (n_rows <= 0) return;
  const bool fresh = a.positions[start] == 0;
  const int g = h / (a.heads / a.kv_heads), dim = a.dim, vd = a.vd;
  const int j0 = jb + warp * 4;   // the warp's first value column
  float* S_st = a.state + (int64_t)a.seq_slots[s] * a.slot_stride + ((int64_t)h * vd + j0) * dim;
  const int64_t qk = (int64_t)a.kv_heads * dim, hv = (int64_t)a.heads * vd;
  const float* qsrc = a.qn + (int64_t)start * qk + (int64_t)g * dim;
  const float* ksrc = a.kn + (int64_t)start * qk + (int64_t)g * dim;
  const float* gsrc = a.decay + (int64_t)start * a.g_row + (int64_t)h * a.g_head;
  const float* vsrc = a.vn + (int64_t)start * hv + (int64_t)h * vd + jb;
  const float* bsrc = a.beta + (int64_t)start * a.heads + h;
  uint64_t S[4][NP];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int d = ds_chan<NP>(lane, i);
      const float* p = S_st + (int64_t)c * dim + d;
      S[c][i] = 0;
      if (!fresh && j0 + c < vd && d < dim) S[c][i] = a.vec ? *reinterpret_cast<const uint64_t*>(p) : f2::pack(p[0], d + 1 < dim ? p[1] : 0.f);
    }
  if (n_rows == 1) {
    // a decode row: nothing to stage; the row's inputs are fetched beside the state
    const float b = bsrc[0], gs = CHAN ? 0.f : gsrc[0];
    uint64_t k[NP], q[NP];
    float d4[4] = {0.f, 0.f, 0.f, 0.f}, o4[4];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int d = ds_chan<NP>(lane, i);
      auto pair = [&](const float* p, int64_t st) { return f2::pack(d < dim ? p[d * st] : 0.f, d + 1 < dim ? p[(d + 1) * st] : 0.f); };
      k[i] = pair(ksrc, 1);
      q[i] = pair(qsrc, 1);
      const uint64_t gg = CHAN ? pair(gsrc, a.g_chan) : f2::both(gs);
#pragma unroll
      for (int c = 0; c < 4; ++c) S[c][i] = f2::mul(S[c][i], gg);
    }
    if (DELTA) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint64_t acc = f2::mul(S[c][0], k[0]);
#pragma unroll
        for (int i = 1; i < NP; ++i) acc = f2::fma(S[c][i], k[i], acc);
        d4[c] = f2::sum(acc);
      }
      ds_reduce<4>(d4, lane);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const uint64_t u = f2::both(b * ((j0 + c < vd ? vsrc[warp * 4 + c] : 0.f) - d4[c]));
      uint64_t acc = 0;
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        S[c][i] = f2::fma(k[i], u, S[c][i]);
        acc = f2::fma(S[c][i], q[i], acc);
      }
      o4[c] = f2::sum(acc);
    }
    ds_reduce<4>(o4, lane);
    const float mine = lane == 0 ? o4[0] : lane == 1 ? o4[1] : lane == 2 ? o4[2] : o4[3];
    if (lane < 4 && j0 + lane < vd) a.out[(int64_t)start * hv + (int64_t)h * vd + j0 + lane] = mine;
  } else {
    float* kq = stage + 2 * BUF;                                          // [kDsStage] per pair of rows: k1 g2 k2, k1 . q1
    float* part = kq + kDsStage + warp * kDsFlush * kDsPartRow;
    if (dim < ROW) {   // zeros beyond dim, once: the copies leave them alone
      for (int e = tid; e < 2 * BUF; e += kDsThreads) stage[e] = 0.f;
      DS_SYNC();
    }
    auto fetch = [&](int b0, float* buf) {
      const int nb = min(kDsStage, n_rows - b0);
      float* sq = buf;
      float* sk = sq + kDsStage * ROW;
      float* sg = sk + kDsStage * ROW;
      float* sv = sq + kDsStage * (CHAN ? 3 : 2) * ROW;
      float* sb = sv + kDsStage * kDsCols;
      if (a.vec) {
#pragma unroll
        for (int e0 = 0; e0 < kDsStage * ROW / 4; e0 += kDsThreads) {
          const int e = e0 + tid, r = e / (ROW / 4), c = (e % (ROW / 4)) * 4;
          if (r < nb && c < dim) {
            f2::cp16(sq + r * ROW + c, qsrc + (b0 + r) * qk + c);
            f2::cp16(sk + r * ROW + c, ksrc + (b0 + r) * qk + c);
            if (CHAN) f2::cp16(sg + r * ROW + c, gsrc + (b0 + r) * a.g_row + c);
          }
        }
      } else {
        for (int e = tid; e < kDsStage * ROW; e += kDsThreads) {
          const int r = e / ROW, c = e % ROW;
          if (r < nb && c < dim) {
            f2::cp4(sq + r * ROW + c, qsrc + (b0 + r) * qk + c);
            f2::cp4(sk + r * ROW + c, ksrc + (b0 + r) * qk + c);
            if (CHAN) f2::cp4(sg + r * ROW + c, gsrc + (b0 + r) * a.g_row + (int64_t)c * a.g_chan);
          }
        }
      }
#pragma unroll
      for (int e0 = 0; e0 < kDsStage * kDsCols; e0 += kDsThreads) {
        const int e = e0 + tid, r = e / kDsCols, c = e % kDsCols;
        if (r < nb && jb + c < vd) f2::cp4(sv + e, vsrc + (b0 + r) * hv + c);
      }
      if (tid < nb) {
        f2::cp4(sb + tid, bsrc + (int64_t)(b0 + tid) * a.heads);
        if (!CHAN) f2::cp4(sb + kDsStage + tid, gsrc + (b0 + tid) * a.g_row);
      }
    };
    fetch(0, stage);
    for (int b0 = 0, it = 0; b0 < n_rows; b0 += kDsStage, ++it) {
      const int nb = min(kDsStage, n_rows - b0);
      const float* sq = stage + (it & 1) * BUF;
      const float* sk = sq + kDsStage * ROW;
      const float* sg = sk + kDsStage * ROW;
      const float* sv = sq + kDsStage * (CHAN ? 3 : 2) * ROW + warp * 4;
      const float* sb = sv - warp * 4 + kDsStage * kDsCols;
      f2::cp_wait_all();
      DS_SYNC();   // the stage has landed for everybody, and the one before has been consumed
      if (b0 + kDsStage < n_rows) fetch(b0 + kDsStage, stage + ((it + 1) & 1) * BUF);
      if (DELTA) {
        for (int r = 2 * warp; r + 1 < nb; r += 2 * kDsWarps) {
          float xy[2] = {0.f, 0.f};
#pragma unroll
          for (int d = 0; d < ROW; d += 32) {
            const float k1 = sk[r * ROW + d + lane], k2 = sk[(r + 1) * ROW + d + lane];
            xy[0] = fmaf(CHAN ? k1 * sg[(r + 1) * ROW + d + lane] : k1, k2, xy[0]);
            xy[1] = fmaf(k1, sq[r * ROW + d + lane], xy[1]);
          }
          ds_reduce<2>(xy, lane);
          if (lane == 0) *reinterpret_cast<float2*>(kq + r) = make_float2(CHAN ? xy[0] : xy[0] * sb[kDsStage + r + 1], xy[1]);
        }
        DS_SYNC();
      }
      auto decay_row = [&](const uint64_t (&gg)[NP]) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < NP; ++i) S[c][i] = f2::mul(S[c][i], gg[i]);
      };
      auto decays = [&](int r, uint64_t (&gg)[NP]) {
        if (CHAN) {
          ds_pairs<NP>(sg + r * ROW, lane, gg);
        } else {
          const uint64_t x = f2::both(sb[kDsStage + r]);
#pragma unroll
          for (int i = 0; i < NP; ++i) gg[i] = x;
        }
      };
      auto dots = [&](const uint64_t (&x)[NP], float* o) {   // the lane's part of S^T x for the four columns
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint64_t acc = f2::mul(S[c][0], x[0]);
#pragma unroll
          for (int i = 1; i < NP; ++i) acc = f2::fma(S[c][i], x[i], acc);
          o[c] = f2::sum(acc);
        }
      };
      int r = 0;
      for (int f0 = 0; f0 < nb; f0 += kDsFlush) {
      const int f1 = min(f0 + kDsFlush, nb);
      if (DELTA) {
        for (; r + 1 < f1; r += 2) {
          uint64_t g1[NP], g2[NP], k1[NP], k2[NP], q1[NP], q2[NP];
          decays(r, g1);
          ds_pairs<NP>(sk + r * ROW, lane, k1);
          decays(r + 1, g2);
          ds_pairs<NP>(sk + (r + 1) * ROW, lane, k2);
          ds_pairs<NP>(sq + r * ROW, lane, q1);
          ds_pairs<NP>(sq + (r + 1) * ROW, lane, q2);
          const float4 v1 = *reinterpret_cast<const float4*>(sv + r * kDsCols), v2 = *reinterpret_cast<const float4*>(sv + (r + 1) * kDsCols);
          const float2 bb = *reinterpret_cast<const float2*>(sb + r), kk = *reinterpret_cast<const float2*>(kq + r);
          float d[8], o1[4], o2[4];
          decay_row(g1);
          dots(k1, d);
          dots(q1, o1);
          decay_row(g2);
          dots(k2, d + 4);
          ds_reduce<8>(d, lane);
          const float va[4] = {v1.x, v1.y, v1.z, v1.w}, vb[4] = {v2.x, v2.y, v2.z, v2.w};
          uint64_t kg[NP];
#pragma unroll
          for (int i = 0; i < NP; ++i) kg[i] = f2::mul(k1[i], g2[i]);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float u1 = bb.x * (va[c] - d[c]), u2 = bb.y * (vb[c] - fmaf(kk.x, u1, d[4 + c]));
            if (lane == 0) o1[c] = fmaf(kk.y, u1, o1[c]);
            const uint64_t w1 = f2::both(u1), w2 = f2::both(u2);
#pragma unroll
            for (int i = 0; i < NP; ++i) S[c][i] = f2::fma(k2[i], w2, f2::fma(kg[i], w1, S[c][i]));
          }
          dots(q2, o2);
          *reinterpret_cast<float4*>(part + (r - f0) * kDsPartRow + 4 * lane) = make_float4(o1[0], o1[1], o1[2], o1[3]);
          *reinterpret_cast<float4*>(part + (r + 1 - f0) * kDsPartRow + 4 * lane) = make_float4(o2[0], o2[1], o2[2], o2[3]);
        }
      }
#pragma unroll 2
      for (; r < f1; ++r) {
        uint64_t gg[NP], k[NP], q[NP];
        decays(r, gg);
        ds_pairs<NP>(sk + r * ROW, lane, k);
        ds_pairs<NP>(sq + r * ROW, lane, q);
        const float4 v4 = *reinterpret_cast<const float4*>(sv + r * kDsCols);
        const float va[4] = {v4.x, v4.y, v4.z, v4.w}, b = sb[r];
        float d[4] = {0.f, 0.f, 0.f, 0.f}, o[4];
        decay_row(gg);
        if (DELTA) {
          dots(k, d);
          ds_reduce<4>(d, lane);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint64_t u = f2::both(b * (va[c] - d[c]));
#pragma unroll
          for (int i = 0; i < NP; ++i) S[c][i] = f2::fma(k[i], u, S[c][i]);
        }
        dots(q, o);
        *reinterpret_cast<float4*>(part + (r - f0) * kDsPartRow + 4 * lane) = make_float4(o[0], o[1], o[2], o[3]);
      }
      __syncwarp();
      {   // four lanes a row, eight lanes' sums each
        const int rr = lane >> 2, quarter = lane & 3;
        const float* src = part + rr * kDsPartRow + quarter * 32;
        uint64_t x = 0, y = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(src + 4 * (i ^ quarter));   // (the four lanes' banks apart)
          x = f2::add(x, t.x);
          y = f2::add(y, t.y);
        }
        float o[4] = {f2::lo(x), f2::hi(x), f2::lo(y), f2::hi(y)};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          o[c] += __shfl_xor_sync(0xffffffffu, o[c], 1);
          o[c] += __shfl_xor_sync(0xffffffffu, o[c], 2);
        }
        const float mine = quarter == 0 ? o[0] : quarter == 1 ? o[1] : quarter == 2 ? o[2] : o[3];
        if (f0 + rr < f1 && j0 + quarter < vd) a.out[(int64_t)(start + b0 + f0 + rr) * hv + (int64_t)h * vd + j0 + quarter] = mine;
      }
      __syncwarp();
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int d = ds_chan<NP>(lane, i);
      float* p = S_st + (int64_t)c * dim + d;
      if (j0 + c >= vd || d >= dim) continue;
      if (a.vec) {
        *reinterpret_cast<uint64_t*>(p) = S[c][i];
      } else {
        p[0] = f2::lo(S[c][i]);
        if (d + 1 < dim) p[1] = f2::hi(S[c][i]);
      }
    }
