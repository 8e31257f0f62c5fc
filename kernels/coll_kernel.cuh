// The generic collective kernel: push -> handshake -> local consume, chunked
// through the double-buffered staging area.
//
// Every rank's staging half is divided into p slots of `cap_b` bytes, one per
// source rank.  In the publish step a rank reads its contribution once from the
// user's send buffer and STORES it into slot [me] of the destination rank's
// staging half over NVLink (remote stores are posted and do not stall the
// issuing threads the way remote loads do; measured on 8 GPUs, pulling with
// loads reached a third of the pushed bandwidth).  After the epoch handshake a
// rank finds everything it needs in its own memory and reduces / copies it to
// the user's receive buffer with local loads.  One template serves all nine
// collectives; Ti/Tw/To are the user-input, wire (staging) and user-output
// element types and Red the reduction functor.  Pure data-movement collectives
// instantiate it once with byte elements.  FAM says which operations an
// instantiation serves, so that the reducing instantiations (one per element
// type and operator) do not carry the code and registers of the data-movement
// operations and the byte instantiation none of the reductions.
#pragma once
#include "datamove.cuh"

namespace Al {
namespace internal {
namespace device {

constexpr int kFamAll = 0;     // every operation (mixed element types)
constexpr int kFamReduce = 1;  // allreduce, reduce, reduce_scatter (+ barrier)
constexpr int kFamMove = 2;    // allgather, alltoall, bcast, gather, scatter (+ barrier)

/** Whether an instantiation of family `fam` serves operation `kind`. */
inline bool family_serves(int fam, DevColl kind) {
  const bool reduces = kind == DevColl::allreduce || kind == DevColl::reduce || kind == DevColl::reduce_scatter;
  return fam == kFamAll || kind == DevColl::barrier || (fam == kFamReduce) == reduces;
}

template <typename Ti, typename Tw, typename To, typename Red, int FAM = kFamAll>
__global__ void __launch_bounds__(512, 1) coll_kernel(const __grid_constant__ CollParams P, Red red) {
  constexpr bool kReduces = FAM != kFamMove, kMoves = FAM != kFamReduce;
  constexpr int kCopyUnroll = FAM == kFamMove ? kUnroll : kUnroll / 2;   // next to the folding loops eight loads per copying thread spill
  constexpr int kPair = FAM == kFamAll ? 1 : 2;   // conversions beside the fold leave registers for one vector of up to four ranks
  const Workspace& ws = P.ws;
  const int p = ws.p;
  const int rank = P.rank0 + (int)blockIdx.y;
  if (poisoned(ws, rank)) return;
  stamp(ws, 0);

  const DevColl kind = (DevColl)P.kind;
  const CountTable& T = P.tab[rank];
  // Operations that also exist as window kernels (registered buffers) announce which protocol this
  // rank runs, so that a rank that chose the other one is not left waiting (see protocols_agree).
  const uint64_t my_proto = proto_word(kProtoStaged, P.kind, P.two_phase | (P.pipelined << 1));
  const bool announces = kind == DevColl::reduce_scatter || kind == DevColl::allgather || kind == DevColl::alltoall ||
                         kind == DevColl::bcast;
  if (announces && blockIdx.x == 0) post_entered(ws, rank, P.seq, my_proto, 0, 0);
  const size_t half = ws.half_bytes;
  const size_t full_e = half / sizeof(Tw);
  const size_t cap_b = (half / (size_t)p) / 256 * 256;           // one slot per source rank
  const size_t cap_e = P.slot_elems ? P.slot_elems : cap_b / sizeof(Tw);  // elements moved per slot and chunk
  const size_t cap2_b = (half / 2 / (size_t)p) / 256 * 256;      // two-phase allreduce: two areas of p slots
  const size_t unit2 = (size_t)p * (cap2_b / sizeof(Tw));        // ... elements per chunk
  const size_t area_b = half / 2 / 256 * 256;                    // byte offset of the second area
  constexpr size_t VEC = 16 / sizeof(Tw);  // split boundaries stay 16-byte aligned in staging
  constexpr bool kSame = std::is_same<Ti, Tw>::value && std::is_same<Tw, To>::value;
  const Ti* send = (const Ti*)P.send[rank];
  To* recv = (To*)P.recv[rank];
  const int root = P.root;
  // What a rank contributes to its own result does not travel through staging: reductions read it from the send
  // buffer, data movement copies it straight to its place (1/p of the staged bytes; the host has checked the buffers).
  const bool own = P.own_direct[rank] != 0;
  const bool two_phase = kReduces && kind == DevColl::allreduce && P.two_phase;
  const bool rooted = kind == DevColl::reduce || kind == DevColl::gather;   // one destination: the root
  const bool from_root = kind == DevColl::bcast || kind == DevColl::scatter;
  // Small slices: the CTA's threads split into p groups that serve all peers at once instead of one peer after the other.
  const unsigned grp_lanes = blockDim.x / (unsigned)p;
  const unsigned grp = threadIdx.x / grp_lanes, grp_lane = threadIdx.x % grp_lanes;
  constexpr size_t kSmallBytes = 65536;  // per-peer slice up to which the peers are served in parallel
  auto longest = [&](const size_t* counts, size_t base, size_t unit) {
    size_t m = 0;
    for (int r = 0; r < p; ++r) {
      const size_t len = clamp_len(counts[r], base, unit);
      m = len > m ? len : m;
    }
    return m;
  };

  // ------------------------------ publish (remote stores) --------------------
  // Each step below is written so that the copying code appears once per family: destinations are either all ranks
  // (one read, p stores) or visited one after the other with a rotated start, so that at every moment the ranks write
  // to distinct peers instead of all converging on one GPU's ingress link.
  auto publish = [&](uint64_t c, unsigned part, unsigned nparts) __attribute__((always_inline)) {
    if (!send || kind == DevColl::barrier || (from_root && rank != root)) return;
    const size_t half_off = (size_t)((P.seq + c) & 1) * half;
    const size_t unit = two_phase ? unit2 : (from_root ? full_e : cap_e), base = c * unit;
    const size_t slot_b = two_phase ? (size_t)rank * cap2_b : (from_root ? 0 : (size_t)rank * cap_b);
    size_t lo, hi;
    int i0 = 0;
    const bool fan = kind == DevColl::allgather || kind == DevColl::bcast || (kind == DevColl::allreduce && !two_phase);
    if (fan) {
      const size_t len = clamp_len(kind == DevColl::allgather ? T.send_counts[rank] : P.count, base, unit);
      split_range(len, part, nparts, VEC, lo, hi);
      unsigned ranks = (1u << p) - 1;
      char* mine = nullptr;   // where the own copy goes if not into staging
      if (own) {
        if (kMoves && kind == DevColl::allgather) mine = (char*)(recv + T.recv_displs[rank] + base + lo);
        if (mine == nullptr || mine == (const char*)(send + base + lo) || ((uintptr_t)mine & 15)) ranks &= ~(1u << rank);
      }
      if (hi > lo)
        cta_publish<Ti, Tw>(ranks, [&](int d) { return d == rank && mine ? mine : ws.stage[d] + half_off + slot_b + lo * sizeof(Tw); },
                            send + base + lo, hi - lo);
      // the own copy of an allgather whose place is not 16-byte aligned is made by the loop below
      if (!(mine && !(ranks >> rank & 1))) return;
      i0 = p - 1;
    }
    int i1 = p;
    unsigned lane = threadIdx.x, lanes = blockDim.x;
    const size_t* counts = kind == DevColl::reduce_scatter ? T.recv_counts : T.send_counts;
    if (!fan && !rooted && !two_phase && grp_lanes >= 32 && longest(counts, base, unit) * sizeof(Tw) <= kSmallBytes) {
      i0 = (int)grp;
      i1 = i0 < p ? i0 + 1 : i0;
      lane = grp_lane;
      lanes = grp_lanes;
    }
    for (int i = i0; i < i1; ++i) {
      const int d = (rank + 1 + i) % p;
      if (rooted && d != root) continue;
      size_t from = base, len;
      if (two_phase) {                       // slice d of the chunk
        size_t s_lo, s_hi;
        split_range(clamp_len(P.count, base, unit), (unsigned)d, (unsigned)p, VEC, s_lo, s_hi);
        from = base + s_lo;
        len = s_hi - s_lo;
      } else if (rooted || fan) {
        len = clamp_len(kind == DevColl::reduce ? P.count : T.send_counts[rank], base, unit);
      } else {
        from = T.send_displs[d] + base;
        len = clamp_len(counts[d], base, unit);
      }
      split_range(len, part, nparts, VEC, lo, hi);
      if (hi <= lo) continue;
      const Ti* src = send + from + lo;
      char* dst = ws.stage[d] + half_off + slot_b + lo * sizeof(Tw);
      if (own && d == rank) {
        if (!kMoves || kind == DevColl::reduce_scatter || kind == DevColl::reduce || two_phase) continue;
        dst = (char*)(recv + T.recv_displs[rank] + base + lo);
        if (dst == (const char*)src) continue;
      }
      group_publish<Ti, Tw, kCopyUnroll>(dst, src, hi - lo, lane, lanes);
    }
  };

  // ------------------------------ consume (local loads) ----------------------
  // Reductions: fold the p contributions of chunk c.  The result goes to the receive buffer or, in the first phase of a
  // two-phase allreduce, to everyone's second area.
  auto fold = [&](uint64_t c, unsigned part, unsigned nparts) __attribute__((always_inline)) {
    if constexpr (kReduces) {
      if (kind == DevColl::reduce && rank != root) return;
      const size_t half_off = (size_t)((P.seq + c) & 1) * half;
      const char* mystage = ws.stage[rank] + half_off;
      const size_t unit = two_phase ? unit2 : cap_e, base = c * unit, slot_b = two_phase ? cap2_b : cap_b;
      size_t len = clamp_len(kind == DevColl::reduce_scatter ? T.recv_counts[rank] : P.count, base, unit), s_lo = 0, s_hi, lo, hi;
      if (two_phase) {
        split_range(len, (unsigned)rank, (unsigned)p, VEC, s_lo, s_hi);
        len = s_hi - s_lo;
      }
      split_range(len, part, nparts, VEC, lo, hi);
      if (hi <= lo || (!two_phase && !recv)) return;
      const char* mine = own ? (const char*)(send + (kind == DevColl::reduce_scatter ? T.send_displs[rank] : 0) + base + s_lo + lo) : nullptr;
      auto src = [&](int r) { return mine && r == rank ? mine : mystage + (size_t)r * slot_b + lo * sizeof(Tw); };
      To* out = recv + base + s_lo + lo;
      auto area = [&](int d) { return ws.stage[d] + half_off + area_b + (size_t)rank * cap2_b + lo * sizeof(Tw); };
      if constexpr (kSame) {
        reduce_to<Tw, To, kPair>(two_phase ? (1u << p) - 1 : 1u << rank, [&](int d) { return !two_phase || (own && d == rank) ? out : (To*)area(d); },
                          src, p, hi - lo, red, P.scale, P.int_div);
      } else if (two_phase) {
        reduce_to<Tw, Tw, kPair>((1u << p) - 1, [&](int d) { return (Tw*)area(d); }, src, p, hi - lo, red, P.scale, P.int_div);
      } else {
        reduce_to<Tw, To, kPair>(1u << rank, [&](int) { return out; }, src, p, hi - lo, red, P.scale, P.int_div);
      }
    }
  };
  // Data movement and the second phase of a two-phase allreduce: copy what the ranks left in this rank's staging half.
  auto copy_out = [&](uint64_t c, unsigned part, unsigned nparts) __attribute__((always_inline)) {
    if (!recv || kind == DevColl::barrier || (kind == DevColl::gather && rank != root) || (kind == DevColl::bcast && rank == root)) return;
    const char* mystage = ws.stage[rank] + (size_t)((P.seq + c) & 1) * half;
    const size_t unit = two_phase ? unit2 : (from_root ? full_e : cap_e), base = c * unit;
    int i0 = 0, i1 = from_root ? 1 : p;
    unsigned lane = threadIdx.x, lanes = blockDim.x;
    if (!from_root && !two_phase && grp_lanes >= 32 && longest(T.recv_counts, base, unit) * sizeof(Tw) <= kSmallBytes) {
      i0 = (int)grp;
      i1 = i0 < p ? i0 + 1 : i0;
      lane = grp_lane;
      lanes = grp_lanes;
    }
    for (int i = i0; i < i1; ++i) {
      const int r = (rank + 1 + i) % p;
      if (own && r == rank) continue;   // already in place
      const char* src = mystage;
      size_t to = base, len, lo, hi;
      if (two_phase) {
        size_t s_lo, s_hi;
        split_range(clamp_len(P.count, base, unit), (unsigned)r, (unsigned)p, VEC, s_lo, s_hi);
        src += area_b + (size_t)r * cap2_b;
        to += s_lo;
        len = s_hi - s_lo;
      } else if (from_root) {
        len = clamp_len(kind == DevColl::bcast ? P.count : T.recv_counts[rank], base, unit);
      } else {
        src += (size_t)r * cap_b;
        to += T.recv_displs[r];
        len = clamp_len(T.recv_counts[r], base, unit);
      }
      split_range(len, part, nparts, VEC, lo, hi);
      if (hi <= lo) continue;
      if constexpr (std::is_same<Tw, To>::value)
        group_copy<kCopyUnroll, Rest::spread>((char*)(recv + to + lo), src + lo * sizeof(Tw), (hi - lo) * sizeof(Tw), true, lane, lanes);
      else if (two_phase)
        cta_expand<Tw, To>(recv + to + lo, (const Tw*)src + lo, hi - lo);
    }
  };

  // =========================== schedule ========================================
  // Serial: every CTA publishes its share of a chunk, waits for everyone's and consumes its share.
  // Pipelined (large uniform reduce_scatter / allgather / alltoall): the lower half of the grid only publishes
  // (NVLink stores), the upper half only consumes (HBM traffic), so chunk c+1 crosses the links while chunk c is
  // copied out.  A slot is reused every second chunk; the publisher waits for the consumers' C flag of the chunk
  // that used it before.
  const bool pipelined = P.pipelined && gridDim.x >= 2;
  const unsigned n_pub = pipelined ? gridDim.x / 2 : gridDim.x, n_con = pipelined ? gridDim.x - n_pub : gridDim.x;
  const bool publishes = blockIdx.x < n_pub, consumes = !pipelined || !publishes;
  const unsigned part = consumes && pipelined ? blockIdx.x - n_pub : blockIdx.x;
  const bool reducing = kReduces && (kind == DevColl::allreduce || kind == DevColl::reduce || kind == DevColl::reduce_scatter);
  __shared__ uint64_t s_chunks;
  uint64_t G = P.local_chunks[rank];
  for (uint64_t c = 0; c < G; ++c) {
    const uint64_t e = make_epoch(P.seq, c + 1);
    if (publishes) {
      if (pipelined && c >= 2 && !wait_all(ws, rank, FlagLayout::off_C, 2, make_epoch(P.seq, c - 1), P.timeout_ns)) return;
      publish(c, part, n_pub);
      arrive_and_post(ws, rank, FlagLayout::off_A, 0, n_pub, e, c == 0, (int)(P.seq & 1), P.local_chunks[rank], my_proto);
      if (c == 0) stamp(ws, 1);
    }
    if (!consumes) continue;
    if (!wait_all(ws, rank, FlagLayout::off_A, 0, e, P.timeout_ns)) return;
    if (c == 0) {
      stamp(ws, 2);
      if (p > 1 && !protocols_agree(ws, rank, P.seq, my_proto)) return;
      if (!pipelined) {   // the ranks' chunk counts may differ (vector forms, rooted operations): everyone does the most
        if (threadIdx.x == 0) {
          uint64_t g = 1;
          for (int r = 0; r < p; ++r) {
            const uint64_t m = ld_relaxed_sys(flag_slot(ws.flags[rank], FlagLayout::off_meta, (int)(P.seq & 1) * kMaxRanks + r));
            g = m > g ? m : g;
          }
          s_chunks = g;
        }
        __syncthreads();
        G = s_chunks;
      }
    }
    if (reducing) fold(c, part, n_con);
    if (two_phase) {
      arrive_and_post(ws, rank, FlagLayout::off_B, 1, n_con, e, false, 0, 0);
      if (!wait_all(ws, rank, FlagLayout::off_B, 1, e, P.timeout_ns)) return;
    }
    if (!reducing || two_phase) copy_out(c, part, n_con);
    if (pipelined) arrive_and_post(ws, rank, FlagLayout::off_C, 2, n_con, e, false, 0, 0);
  }

  stamp(ws, 3);
  if (pipelined) {
    // Closing barrier: every peer has consumed every chunk, both halves are free.
    (void)wait_all(ws, rank, FlagLayout::off_C, 2, make_epoch(P.seq, G), P.timeout_ns);
  } else if (G > 1) {
    // Both halves were used: make sure every peer is done with them before the
    // next launch (which may start on either half) writes into them.
    const uint64_t e = make_epoch(P.seq, 1);
    arrive_and_post(ws, rank, FlagLayout::off_C, 2, gridDim.x, e, false, 0, 0);
    (void)wait_all(ws, rank, FlagLayout::off_C, 2, e, P.timeout_ns);
  }
}

}  // namespace device
}  // namespace internal
}  // namespace Al
