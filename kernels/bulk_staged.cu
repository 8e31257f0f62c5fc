// The staged protocol with every rank of the communicator on this GPU, large uniform operations: the data is
// moved by the bulk copy engine (cp.async.bulk) through shared memory.
//
// Publish, handshake, consume, chunks, epochs and flags are those of the serial schedule of coll_kernel.cuh.  What differs is
// what bounds it: with all ranks on one GPU the staging traffic is HBM traffic, and the load / store loops of that kernel keep
// what 16 warps per SM hold in registers under way.  Here one thread per CTA keeps up to 160 KB of loads under way per SM,
// across destinations and sources without a gap, and needs no registers for them; reductions are folded out of shared
// memory while the next tiles arrive.  Loops / bulk copies, us: bucket of 4 x 26 MB 104 / 99 (525 MB of staged traffic, 5.3 TB/s),
// bf16 allreduce of 2 x 128 MiB 303 / 240, reduce_scatter of 4 x 128 MiB 307 / 258, alltoall of 8 x 4 MiB 42.8 / 28.3, bucket of 8 x 12 MB
// with a bf16 wire, converted between the tiles and staging by all threads, 103 / 90.  Slices that begin anywhere are shifted into
// the destination's words out of the tiles, which is what gains most: reduce_scatter of 4 x 256 MiB 1127 / 604, of 8 x 128 MiB 843 / 655,
// allgather of 2 x 128 MiB 209 / 157.  (Reduce_scatter of eight ranks in whole words is the other way round from 32 MiB on: 144 / 161.)
// (Between GPUs the engine's stores to peers were slower than SM stores - 4 GPUs, 1 GiB allgather 1534 us against
// 1291 us - so ranks on GPUs of their own keep coll_kernel.)
//
// Every load reads this GPU's own memory and has exactly one destination CTA.  Every wait is bounded.
#include "al/cuda/cuda.hpp"
#include "al/device/kernels.hpp"
#include "bulk_copy.cuh"
#include "datamove.cuh"

namespace Al {
namespace internal {
namespace device {

namespace {

constexpr int kBufs = 6;
constexpr int kTile = 32768;
constexpr size_t kSmem = (size_t)kBufs * kTile + 128;  // tiles + barriers
constexpr int kThreads = 512;

/** T: element type in staging; U: element type of the user's buffers (another one for an allreduce with a narrower wire type);
 *  RAGGED: slices do not begin on 16-byte boundaries of the user's buffers (as a run-time choice it cost the others 4 %). */
template <typename T, typename U, bool RAGGED, typename Red>
__global__ void __launch_bounds__(kThreads, 1) bulk_staged_kernel(const __grid_constant__ CollParams P, Red red) {
  constexpr bool kMixed = !std::is_same<T, U>::value;
  extern __shared__ __align__(128) unsigned char dyn_smem[];
  const Workspace& ws = P.ws;
  const int p = ws.p;
  const int rank = P.rank0 + (int)blockIdx.y;
  if (poisoned(ws, rank)) return;
  stamp(ws, 0);
  const DevColl kind = (DevColl)P.kind;
  const uint64_t my_proto = proto_word(kProtoStaged, P.kind, P.two_phase);
  const bool announces = kind != DevColl::allreduce;
  if (announces && blockIdx.x == 0) post_entered(ws, rank, P.seq, my_proto, 0, 0);

  constexpr size_t VEC = 16 / sizeof(T);
  const size_t half = ws.half_bytes;
  const size_t cap_b = (half / (size_t)p) / 256 * 256, cap2_b = (half / 2 / (size_t)p) / 256 * 256;
  const size_t area_b = half / 2 / 256 * 256;
  const bool reduces = kind == DevColl::allreduce || kind == DevColl::reduce_scatter;
  const bool two_phase = kind == DevColl::allreduce && P.two_phase;
  const size_t slot_b = two_phase ? cap2_b : cap_b;
  const size_t unit = two_phase ? (size_t)p * (cap2_b / sizeof(T)) : cap_b / sizeof(T);  // elements per chunk (of a slice)
  const size_t count = P.count;                                                          // vector, or one rank's slice
  constexpr bool ragged = RAGGED;
  const char* send = (const char*)P.send[rank];
  char* recv = (char*)P.recv[rank];
  const unsigned cta = blockIdx.x, nct = gridDim.x;

  bulk::Ring<kBufs, kTile> ring;   // its parities live in thread 0 between the streams below
  if (threadIdx.x == 0) ring.init(dyn_smem, dyn_smem + (size_t)kBufs * kTile);
  const uint32_t tiles = bulk::smem_addr(dyn_smem), bars = tiles + kBufs * kTile;
  __syncthreads();

  /** Elements of slice `d` of chunk c that this CTA handles: [lo, hi) of the slice's part of the chunk, which starts at `base`. */
  struct Part { size_t base, lo, hi; };
  auto part_of = [&](uint64_t c, int d) {
    Part q;
    const size_t base = c * unit;
    size_t len = clamp_len(count, base, unit), s_lo = 0, s_hi;
    if (two_phase) {
      split_range(len, (unsigned)d, (unsigned)p, VEC, s_lo, s_hi);
      len = s_hi - s_lo;
    }
    split_range(len, cta, nct, VEC, q.lo, q.hi);
    q.base = base + s_lo;
    return q;
  };
  /** One copy: `bytes` from src to dst[0..ndst). */
  struct Job { const char* src; char* dst[kMaxRanks]; int ndst; size_t bytes; };
  __shared__ Job jobs[kMaxRanks];
  /** Run jobs[0..n) (filled by the first n threads): thread 0 streams their whole 16-byte words, tiles taking turns among the
   *  jobs; the few bytes that are left are copied by other threads meanwhile. */
  auto copy_jobs = [&](int n) {
    __syncthreads();
    bool ok = true;
    if (threadIdx.x == 0) {
      size_t total = 0;
      for (int j = 0; j < n; ++j) total += (jobs[j].bytes / 16 * 16 + kTile - 1) / kTile;
      struct Cursor { int j; size_t off; };
      auto seek = [&](Cursor& at) {   // to the next tile that exists; called only while there is one
        for (;;) {
          if (at.j == n) { at.j = 0; at.off += kTile; }
          if (at.off < jobs[at.j].bytes / 16 * 16) return;
          ++at.j;
        }
      };
      auto len = [&](const Cursor& at) {
        const size_t left = jobs[at.j].bytes / 16 * 16 - at.off;
        return (uint32_t)(left < kTile ? left : kTile);
      };
      Cursor in{0, 0}, out{0, 0};
      auto load = [&](size_t t) {
        const int s = (int)(t % kBufs);
        seek(in);
        bulk::mbar_expect_tx(ring.bar(s), len(in));
        bulk::g2s(ring.tile(s), jobs[in.j].src + in.off, len(in), ring.bar(s));
        ++in.j;
      };
      bulk::fence_proxy_async();  // flag acquires and plain stores before the engine touches the data
      size_t loaded = 0;
      for (; loaded < total && loaded < kBufs - 1; ++loaded) load(loaded);
      size_t t = 0;
      for (; t < total; ++t) {
        const int s = (int)(t % kBufs);
        if (!bulk::mbar_wait(ring.bar(s), (ring.parity >> s) & 1u, P.timeout_ns)) { ok = false; break; }
        ring.parity ^= 1u << s;
        seek(out);
        const Job& job = jobs[out.j];
        for (int i = 0; i < job.ndst; ++i) bulk::s2g(job.dst[i] + out.off, ring.tile(s), len(out));
        bulk::commit();
        ++out.j;
        if (loaded < total) {   // goes into the tile that the stores before these read from
          bulk::wait_read<1>();
          load(loaded++);
        }
      }
      if (!ok)                  // the copies in flight end before the block does (or it gives up on them)
        for (size_t u = t + 1; u < loaded; ++u) (void)bulk::mbar_wait(ring.bar((int)(u % kBufs)), (ring.parity >> (u % kBufs)) & 1u, P.timeout_ns);
      bulk::wait_all();
      bulk::fence_proxy_async();
      __threadfence_system();
    } else if (threadIdx.x >= 32 && threadIdx.x < 48) {
      for (int j = 0; j < n; ++j) {
        const size_t at = jobs[j].bytes / 16 * 16 + (threadIdx.x - 32);
        if (at < jobs[j].bytes)
          for (int i = 0; i < jobs[j].ndst; ++i) jobs[j].dst[i][at] = __ldcg(jobs[j].src + at);
      }
      bulk::fence_proxy_async();
    }
    const int bad = __syncthreads_or(!ok);
    if (bad && threadIdx.x == 0) report_timeout(ws, rank, rank, 6, make_epoch(P.seq, 1), 0);
    return bad == 0;
  };

  uint32_t parity = 0;   // every thread's view of the ring's parities (thread 0 hands them over)
  __shared__ uint32_t s_parity;
  /** The same for jobs of one destination where source and destination lie differently in their 16-byte words: tiles of aligned
   *  words arrive by the engine, all threads shift them into the destination's words. */
  auto shift_jobs = [&](int n) {
    constexpr uint32_t kWords = kTile / 16 - 1;   // of the destination; an unaligned source takes one more
    __syncthreads();
    auto words_of = [&](int j) {
      const size_t head = (0 - (uintptr_t)jobs[j].dst[0]) & 15;
      return jobs[j].bytes > head ? (jobs[j].bytes - head) / 16 : (size_t)0;
    };
    size_t total = 0;
    for (int j = 0; j < n; ++j) total += (words_of(j) + kWords - 1) / kWords;
    struct Cursor { int j; size_t off; };
    auto seek = [&](Cursor& at) {   // to the next tile that exists; called only while there is one
      for (;;) {
        if (at.j == n) { at.j = 0; at.off += kWords; }
        if (at.off < words_of(at.j)) return;
        ++at.j;
      }
    };
    auto len = [&](const Cursor& at) {
      const size_t left = words_of(at.j) - at.off;
      return (uint32_t)(left < kWords ? left : kWords);
    };
    Cursor in{0, 0}, out{0, 0};
    auto load = [&](size_t t) {
      const int s = (int)(t % kBufs);
      seek(in);
      const char* src = jobs[in.j].src + ((0 - (uintptr_t)jobs[in.j].dst[0]) & 15) + 16 * in.off;
      const unsigned sh = (unsigned)((uintptr_t)src & 15);
      const uint32_t bytes = 16 * (len(in) + (sh ? 1u : 0u));
      bulk::mbar_expect_tx(ring.bar(s), bytes);
      bulk::g2s(ring.tile(s), src - sh, bytes, ring.bar(s));
      ++in.j;
    };
    if (threadIdx.x == 0) {
      s_parity = ring.parity;
      bulk::fence_proxy_async();
      for (size_t t = 0; t < total && t < kBufs; ++t) load(t);
    }
    __syncthreads();
    parity = s_parity;
    bool good = true;
    for (size_t t = 0; t < total; ++t) {
      const int s = (int)(t % kBufs);
      const bool ok = bulk::mbar_wait(bars + 8 * s, (parity >> s) & 1u, P.timeout_ns);
      parity ^= 1u << s;
      seek(out);
      const size_t head = (0 - (uintptr_t)jobs[out.j].dst[0]) & 15;
      const uint32_t words = len(out);
      WordSource from((const char*)dyn_smem + (size_t)s * kTile, false);
      from.sh = (unsigned)((uintptr_t)(jobs[out.j].src + head) & 15);
      uint4* d = (uint4*)(jobs[out.j].dst[0] + head) + out.off;
      if (ok) {
        if (from.sh)
          for (uint32_t w = threadIdx.x; w < words; w += kThreads) d[w] = from.shifted(w);
        else
          for (uint32_t w = threadIdx.x; w < words; w += kThreads) d[w] = from.base[w];
      }
      ++out.j;
      if (__syncthreads_or(!ok)) {   // also: everyone has read the tile
        good = false;
        if (threadIdx.x == 0)        // the copies in flight end before the block does (or it gives up on them)
          for (size_t u = t; u < total && u < t + kBufs; ++u)
            (void)bulk::mbar_wait(bars + 8 * (u % kBufs), (parity >> (u % kBufs) ^ (u == t)) & 1u, P.timeout_ns);
        break;
      }
      if (threadIdx.x == 0 && t + kBufs < total) load(t + kBufs);
    }
    if (threadIdx.x == 0) ring.parity = parity;
    for (int j = 0; j < n; ++j) {    // bytes in front of the first word and behind the last
      const size_t head = (0 - (uintptr_t)jobs[j].dst[0]) & 15, behind = head + 16 * words_of(j) + (threadIdx.x - 16);
      if (threadIdx.x < 16 && threadIdx.x < head && threadIdx.x < jobs[j].bytes) jobs[j].dst[0][threadIdx.x] = __ldcg(jobs[j].src + threadIdx.x);
      if (threadIdx.x >= 16 && threadIdx.x < 32 && behind < jobs[j].bytes) jobs[j].dst[0][behind] = __ldcg(jobs[j].src + behind);
    }
    bulk::fence_proxy_async();       // plain stores above, engine loads behind the next flag
    __syncthreads();                 // the list may be filled again
    if (!good && threadIdx.x == 0) report_timeout(ws, rank, rank, 6, make_epoch(P.seq, 1), 0);
    return good;
  };
  /** The same with conversion: jobs[0..n) whose `bytes` counts elements of In, converted to Out.  All threads convert out of
   *  the tiles; eight elements are one or two 16-byte words on either side. */
  auto convert_jobs = [&](int n, auto in_type, auto out_type) {
    using In = decltype(in_type);
    using Out = decltype(out_type);
    constexpr uint32_t kElems = kTile / sizeof(In);
    __syncthreads();
    size_t total = 0;
    for (int j = 0; j < n; ++j) total += (jobs[j].bytes / 8 * 8 + kElems - 1) / kElems;
    struct Cursor { int j; size_t off; };
    auto seek = [&](Cursor& at) {   // to the next tile that exists; called only while there is one
      for (;;) {
        if (at.j == n) { at.j = 0; at.off += kElems; }
        if (at.off < jobs[at.j].bytes / 8 * 8) return;
        ++at.j;
      }
    };
    auto len = [&](const Cursor& at) {
      const size_t left = jobs[at.j].bytes / 8 * 8 - at.off;
      return (uint32_t)(left < kElems ? left : kElems);
    };
    Cursor in{0, 0}, out{0, 0};
    auto load = [&](size_t t) {
      const int s = (int)(t % kBufs);
      seek(in);
      const uint32_t bytes = len(in) * (uint32_t)sizeof(In);
      bulk::mbar_expect_tx(ring.bar(s), bytes);
      bulk::g2s(ring.tile(s), jobs[in.j].src + in.off * sizeof(In), bytes, ring.bar(s));
      ++in.j;
    };
    if (threadIdx.x == 0) {
      s_parity = ring.parity;
      bulk::fence_proxy_async();
      for (size_t t = 0; t < total && t < kBufs; ++t) load(t);
    }
    __syncthreads();
    parity = s_parity;
    struct alignas(8 * sizeof(In) < 16 ? 8 * sizeof(In) : 16) Ins { In e[8]; };
    union Outs { Out e[8]; uint4 u[8 * sizeof(Out) / 16]; };
    bool good = true;
    for (size_t t = 0; t < total; ++t) {
      const int s = (int)(t % kBufs);
      const bool ok = bulk::mbar_wait(bars + 8 * s, (parity >> s) & 1u, P.timeout_ns);
      parity ^= 1u << s;
      seek(out);
      const Job& job = jobs[out.j];
      const uint32_t groups = len(out) / 8;
      if (ok)
        for (uint32_t g = threadIdx.x; g < groups; g += kThreads) {
          const Ins v = ((const Ins*)(dyn_smem + (size_t)s * kTile))[g];
          Outs o;
#pragma unroll
          for (int k = 0; k < 8; ++k) o.e[k] = Elem<Out>::down(Elem<In>::up(v.e[k]));
          for (int i = 0; i < job.ndst; ++i) {
            uint4* d = (uint4*)(job.dst[i] + (out.off + 8 * (size_t)g) * sizeof(Out));
#pragma unroll
            for (int q = 0; q < (int)(8 * sizeof(Out) / 16); ++q) d[q] = o.u[q];
          }
        }
      ++out.j;
      if (__syncthreads_or(!ok)) {   // also: everyone has read the tile
        good = false;
        if (threadIdx.x == 0)        // the copies in flight end before the block does (or it gives up on them)
          for (size_t u = t; u < total && u < t + kBufs; ++u)
            (void)bulk::mbar_wait(bars + 8 * (u % kBufs), (parity >> (u % kBufs) ^ (u == t)) & 1u, P.timeout_ns);
        break;
      }
      if (threadIdx.x == 0 && t + kBufs < total) load(t + kBufs);
    }
    if (threadIdx.x == 0) ring.parity = parity;
    for (int j = 0; j < n; ++j) {    // the elements behind the last eight
      const size_t e = jobs[j].bytes / 8 * 8 + threadIdx.x;
      if (e < jobs[j].bytes) {
        const Out o = Elem<Out>::down(Elem<In>::up(__ldcg((const In*)jobs[j].src + e)));
        for (int i = 0; i < jobs[j].ndst; ++i) ((Out*)jobs[j].dst[i])[e] = o;
      }
    }
    bulk::fence_proxy_async();       // plain stores above, engine loads behind the next flag
    __syncthreads();                 // the list may be filled again
    if (!good && threadIdx.x == 0) report_timeout(ws, rank, rank, 6, make_epoch(P.seq, 1), 0);
    return good;
  };

  auto publish = [&](uint64_t c) {
    const size_t half_off = (size_t)((P.seq + c) & 1) * half;
    if constexpr (kMixed) {   // allreduce; the own slice is rounded to the wire type like the others and goes through staging
      const int n = two_phase ? p : 1;
      if ((int)threadIdx.x < n) {
        Job& job = jobs[threadIdx.x];
        const int d = (rank + 1 + (int)threadIdx.x) % p;
        const Part q = part_of(c, d);
        job.src = send + (q.base + q.lo) * sizeof(U);
        job.bytes = q.hi - q.lo;
        job.ndst = 0;
        for (int i = 0; i < (two_phase ? 1 : p); ++i)
          job.dst[job.ndst++] = ws.stage[two_phase ? d : (rank + 1 + i) % p] + half_off + (size_t)rank * slot_b + q.lo * sizeof(T);
      }
      return convert_jobs(n, U(), T());
    }
    if (kind == DevColl::allgather || (kind == DevColl::allreduce && !two_phase)) {  // one read, a store per rank
      if (threadIdx.x == 0) {
        Job& job = jobs[0];
        const Part q = part_of(c, rank);
        job.src = send + (q.base + q.lo) * sizeof(T);
        job.bytes = (q.hi - q.lo) * sizeof(T);
        job.ndst = 0;
        for (int i = 1; i < p; ++i) job.dst[job.ndst++] = ws.stage[(rank + i) % p] + half_off + (size_t)rank * slot_b + q.lo * sizeof(T);
        char* mine = recv + ((size_t)rank * count + q.base + q.lo) * sizeof(T);
        if (kind == DevColl::allgather) {
          if (ragged) {   // the own part does not lie on word boundaries of the receive buffer
            jobs[1] = job;
            jobs[1].dst[0] = mine;
            jobs[1].ndst = 1;
            if (mine == job.src) jobs[1].bytes = 0;
          } else if (mine != job.src) {
            job.dst[job.ndst++] = mine;
          }
        }
      }
      const bool done = copy_jobs(1);
      if constexpr (ragged) {
        if (!done) return false;
        if (threadIdx.x == 0) jobs[0] = jobs[1];
        return shift_jobs(1);
      }
      return done;
    }
    // slice d goes to rank d; the own one stays (reductions) or is copied to its place
    const size_t pitch = two_phase ? 0 : count;
    const bool keep = two_phase || (reduces && !ragged) || (!reduces && send == recv);   // a ragged own slice is folded out of staging
    const int n = keep ? p - 1 : p;
    if ((int)threadIdx.x < n) {
      Job& job = jobs[threadIdx.x];
      const int d = (rank + 1 + (int)threadIdx.x) % p;
      const Part q = part_of(c, d);
      job.src = send + ((size_t)d * pitch + q.base + q.lo) * sizeof(T);
      job.bytes = (q.hi - q.lo) * sizeof(T);
      job.ndst = 1;
      job.dst[0] = d == rank && !reduces ? recv + ((size_t)rank * count + q.base + q.lo) * sizeof(T)
                             : ws.stage[d] + half_off + (size_t)rank * slot_b + q.lo * sizeof(T);
    }
    if constexpr (ragged) return shift_jobs(n);
    else return copy_jobs(n);
  };

  /** Fold the p contributions of the own slice; the result goes to the receive buffer and, in two phases, to every peer. */
  auto fold = [&](uint64_t c) {
    const size_t half_off = (size_t)((P.seq + c) & 1) * half;
    const Part q = part_of(c, rank);
    const size_t bytes = (q.hi - q.lo) * sizeof(T), whole = bytes / 16 * 16;
    const size_t pitch = kind == DevColl::reduce_scatter ? (size_t)rank * count : 0;
    const char* own = send + (pitch + q.base + q.lo) * sizeof(T);
    const char* slots = ws.stage[rank] + half_off + q.lo * sizeof(T);
    auto src = [&](int r) { return !kMixed && !ragged && r == rank ? own : slots + (size_t)r * slot_b; };
    auto dst = [&](int d) {
      return d == rank && !(kMixed && two_phase) ? recv + (q.base + q.lo) * sizeof(U) : ws.stage[d] + half_off + area_b + (size_t)rank * cap2_b + q.lo * sizeof(T);
    };
    const uint32_t sub = (uint32_t)(kTile / p) / 256 * 256;   // bytes of one rank's part of a tile
    const size_t n = (whole + sub - 1) / sub;
    auto load = [&](size_t t) {
      const int s = (int)(t % kBufs);
      const size_t off = t * sub;
      const uint32_t len = (uint32_t)(whole - off < sub ? whole - off : sub);
      bulk::mbar_expect_tx(ring.bar(s), len * (uint32_t)p);
      for (int r = 0; r < p; ++r) bulk::g2s(ring.tile(s) + (uint32_t)r * sub, src(r) + off, len, ring.bar(s));
    };
    if (threadIdx.x == 0) {
      s_parity = ring.parity;
      bulk::fence_proxy_async();
      for (size_t t = 0; t < n && t < kBufs; ++t) load(t);
    }
    __syncthreads();
    parity = s_parity;
    using A = typename Elem<T>::Acc;
    union Pack { uint4 u; T e[VEC]; };
    bool good = true;
    for (size_t t = 0; t < n; ++t) {
      const int s = (int)(t % kBufs);
      const bool ok = bulk::mbar_wait(bars + 8 * s, (parity >> s) & 1u, P.timeout_ns);
      parity ^= 1u << s;
      const size_t off = t * sub;
      const uint32_t words = (uint32_t)((whole - off < sub ? whole - off : sub) / 16);
      if (ok)
        for (uint32_t w = threadIdx.x; w < words; w += kThreads) {
          const uint4* in = (const uint4*)(dyn_smem + (size_t)s * kTile) + w;
          A acc[VEC];
#pragma unroll
          for (int r = 0; r < kMaxRanks; ++r)
            if (r < p) {
              Pack x;
              x.u = in[(size_t)r * (sub / 16)];
#pragma unroll
              for (int k = 0; k < (int)VEC; ++k) {
                const A a = Elem<T>::up(x.e[k]);
                acc[k] = r == 0 ? a : red(acc[k], a);
              }
            }
          if (kMixed && !two_phase) {
            union { U e[VEC]; uint4 u[(VEC * sizeof(U) + 15) / 16]; } o;
#pragma unroll
            for (int k = 0; k < (int)VEC; ++k) o.e[k] = Elem<U>::down(finish_acc(acc[k], P.scale, P.int_div));
            uint4* d = (uint4*)(dst(rank) + (off / sizeof(T) + VEC * (size_t)w) * sizeof(U));
#pragma unroll
            for (int q4 = 0; q4 < (int)(VEC * sizeof(U) / 16); ++q4) d[q4] = o.u[q4];
            continue;
          }
          Pack o;
#pragma unroll
          for (int k = 0; k < (int)VEC; ++k) o.e[k] = Elem<T>::down(finish_acc(acc[k], P.scale, P.int_div));
          if (two_phase) {
#pragma unroll
            for (int d = 0; d < kMaxRanks; ++d)
              if (d < p) *(uint4*)(dst(d) + off + 16 * (size_t)w) = o.u;
          } else {
            *(uint4*)(dst(rank) + off + 16 * (size_t)w) = o.u;
          }
        }
      if (__syncthreads_or(!ok)) {   // also: everyone has read the tile
        good = false;
        if (threadIdx.x == 0)        // the copies in flight end before the block does (or it gives up on them)
          for (size_t u = t; u < n && u < t + kBufs; ++u)
            (void)bulk::mbar_wait(bars + 8 * (u % kBufs), (parity >> (u % kBufs) ^ (u == t)) & 1u, P.timeout_ns);
        break;
      }
      if (threadIdx.x == 0 && t + kBufs < n) load(t + kBufs);
    }
    if (threadIdx.x == 0) ring.parity = parity;
    // the elements behind the last whole word
    const size_t e = whole / sizeof(T) + threadIdx.x;
    if (e < q.hi - q.lo) {
      A acc = A();
      for (int r = 0; r < p; ++r) {
        const A a = Elem<T>::up(__ldcg((const T*)src(r) + e));
        acc = r == 0 ? a : red(acc, a);
      }
      const A v = finish_acc(acc, P.scale, P.int_div);
      if (two_phase) {
        for (int d = 0; d < p; ++d) ((T*)dst(d))[e] = Elem<T>::down(v);
      } else {
        ((U*)dst(rank))[e] = Elem<U>::down(v);
      }
    }
    bulk::fence_proxy_async();   // plain stores above, engine loads of the peers behind the next flag
    if (!good && threadIdx.x == 0) report_timeout(ws, rank, rank, 6, make_epoch(P.seq, 1), 0);
    return good;
  };

  auto copy_out = [&](uint64_t c) {
    const char* mystage = ws.stage[rank] + (size_t)((P.seq + c) & 1) * half + (two_phase ? area_b : 0);
    const size_t pitch = two_phase ? 0 : count;
    const int n = kMixed ? p : p - 1;   // the own slice is in place unless it still has to be converted
    if ((int)threadIdx.x < n) {
      Job& job = jobs[threadIdx.x];
      const int r = (rank + 1 + (int)threadIdx.x) % p;
      const Part q = part_of(c, r);
      job.src = mystage + (size_t)r * slot_b + q.lo * sizeof(T);
      job.bytes = (q.hi - q.lo) * (kMixed ? 1 : sizeof(T));
      job.ndst = 1;
      job.dst[0] = recv + ((size_t)r * pitch + q.base + q.lo) * sizeof(U);
    }
    if constexpr (kMixed) return convert_jobs(n, T(), U());
    if constexpr (ragged) return shift_jobs(n);
    return copy_jobs(n);
  };

  const uint64_t G = P.local_chunks[rank];
  for (uint64_t c = 0; c < G; ++c) {
    const uint64_t e = make_epoch(P.seq, c + 1);
    if (!publish(c)) return;
    if (c == 0) stamp(ws, 1);
    arrive_and_post(ws, rank, FlagLayout::off_A, 0, nct, e, c == 0, (int)(P.seq & 1), G, my_proto);
    if (!wait_all(ws, rank, FlagLayout::off_A, 0, e, P.timeout_ns)) return;
    if (c == 0) {
      stamp(ws, 2);
      if (!protocols_agree(ws, rank, P.seq, my_proto)) return;
    }
    if (reduces && !fold(c)) return;
    if (two_phase) {
      arrive_and_post(ws, rank, FlagLayout::off_B, 1, nct, e, false, 0, 0);
      if (!wait_all(ws, rank, FlagLayout::off_B, 1, e, P.timeout_ns)) return;
    }
    if ((!reduces || two_phase) && !copy_out(c)) return;
  }
  stamp(ws, 3);
  if (G > 1) {   // both halves were used
    const uint64_t e = make_epoch(P.seq, 1);
    arrive_and_post(ws, rank, FlagLayout::off_C, 2, nct, e, false, 0, 0);
    (void)wait_all(ws, rank, FlagLayout::off_C, 2, e, P.timeout_ns);
  }
}

template <typename T, typename U = T, typename Red>
void launch_one(const CollParams& P, Red red, int ctas, int local_ranks, cudaStream_t stream) {
  auto k = bulk_staged_kernel<T, U, false, Red>;
  if ((DevColl)P.kind != DevColl::allreduce && P.count * sizeof(T) % 16 != 0) k = bulk_staged_kernel<T, T, true, Red>;
  AL_CHECK_CUDA(cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
  void* args[] = {(void*)&P, (void*)&red};
  AL_CHECK_CUDA(cudaLaunchCooperativeKernel((const void*)k, dim3((unsigned)ctas, (unsigned)local_ranks, 1), dim3(kThreads), args, kSmem, stream));
}

}  // namespace

bool bulk_staged_supported(DevColl kind, DType user, DType wire, ReductionOperator op) {
  if (kind == DevColl::allgather || kind == DevColl::alltoall) return user == DType::u8 && wire == DType::u8;
  if ((kind != DevColl::allreduce && kind != DevColl::reduce_scatter) || (op != ReductionOperator::sum && op != ReductionOperator::avg)) return false;
  if (user == wire) return user == DType::f32 || user == DType::bf16 || user == DType::f16;
  return kind == DevColl::allreduce && user == DType::f32 && (wire == DType::bf16 || wire == DType::f16);
}

void launch_bulk_staged(const CollParams& P, DType user, DType wire, int ctas, int local_ranks, cudaStream_t stream) {
  const DevColl kind = (DevColl)P.kind;
  if (!bulk_staged_supported(kind, user, wire, (ReductionOperator)P.op) || P.pipelined || P.slot_elems)
    throw_al_exception("bulk staged kernel: unsupported operation");
  const bool mixed = user != wire;
  switch (wire) {
    case DType::f32: return launch_one<float>(P, RedSum(), ctas, local_ranks, stream);
    case DType::bf16:
      return mixed ? launch_one<__nv_bfloat16, float>(P, RedSum(), ctas, local_ranks, stream) : launch_one<__nv_bfloat16>(P, RedSum(), ctas, local_ranks, stream);
    case DType::f16: return mixed ? launch_one<__half, float>(P, RedSum(), ctas, local_ranks, stream) : launch_one<__half>(P, RedSum(), ctas, local_ranks, stream);
    default: return launch_one<unsigned char>(P, RedNone(), ctas, local_ranks, stream);
  }
}

}  // namespace device
}  // namespace internal
}  // namespace Al
