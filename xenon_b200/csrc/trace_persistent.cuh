// trace_persistent.cuh — persistent-warp traversal of a ray queue with per-lane refill, the one
// traversal of every kernel that traces rays.
//
// A warp holds 32 rays, and its lanes are at one of three kinds of work: a pair of nodes (of the
// TLAS or of a BLAS: one code), a BLAS leaf's triangles, or the way between TLAS and BLAS. Each
// step the warp does the kind that most of its lanes wait for, for those lanes; the others wait.
// It stays with node pairs until half of the lanes that began them have left. A lane that has
// finished waits until `refill` lanes have, then they write their answers and take new rays
// together. refill = 32 is one ray per thread.
//
// What bounds it: issue slots and the latency of the dependent node loads (DRAM under 5 %), so the
// aim is lanes per instruction and instructions per node. B200, one wave at a time, ms per sample
// at 1920x1080, closest hits / any hits:
//                                              1.31 M triangles,   261 instances of
//                                              one instance        12 meshes
//   each lane does whatever it is at            1.43 / 1.10         6.41 / 4.67
//   votes, packed slab test, 256-bit loads      1.24 / 0.93         5.85 / 4.05
//   and TLAS children tested with their parent  1.24 / 0.95         4.78 / 2.89
// Tried and slower: voting again after every node pair (3 %), staying with node pairs down to 8
// lanes (3 %), 64 registers for 8 blocks an SM (1-20 %), the waiting words in registers (4 %), an
// entry distance with every BLAS entry, to drop those beyond the hit at the pop (4 %).
//
// Per ray, the leaves and triangles are visited in the order of the reference's recursive loops
// (tlas.cpp:172-245, blas.cpp:211-265), so closest-hit results, including which of two equal-t
// triangles wins, are the reference's. A BLAS child's test is the reference's, made when its parent
// is expanded. A TLAS child is tested when its parent is expanded, too, where the reference tests
// it when it is popped: the closest hit only comes nearer, so a child that misses then would miss
// later; one that hits carries its entry distance on the stack, and its test at the pop is that
// distance against the hit by then, the only term of the reference's test that has changed.
// Any-hit rays (kAny) only need *whether* some triangle lies in [tmin, tmax], which does not depend
// on order: shadow rays descend farther child first by default (they start on a surface, among boxes
// that do not occlude them: 1-8 % per sample), ray queries nearer first (1 M uniform rays on 261
// instances 397 us, farther first 461).
#pragma once

#include <type_traits>

#include "dev_scene.cuh"
#include "trace_grid.h"

namespace xbd {

struct TraceQueue {
  const float4* ray_o;      // org xyz, w = tmin (closest) / tmax (any-hit shadow items)
  const float4* ray_d;      // dir xyz, w = tmax (closest) / bits(path) (shadow items)
  const int32_t* count;     // number of rays (device)
  int32_t* fetch;           // work cursor (device, zeroed before launch)
  // closest-hit outputs
  float4* hit;              // t, u, v, bits(prim)
  int32_t* hit_inst;
  // any-hit (shadow) outputs: unoccluded items add contrib to L[path]
  const float4* contrib;
  float4* L;
  unsigned long long* stats;
  int far_first;            // any-hit: descend into the farther child first
};

// Where a warp's rays come from and where their answers go: the renderer's queues, the rays
// taken from a shared cursor (a TraceQueue; xb_trace_rays_device has its own, in renderer.cu).
//   end()                   one past the last ray index this warp may take
//   lanes()                 how many of the warp's lanes take rays
//   grab(lane, leader, k)   the first of k consecutive ray indices for the warp's idle lanes
//                           (warp-uniform: every lane calls it with the same k)
//   load<kAny>(ray, o, d, tmin, tmax), finish_any(ray, occluded),
//   finish_closest(sc, ray, o, d, tmin, tmax, h), stats()
// A queue shorter than the lanes of the launch's warps that fit on the GPU at once is spread over all
// of those warps (trace_grid.h): a warp's time is the union of what its lanes do, one kind of work after the other,
// so 8 rays on each of four warps are done sooner than 32 on one. That is most bounces of a path:
// ms per sample at 1920x1080, closest / any hits, 261 instances 4.76 / 2.90 -> 4.05 / 2.43, one
// instance 1.25 / 0.95 -> 1.12 / 0.87; a 256x256 sample in a box 0.276 / 0.203 -> 0.235 / 0.185
// (5 % of the closest hits' gain is the seventh block an SM that 72 registers allow). Shading the
// same way was 4-15 % slower. A warp's first rays are its own by its number; only later ones come
// from the cursor.
struct QueueIO {
  TraceQueue q;
  int n, per_warp;
  bool first;
  __device__ __forceinline__ QueueIO(const TraceQueue& tq, int warps)
      : q(tq), n(*tq.count), per_warp(xb::queue_lanes(n, warps)), first(true) {}
  __device__ __forceinline__ int end() const { return n; }
  __device__ __forceinline__ int lanes() const { return per_warp; }
  __device__ __forceinline__ int grab(int lane, int leader, int k) {
    const int grid_warps = (int)((gridDim.x * blockDim.x) >> 5);
    if (first) {   // every lane is idle: k = per_warp
      first = false;
      return (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per_warp;
    }
    int base = 0;
    if (lane == leader) base = atomicAdd(q.fetch, k);
    return __shfl_sync(0xffffffffu, base, leader) + grid_warps * per_warp;
  }
  template <bool kAny>
  __device__ __forceinline__ void load(int ray, V3& o, V3& d, float& tmin, float& tmax) const {
    const float4 a = q.ray_o[ray], b = q.ray_d[ray];
    o = v3(a.x, a.y, a.z);
    d = v3(b.x, b.y, b.z);
    if (kAny) { tmin = kShadowEps; tmax = a.w; }
    else { tmin = a.w; tmax = b.w; }
  }
  __device__ __forceinline__ void finish_any(int ray, bool occluded) const {
    if (occluded) return;
    const float4 c = q.contrib[ray];
    const int p = __float_as_int(q.ray_d[ray].w);
    float4 l = q.L[p];
    l.x = l.x + c.x; l.y = l.y + c.y; l.z = l.z + c.z;
    q.L[p] = l;
  }
  __device__ __forceinline__ void finish_closest(const DevScene&, int ray, V3, V3, float, float,
                                                 const HitState& h) const {
    q.hit[ray] = make_float4(h.t, h.u, h.v, __int_as_float(h.prim));
    q.hit_inst[ray] = h.inst;
  }
  __device__ __forceinline__ unsigned long long* stats() const { return q.stats; }
};

// Adds a block's traversal counters to four device totals: one atomic per block and counter. Every
// thread of the block calls it.
__device__ __forceinline__ void flush_counters(unsigned long long* dst, const TraversalCounters& c) {
  __shared__ unsigned long long s_sum[4];
  if (threadIdx.x < 4) s_sum[threadIdx.x] = 0ull;
  __syncthreads();
  const uint32_t v[4] = {c.nodes, c.tris, c.tlas, c.inst};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    // the sums of the 16-bit halves fit 32 bits
    const uint32_t lo = __reduce_add_sync(0xffffffffu, v[k] & 0xffffu), hi = __reduce_add_sync(0xffffffffu, v[k] >> 16);
    if ((threadIdx.x & 31) == 0) atomicAdd(s_sum + k, ((unsigned long long)hi << 16) + lo);
  }
  __syncthreads();
  if (threadIdx.x < 4) atomicAdd(dst + threadIdx.x, s_sum[threadIdx.x]);
}

template <bool kAny, bool kCount, int kSh, class IO>
__device__ __forceinline__ void trace_persistent(const DevScene& sc, IO& io, int refill, bool far_first) {
  constexpr unsigned FULL = 0xffffffffu;
  using Stack = TStack<uint32_t, kSh>;
  const int lane = threadIdx.x & 31;
  // a closest-hit ray's TLAS entries are two words, the entry distance below the entry
  constexpr int kTlasWords = kAny ? 1 : 2;
  uint32_t stack_local[(kTlasWords + 1) * kStackSize];
  extern __shared__ uint32_t s_stack[];
  const Stack stack{s_stack + threadIdx.x, stack_local};
  // What a ray needs only between TLAS and BLAS, at a hit and at its end waits in shared memory.
  enum { W_ORG = 0, W_DIR = 3, W_INV = 6, W_LDIR = 9, W_TMAX = 12, W_U = 13, W_V, W_PRIM, W_INST, W_WORDS };
  __shared__ float s_ray[W_WORDS * kShStride];
  float* const w = s_ray + threadIdx.x;
  auto get3 = [w](int k) { return v3(w[k * kShStride], w[(k + 1) * kShStride], w[(k + 2) * kShStride]); };
  auto put3 = [w](int k, V3 a) { w[k * kShStride] = a.x; w[(k + 1) * kShStride] = a.y; w[(k + 2) * kShStride] = a.z; };
  auto put_hit = [w](float u, float v, int prim, int inst) {
    w[W_U * kShStride] = u; w[W_V * kShStride] = v;
    w[W_PRIM * kShStride] = __int_as_float(prim); w[W_INST * kShStride] = __int_as_float(inst);
  };
  // The TLAS root, read by the launch (which may be part of a captured graph) from where a refit
  // moves it; a copy per warp, for new rays.
  __shared__ float4 s_root[2 * (kShStride / 32)];
  const int warp = threadIdx.x >> 5;
  if (lane < 2 && sc.num_tlas_nodes > 0) s_root[2 * warp + lane] = ldg4(sc.nodes + lane);
  __syncwarp();
  TraversalCounters cnt{0, 0, 0, 0};
  bool overflow = false;

  int ray = -1;                   // queue index of this lane's ray, -1 = idle
  bool exhausted = false;         // the queue has no more rays for this warp
  float tmin = 0.f, t_best = 0.f; // closest hits: the hit's t so far; any hits: the ray's tmax
  SlabRay sr;                     // the ray in the space of the nodes it is among
  sr.set(v3s(0.f), v3s(0.f));
  bool odd = false, world_odd = false, in_blas = false;
  int sp = 0, base = 0;           // stack entries [base, sp) belong to the BLAS (or the TLAS) it is in
  uint32_t cur = kDone;           // the entry to expand; kNoWork: back to the TLAS; kDone: none left
  int cur_inst = -1;
  uint32_t tl_next = 0, tl_end = 0;   // instances left of the current TLAS leaf
  bool occluded = false;

  // what follows the stack's last entry: the TLAS while it holds anything
  auto none = [&]() -> uint32_t { return in_blas && (base > 0 || tl_next != tl_end) ? kNoWork : kDone; };
  auto pop_blas = [&]() -> uint32_t { return sp > base ? stack.get(--sp) : none(); };
  auto pop_tlas = [&]() -> uint32_t {
    while (sp > 0) {
      const uint32_t e = stack.get(--sp);
      if (kAny || __uint_as_float(stack.get(--sp)) <= t_best) return e;
    }
    return kDone;
  };

  // A pair of nodes (tlas.cpp:186-242, blas.cpp:222-263): the near child continues in cur, the far
  // one is pushed. mixed: some lanes are in the TLAS (without: 5 % faster where there is one
  // instance).
  auto step = [&](auto mixed) {
    const bool blas = decltype(mixed)::value ? in_blas : true;
    if (cur < kLeafEntry) {
      if (kCount) {
        if (blas) cnt.nodes++;
        else cnt.tlas += 2;
      }
      const float4* pp = sc.nodes + 2 * (size_t)cur;
      float4 la, lb, ra, rb;
      ldg8(pp, la, lb);
      ldg8(pp + 2, ra, rb);
      uint32_t el = __float_as_uint(lb.z), er = __float_as_uint(rb.z);
      float tl, tr;
      bool hl, hr;
      if (!odd) {
        hl = sr.slab(la, lb, tmin, t_best, tl);
        hr = sr.slab(ra, rb, tmin, t_best, tr);
      } else if (blas) {
        hl = slab_sse(la, lb, sr.inv(), sr.org(), tmin, t_best, tl);
        hr = slab_sse(ra, rb, sr.inv(), sr.org(), tmin, t_best, tr);
      } else {
        hl = aabb_fast(la, lb, sr.inv(), sr.org(), get3(W_DIR), tmin, t_best, tl);
        hr = aabb_fast(ra, rb, sr.inv(), sr.org(), get3(W_DIR), tmin, t_best, tr);
      }
      bool left = (tl < tr) != (kAny && far_first);
      if (!blas) {
        if (!kAny) {
          // the child whose centre comes first along the parent's widest axis
          const bool ay = (el & 1u) != 0, az = (er & 1u) != 0;
          const V3 no = sr.norg(), iv = sr.inv();
          const float o = az ? no.z : (ay ? no.y : no.x), i = az ? iv.z : (ay ? iv.y : iv.x);
          left = (lb.w + o) * i < (rb.w + o) * i;
        }
        if (el < kLeafEntry) el >>= 1;
        if (er < kLeafEntry) er >>= 1;
      }
      if (hl && hr) {
        if (sp - base >= (blas ? kStackSize : kTlasWords * (kStackSize - 1))) {
          overflow = true;
          cur = kDone;            // abandon (reported as overflow)
        } else {
          const uint32_t far = left ? er : el;
          if (!kAny && !blas) stack.put(sp++, __float_as_uint(left ? tr : tl));
          stack.put(sp++, far);
          cur = left ? el : er;
        }
      } else if (hl || hr) {
        cur = hl ? el : er;
      } else {
        cur = blas ? pop_blas() : pop_tlas();
      }
    }
  };

  const unsigned takers = FULL >> (32 - io.lanes());   // the lanes that take rays
  refill = min(refill, io.lanes());
  for (;;) {
    // ── write finished rays' answers and take new ones, several lanes at once ──
    unsigned idle = __ballot_sync(FULL, cur == kDone);
    bool to_top = false;
    if (idle == FULL || (!exhausted && __popc(idle & takers) >= refill)) {
      if (cur == kDone && ray >= 0) {
        if (kAny) io.finish_any(ray, occluded);
        else io.finish_closest(sc, ray, get3(W_ORG), get3(W_DIR), tmin, w[W_TMAX * kShStride],
                               HitState{t_best, w[W_U * kShStride], w[W_V * kShStride],
                                        __float_as_int(w[W_PRIM * kShStride]), __float_as_int(w[W_INST * kShStride])});
        ray = -1;
      }
      if (exhausted) break;
      const unsigned take = idle & takers;
      const int first = io.grab(lane, __ffs(take) - 1, __popc(take));
      if (first >= io.end()) exhausted = true;
      if ((take >> lane) & 1u) {
        const int mine = first + __popc(take & ((1u << lane) - 1u));
        if (mine < io.end()) {
          ray = mine;
          V3 wo, wd;
          float tmax;
          io.template load<kAny>(ray, wo, wd, tmin, tmax);
          const V3 winv = v3(1.f / wd.x, 1.f / wd.y, 1.f / wd.z);
          put3(W_ORG, wo);
          put3(W_DIR, wd);
          put3(W_INV, winv);
          w[W_TMAX * kShStride] = tmax;
          t_best = kAny ? tmax : kInf;
          if (!kAny) put_hit(0.f, 0.f, -1, -1);
          sr.set(wo, winv);
          odd = world_odd = SlabRay::odd(sc, wo, winv, tmin, t_best);
          sp = 0; base = 0; tl_next = 0; tl_end = 0;
          in_blas = false;
          occluded = false;
          if (sc.num_tlas_nodes > 0) {
            if (kCount) cnt.tlas++;
            const float4 root_a = s_root[2 * warp], root_b = s_root[2 * warp + 1];
            odd = world_odd = world_odd || root_b.w != 0.f;
            float tn;
            if (odd ? aabb_fast(root_a, root_b, winv, wo, wd, tmin, t_best, tn)
                    : sr.slab(root_a, root_b, tmin, t_best, tn)) {
              cur = __float_as_uint(root_b.z);
              if (cur < kLeafEntry) cur >>= 1;
            }
          }
        }
      }
      // then the way into an instance, for new rays whose TLAS is one leaf, while they are together
      idle = __ballot_sync(FULL, cur == kDone);
      to_top = true;
    }
    // ── one kind of work for the lanes that are at it: the kind most lanes wait for ──
    const int n_inner = __popc(__ballot_sync(FULL, cur < kLeafEntry));
    const int n_leaf = __popc(__ballot_sync(FULL, in_blas && cur >= kLeafEntry && cur < kDone));
    const int n_top = 32 - n_inner - n_leaf - __popc(idle);
    if (!to_top && n_inner >= n_leaf && n_inner >= n_top) {
      const int keep = max(1, (n_inner + 1) / 2);
      if (__any_sync(FULL, cur < kLeafEntry && !in_blas)) {
        do step(std::true_type{}); while (__popc(__ballot_sync(FULL, cur < kLeafEntry)) >= keep);
      } else {
        do step(std::false_type{}); while (__popc(__ballot_sync(FULL, cur < kLeafEntry)) >= keep);
      }
    } else if (!to_top && n_leaf >= n_top) {
      if (in_blas && cur >= kLeafEntry && cur < kDone) {
        // the leaf's triangles (blas.cpp:224-233 / 281-287)
        uint32_t first, count;
        leaf_unpack(sc, cur, first, count);
        const V3 lo = sr.org(), linv = sr.inv(), ld = get3(W_LDIR);
        for (uint32_t i = 0; i < count; ++i) {
          const float4* tp = sc.tris + 3 * (size_t)(first + i);
          const float4 a = ldg4(tp), b = ldg4(tp + 1), c = ldg4(tp + 2);
          if (kCount) cnt.tris++;
          float t, u, v;
          if (tri_hit(sc, lo, ld, linv, tmin, ld3(a), ld3(b), ld3(c), t_best, t, u, v)) {
            if (kAny) {
              occluded = true;
              break;
            }
            t_best = t;
            put_hit(u, v, (int)(first + i), cur_inst);
          }
        }
        cur = kAny && occluded ? kDone : pop_blas();
      }
    } else if (cur >= kLeafEntry && cur != kDone && (!in_blas || cur == kNoWork)) {
      if (cur == kNoWork && tl_next == tl_end) {
        // back among the TLAS nodes
        in_blas = false;
        base = 0;
        odd = world_odd;
        sr.set(get3(W_ORG), get3(W_INV));
        cur = pop_tlas();
      }
      if (cur >= kLeafEntry && cur < kDone) {
        uint32_t first, count;
        leaf_unpack(sc, cur, first, count, 1);
        tl_next = first;
        tl_end = first + count;
        cur = kNoWork;
      }
      if (cur == kNoWork && tl_next != tl_end) {
        // enter the next instance of the current TLAS leaf (tlas.cpp:200-218)
        const int ii = (int)tl_next++;
        const DevInstance in = load_instance(sc.inst + ii);
        if (kCount) cnt.inst++;
        const Ray lr = to_local(in, Ray{get3(W_ORG), get3(W_DIR), tmin, w[W_TMAX * kShStride]});
        if (in.kind == 0) {
          const V3 linv = v3(1.f / lr.d.x, 1.f / lr.d.y, 1.f / lr.d.z);
          put3(W_LDIR, lr.d);
          sr.set(lr.o, linv);
          odd = SlabRay::odd(sc, lr.o, linv, tmin, t_best);
          in_blas = true;
          base = sp;
          cur_inst = ii;
          cur = in.root;
        } else {
          // analytic prims: a short scalar walk, done in place
          const StackAbove<Stack> above{stack, sp};
          if (kAny) {
            if (pblas_any(sc, lr, above, overflow)) { occluded = true; cur = kDone; }
          } else {
            HitState h{t_best, 0.f, 0.f, -1, -1};
            if (pblas_closest(sc, lr, h, ii, above, overflow)) {
              t_best = h.t;
              put_hit(h.u, h.v, h.prim, h.inst);
            }
          }
        }
      }
    }
  }
  if (overflow) atomicAdd(io.stats() + 3, 1ull);
  if (kCount) flush_counters(io.stats() + (kAny ? 12 : 8), cnt);
}

}  // namespace xbd
