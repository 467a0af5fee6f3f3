// persistent_kernel.cuh -- the whole explicit cycle of a small mesh in one launch.
//
// For a mesh whose element and nodal state fit on the chip (one part of BT shells or of
// hexas), cycle_persistent_kernel runs all the cycles of a step in a
// single cooperative launch of one CTA per SM.  Every CTA keeps its patches' element
// state in registers and all the nodes they touch in shared memory; a node that several
// CTAs hold is updated identically by each of them.  A cycle:
//
//   element phase   the patches' elements, corner forces to shared memory.  The time step
//                   of an element is known before its forces (a shell's from its geometry
//                   alone): each warp hands in its minimum as soon as it has it, and one
//                   thread (of a warp without elements, where there is one, else of the warp
//                   that hands in last) sends the CTA's minimum to the grid and counts the CTA
//                   as arrived, while the elements' arithmetic goes on.
//   shared nodes    partial sums, patch by patch, of the nodes other CTAs hold too, to the
//                   node-major slot skyline; then the node's slots of all CTAs are polled
//                   until they are there, summed (ASSPAR4) and the node updated
//   own nodes       all other nodes: patch partials summed from shared memory in the same
//                   order, then the dt logic, ACCELE, BCS10, VELOCITY, DEPLA (node_update
//                   of the node pass), by other threads at the same time
//
// A slot is its own flag: until its CTA has written it, every word of it holds NO_SLOT, a
// NaN that is never written as a value.  The node phases need no barrier, fence or counter
// then; a CTA's threads meet once after the elements and once after the nodes.  Against a
// second grid counter between the write and the read of the slots (B200): the 200x200 split
// plate 7.3 us a cycle, now 6.75; 22,801 FP64 shells with the Newton return 13.0, now 12.5;
// 40,687 FP64 hexas 20.0, now 19.6; 4,000 FP64 hexas 7.70, now 7.82 (the clearing stores).
//
// With one grid barrier between all elements and all nodes, and every patch partial
// through L2, the split plate took 7.5 us.  Hexas took two launches a cycle: 4,000 in FP64
// 9.9 us; 28,952 in the split form 12.6, with the second counter 9.1.  What is left is
// latency: an element's chain (3.2 us of the split plate's cycle), the assembly from shared
// memory, an L2 round trip for the time step and one for the slots.
//
// Only the shared nodes' slots and the time-step reduction cross between SMs (through
// L2).  The slots are double-buffered by cycle parity, and a CTA clears its slots of the
// other parity when it writes a cycle's: it has passed the cycle's time-step counter, which
// every CTA reaches after it has read the cycle before, and nobody polls them until the next
// one, which this CTA reaches after it has cleared them.  The reduction is triple-buffered:
// a CTA reaches the reuse of a buffer only after a counter that every reader has passed.
// The result is that of the patch and node kernels: the same operations in the same order
// (for hexas in the split form see hex_pair.cuh).  After the last cycle each node's owner
// (the lowest CTA that holds it) writes it back, the element state is written back, and the
// kinetic energy is summed per node tile exactly as the node pass sums it.
//
// The counter and the slots are polled with a time limit: past the limit a CTA sets the
// OR_E_TIMEOUT error word and an abort flag, and every CTA leaves at its next wait, so
// the launch always ends, with nothing written back.
#pragma once
#include "ecycle_kernels.cuh"
#include "hex_pair.cuh"

namespace orb {

// host-built layout of the persistent launch (one part, shell groups or hexa groups only)
struct PersistArgs {
  const int* node_ofs;        // G + 1: CTA c holds nodes node_ofs[c] .. node_ofs[c+1]-1 of the lists below
  const int* node_glob;       // padded global node number of each held node: a CTA's shared nodes, then its own
  const int* node_nshared;    // G: how many of them are shared with other CTAs
  const unsigned char* owner; // 1 where the CTA is the lowest that holds the node
  const unsigned short* pconn;  // per padded element: its 4 or 8 corners' CTA-local node indices
  // Corner lists: held node i of the lists above has the words list[list_ofs[i]] ..
  // list[list_ofs[i+1]-1].  For each patch of the CTA that touches it, in ascending order:
  // slot << 8 | count, then the count corners in ascending (element, corner) order, each
  // as the offset of its first value among the CTA's corner forces.
  const int* list_ofs;
  const int* list;
  void* fslot2;               // second slot buffers (odd cycles); the handle's fslot / mslot serve even ones
  void* mslot2;
  PartAcc* acc3;              // triple-buffered time-step reduction
  double* ek_node;            // last cycle's kinetic energy of every node (owners write)
  double* ekr_node;
  unsigned* sync;             // [0] time-step counter, [1] abort flag, [SYNC_END] counter of the launch's end
  int patches_per_cta;        // P
  int ncmax;                  // node capacity of a CTA (stride of the shared planes)
  int nlist;                  // list capacity of a CTA
  int ntiles_node;            // node tiles of NODE tile size 128 (kinetic energy partials)
  // Test hooks, -1 off: this CTA does not arrive at the first cycle's counter
  // (OR_ECYCLE_TEST_STALL_CTA), or does not write that cycle's slots
  // (OR_ECYCLE_TEST_STALL_SLOTS), so that the others' bounded waits run out.
  int stall_cta, stall_slots;
};
constexpr int SYNC_END = 32, SYNC_WORDS = 64;        // the two counters on lines of their own

// Loads and stores of the slots, which CTAs exchange during the launch: relaxed at GPU
// scope, every word (4 bytes in the split form, 8 in FP64) written and read as a whole
__device__ __forceinline__ float4 ld_slot(const float4* p) {
  float4 v;
  asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ double4 ld_slot(const double4* p) {
  double4 v;
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];"
               : "=d"(v.z) : "l"(reinterpret_cast<const double*>(p) + 2) : "memory");
  v.w = 0.0;
  return v;
}
__device__ __forceinline__ void st_slot(float4* p, float x, float y, float z) {
  asm volatile("st.relaxed.gpu.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(x), "f"(y), "f"(z), "f"(0.f) : "memory");
}
__device__ __forceinline__ void st_slot(double4* p, double x, double y, double z) {
  asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(x), "d"(y) : "memory");
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(reinterpret_cast<double*>(p) + 2), "d"(z) : "memory");
}
// NO_SLOT: all ones.  Arithmetic makes no such NaN but by negating its own, so a NaN force is
// written as another one.
__device__ __forceinline__ float no_slot(float) { return __uint_as_float(0xffffffffu); }
__device__ __forceinline__ double no_slot(double) { return __longlong_as_double(-1ll); }
__device__ __forceinline__ bool is_slot(float x) { return __float_as_uint(x) != 0xffffffffu; }
__device__ __forceinline__ bool is_slot(double x) { return __double_as_longlong(x) != -1ll; }
__device__ __forceinline__ float slot_value(float x) { return is_slot(x) ? x : __uint_as_float(0x7fffffffu); }
__device__ __forceinline__ double slot_value(double x) { return is_slot(x) ? x : __longlong_as_double(0x7fffffffffffffffll); }

// One thread's part of a grid-wide counter.  Arrive: release what the CTA wrote before.
__device__ __forceinline__ void grid_arrive(unsigned* count) {
  __threadfence();
  atomicAdd(count, 1u);
}
// Ends the launch with OR_E_TIMEOUT.  A CTA that leaves on the flag raises nothing of its own.
__device__ __forceinline__ void give_up(unsigned* abort, ErrorWord* err) {
  raise_error(err, 7, (int)blockIdx.x);
  atomicExch(abort, 1u);
}
// Wait until `target` arrivals were counted; true when the launch must end (a CTA gave up)
__device__ __forceinline__ bool grid_wait(unsigned* count, unsigned target, unsigned* abort, ErrorWord* err) {
  const long long t0 = clock64();
  for (;;) {
    if (ld_acquire(count) >= target) return false;  // acquire: every CTA's writes before its arrival
    if (__ldcg(abort)) break;
    if (clock64() - t0 > (1ll << 31)) {             // about a second at the SM clock
      give_up(abort, err);
      break;
    }
    __nanosleep(20);
  }
  __threadfence();
  return true;
}

// pairs of reals for the corner-force planes of the persistent kernel
template <class R> struct Vec2;
template <> struct Vec2<float> { typedef float2 T; };
template <> struct Vec2<double> { typedef double2 T; };
__device__ __forceinline__ float2 mk2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 mk2(double a, double b) { return make_double2(a, b); }

// the two energy sums of a group of NT threads (threads g*NT .. g*NT+NT-1), with the
// operation order of block_reduce
template <int NT>
__device__ inline void group_sums(double& s0, double& s1, double* ss0, double* ss1) {
  const int lt = threadIdx.x % NT;
  const int lane = lt & 31, warp = lt >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
  }
  if (lane == 0) { ss0[warp] = s0; ss1[warp] = s1; }
  __syncthreads();
  if (warp == 0) {
    constexpr int NW = NT / 32;
    s0 = lane < NW ? ss0[lane] : 0.0;
    s1 = lane < NW ? ss1[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s0 += __shfl_xor_sync(0xffffffffu, s0, o);
      s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    }
  }
}

// Threads per CTA: at least one per element (per pair of hexas in the split form), raised
// to cover the CTA's held nodes (one per node in the node phases) and a warp without
// elements, and at most PERSIST_THREADS; one CTA per SM.  The threads beyond the elements'
// work on the time step and the nodes only.  MAXT is the thread count that a kernel's
// register budget is for: PERSIST_THREADS (168 registers), or 256 (255), where FP64
// elements spill less.
constexpr int PERSIST_THREADS = 384;
constexpr int persist_maxt(int threads, bool fp64) { return fp64 && threads <= 256 ? 256 : PERSIST_THREADS; }

// ---- the elements of a thread -------------------------------------------------
// Kind: NODE_R, reals per held node beside the coordinates; C, force components per
// corner; TILE elements and NT threads per patch; CORNER_R, reals of corner forces per
// patch, and STATE_R, of element state kept in shared memory.  element() evaluates the thread's elements into the corner forces, corner() reads
// one corner back.

// one shell; corner forces and moments as three planes of pairs (fx fy | fz mx | my mz),
// corner k of element t at pair k * TILE + t.  In FP64 the integration points' state (60
// registers for 5 points) is kept in shared planes instead of registers, which spilled:
// the 200x200 plate 18.9 -> 16.1 us a cycle together with the single node update below.
// Where the planes do not fit (six patches of 64 a CTA), 5 points of Ishell 1 stay in
// registers (REGS): 47,961 shells 20.6 us a cycle, 24.7 with the state read from memory.
template <class R, int TILE_, int NPT, bool GEN, bool REGS = false>
struct PersistShell {
  typedef ShellArgs<R> Args;
  typedef typename Vec2<R>::T R2;
  static constexpr bool KEEP = NPT > 0, PLANES = KEEP && sizeof(R) == 8 && !REGS;
  static constexpr int TILE = TILE_, NT = TILE, C = 6, NODE_R = 8, CORNER_R = 24 * TILE,
                       STATE_R = PLANES ? 6 * NPT * TILE : 0;
  ShellState<R, NPT> st;
  int lc[4], e, lt;
  ShellGroupDesc gd;
  const float* zw;
  R* sc;                        // the patch's corner forces
  R* sp;                        // PLANES: this thread's entry of the patch's state planes
  __device__ __forceinline__ bool load(const Args& a, const PersistArgs& pa, const float* z, int p, bool has, int t, R* c,
                                       R* state) {
    zw = z; sc = c; sp = state + t; lt = t; e = (has ? p : 0) * TILE + t;
    if (KEEP) shell_load_state<R, NPT, !PLANES>(a, e, st);
    if constexpr (PLANES) {
      if (has) {
#pragma unroll 5
        for (int q = 0; q < 5 * NPT; ++q) sp[q * TILE] = a.sig[q * a.nelpad + e];
#pragma unroll
        for (int ip = 0; ip < NPT; ++ip) sp[(5 * NPT + ip) * TILE] = a.pla[ip * a.nelpad + e];
      }
    }
    const uint2 w = reinterpret_cast<const uint2*>(pa.pconn)[e];
    lc[0] = w.x & 0xffffu; lc[1] = w.x >> 16; lc[2] = w.y & 0xffffu; lc[3] = w.y >> 16;
    gd = a.groups[has ? a.patch[p].group : 0];
    return has && t < a.patch[p].nel;
  }
  template <class Early>
  __device__ __forceinline__ void element(const Args& a, const R DT1, const double* sx, const double* sy,
                                          const double* sz, const R* sv, const int NC, const Early& early,
                                          double& ehou, double& wpla) {
    R Fg[3][4], Mg[3][4];
    unsigned long long key = ~0ull, bits = ~0ull;
    double h = 0.0, w = 0.0;
    if (!KEEP) shell_load_state<R, NPT>(a, e, st);
    const ShellNodePlanes<R> nd{sx, sy, sz, sv, NC, lc};
    shell_element<R, NPT, KEEP, PLANES, GEN>(a, e, gd, DT1, zw, nd, st, Fg, Mg, key, bits, h, w, sp, TILE, early);
    R2* q = reinterpret_cast<R2*>(sc);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      q[(0 * 4 + k) * TILE + lt] = mk2(Fg[0][k], Fg[1][k]);
      q[(1 * 4 + k) * TILE + lt] = mk2(Fg[2][k], Mg[0][k]);
      q[(2 * 4 + k) * TILE + lt] = mk2(Mg[1][k], Mg[2][k]);
    }
    ehou += h;
    wpla += w;
  }
  static __device__ __forceinline__ void corner(const R* all, int o, R (&f)[C]) {
    const R2* q = reinterpret_cast<const R2*>(all);
    const R2 p0 = q[o], p1 = q[4 * TILE + o], p2 = q[8 * TILE + o];
    f[0] += p0.x; f[1] += p0.y; f[2] += p1.x; f[3] += p1.y; f[4] += p2.x; f[5] += p2.y;
  }
  __device__ __forceinline__ void store(const Args& a, bool has) const {
    if (!has) return;
    if constexpr (KEEP) shell_store_state<R, NPT, !PLANES>(a, e, st);
    if constexpr (PLANES) {
#pragma unroll 5
      for (int q = 0; q < 5 * NPT; ++q) a.sig[q * a.nelpad + e] = sp[q * TILE];
#pragma unroll
      for (int ip = 0; ip < NPT; ++ip) a.pla[ip * a.nelpad + e] = sp[(5 * NPT + ip) * TILE];
    }
  }
};

// two hexas in the split form (hex_pair.cuh); corner forces in three planes of TILE x 8,
// corner k of element t at k * TILE + t
template <int TILE_, int CORO>
struct PersistHexPair {
  typedef float R;
  typedef HexArgs<R> Args;
  typedef Pair K;
  typedef F2 W;
  static constexpr int N = K::N, TILE = TILE_, NT = TILE / N, C = 3, NODE_R = 5, CORNER_R = 24 * TILE, STATE_R = 0;
  W sig_[6], eint_, rho_, qvis_, vol0_, pla_, epsd_;
  double v0_[N];
  int eid_[N], lc[N][8], e, t0;
  bool act[N];
  HexGroupDesc gd;
  R* sc;
  __device__ __forceinline__ bool load(const Args& a, const PersistArgs& pa, const float*, int p, bool has, int t, R* c,
                                       R*) {
    sc = c; t0 = N * t; e = (has ? p : 0) * TILE + t0;
    const int nel = has ? a.patch[p].nel : 0;
    auto ld = [&](const R* q) { return K::map([&](int i) { return q[e + i]; }); };
#pragma unroll
    for (int k = 0; k < 6; ++k) sig_[k] = ld(a.sig + (size_t)k * a.nelpad);
    eint_ = ld(a.eint); rho_ = ld(a.rho); qvis_ = ld(a.qvis); vol0_ = ld(a.vol0); pla_ = ld(a.pla); epsd_ = ld(a.epsd);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      act[i] = t0 + i < nel;
      eid_[i] = a.elem_id[e + i];
      v0_[i] = a.vol0dp[e + i];
      const uint4 w = reinterpret_cast<const uint4*>(pa.pconn)[e + i];
      const unsigned q[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int k = 0; k < 8; ++k) lc[i][k] = (q[k / 2] >> (16 * (k & 1))) & 0xffffu;
    }
    gd = a.groups[has ? a.patch[p].group : 0];
    return act[0];
  }
  // what hex_element asks for
  template <class Early>
  struct IO {
    PersistHexPair& h;
    const double *sx, *sy, *sz;
    const R* sv;
    const int NC;
    const Early& hand_in;
    __device__ __forceinline__ void x(int i, int k, double (&o)[3]) const {
      const int l = h.lc[i][k];
      o[0] = sx[l]; o[1] = sy[l]; o[2] = sz[l];
    }
    __device__ __forceinline__ void v(int i, int k, R (&o)[3]) const {
      const int l = h.lc[i][k];
      o[0] = sv[l]; o[1] = sv[NC + l]; o[2] = sv[2 * NC + l];
    }
    __device__ __forceinline__ int eid(int i) const { return h.eid_[i]; }
    __device__ __forceinline__ double vol0dp(int i) const { return h.v0_[i]; }
    __device__ __forceinline__ W sig(int c) const { return h.sig_[c]; }
    __device__ __forceinline__ W eint() const { return h.eint_; }
    __device__ __forceinline__ W rho() const { return h.rho_; }
    __device__ __forceinline__ W qvis() const { return h.qvis_; }
    __device__ __forceinline__ W vol0() const { return h.vol0_; }
    __device__ __forceinline__ W pla() const { return h.pla_; }
    __device__ __forceinline__ void put_sig(int c, W a) const { h.sig_[c] = a; }
    __device__ __forceinline__ void put_eint(W a) const { h.eint_ = a; }
    __device__ __forceinline__ void put_rho(W a) const { h.rho_ = a; }
    __device__ __forceinline__ void put_qvis(W a) const { h.qvis_ = a; }
    __device__ __forceinline__ void put_pla(W a) const { h.pla_ = a; }
    __device__ __forceinline__ void put_epsd(W a) const { h.epsd_ = a; }
    __device__ __forceinline__ void early(unsigned long long k, unsigned long long b) const { hand_in(k, b); }
    __device__ __forceinline__ void corner(int k, const W (&f)[3]) const {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        R* q = h.sc + (8 * c + k) * TILE + h.t0;
        *reinterpret_cast<float2*>(q) = make_float2(f2_get(f[c], 0), f2_get(f[c], 1));
      }
    }
  };
  template <class Early>
  __device__ __forceinline__ void element(const Args& a, const R DT1, const double* sx, const double* sy,
                                          const double* sz, const R* sv, const int NC, const Early& early,
                                          double& ehou, double& wpla) {
    IO<Early> io{*this, sx, sy, sz, sv, NC, early};
    hex_pair<CORO>(gd, act, DT1, io, a.err, ehou, wpla);
  }
  static __device__ __forceinline__ void corner(const R* all, int o, R (&f)[C]) {
    f[0] += all[o]; f[1] += all[8 * TILE + o]; f[2] += all[16 * TILE + o];
  }
  __device__ __forceinline__ void store(const Args& a, bool has) const {
    if (!has) return;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (!act[i]) continue;
#pragma unroll
      for (int c = 0; c < 6; ++c) a.sig[(size_t)c * a.nelpad + e + i] = K::get(sig_[c], i);
      a.eint[e + i] = K::get(eint_, i);
      a.rho[e + i] = K::get(rho_, i);
      a.qvis[e + i] = K::get(qvis_, i);
      a.pla[e + i] = K::get(pla_, i);
      a.epsd[e + i] = K::get(epsd_, i);
    }
  }
};

// one FP64 hexa (hex_element), corner forces as above
template <int TILE_, int CORO>
struct PersistHexa {
  typedef double R;
  typedef HexArgs<R> Args;
  static constexpr int TILE = TILE_, NT = TILE, C = 3, NODE_R = 5, CORNER_R = 24 * TILE, STATE_R = 0;
  R sig_[6], eint_, rho_, qvis_, vol0_, pla_, epsd_;
  int eid_, lc[8], e, t;
  HexGroupDesc gd;
  R* sc;
  __device__ __forceinline__ bool load(const Args& a, const PersistArgs& pa, const float*, int p, bool has, int lt, R* c,
                                       R*) {
    sc = c; t = lt; e = (has ? p : 0) * TILE + t;
#pragma unroll
    for (int k = 0; k < 6; ++k) sig_[k] = a.sig[(size_t)k * a.nelpad + e];
    eint_ = a.eint[e]; rho_ = a.rho[e]; qvis_ = a.qvis[e]; vol0_ = a.vol0[e]; pla_ = a.pla[e]; epsd_ = a.epsd[e];
    eid_ = a.elem_id[e];
    const uint4 w = reinterpret_cast<const uint4*>(pa.pconn)[e];
    const unsigned q[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int k = 0; k < 8; ++k) lc[k] = (q[k / 2] >> (16 * (k & 1))) & 0xffffu;
    gd = a.groups[has ? a.patch[p].group : 0];
    return has && t < a.patch[p].nel;
  }
  // what hex_element asks for
  template <class Early>
  struct IO {
    PersistHexa& h;
    R (&held)[24];
    const double *sx, *sy, *sz;
    const R* sv;
    const int NC;
    const Early& hand_in;
    __device__ __forceinline__ void x(int k, double& x, double& y, double& z) const {
      const int l = h.lc[k];
      x = sx[l]; y = sy[l]; z = sz[l];
    }
    __device__ __forceinline__ double4 v(int k) const {
      const int l = h.lc[k];
      return make_double4(sv[l], sv[NC + l], sv[2 * NC + l], 0.0);
    }
    __device__ __forceinline__ int eid() const { return h.eid_; }
    __device__ __forceinline__ double vol0dp() const { return h.vol0_; }
    __device__ __forceinline__ R sig(int c) const { return h.sig_[c]; }
    __device__ __forceinline__ R eint() const { return h.eint_; }
    __device__ __forceinline__ R rho() const { return h.rho_; }
    __device__ __forceinline__ R qvis() const { return h.qvis_; }
    __device__ __forceinline__ R vol0() const { return h.vol0_; }
    __device__ __forceinline__ R pla() const { return h.pla_; }
    __device__ __forceinline__ void put_sig(int c, R v) const { h.sig_[c] = v; }
    __device__ __forceinline__ void put_eint(R v) const { h.eint_ = v; }
    __device__ __forceinline__ void put_rho(R v) const { h.rho_ = v; }
    __device__ __forceinline__ void put_qvis(R v) const { h.qvis_ = v; }
    __device__ __forceinline__ void put_pla(R v) const { h.pla_ = v; }
    __device__ __forceinline__ void put_epsd(R v) const { h.epsd_ = v; }
    __device__ __forceinline__ void early(unsigned long long k, unsigned long long b) const { hand_in(k, b); }
    __device__ __forceinline__ void park(int q, R v) const { held[q] = v; }
    __device__ __forceinline__ R unpark(int q) const { return held[q]; }
    __device__ __forceinline__ void corner(int k, R fx, R fy, R fz) const {
      h.sc[k * TILE + h.t] = fx; h.sc[(8 + k) * TILE + h.t] = fy; h.sc[(16 + k) * TILE + h.t] = fz;
    }
  };
  template <class Early>
  __device__ __forceinline__ void element(const Args& a, const R DT1, const double* sx, const double* sy,
                                          const double* sz, const R* sv, const int NC, const Early& early,
                                          double& ehou, double& wpla) {
    R held[24];
    const IO<Early> io{*this, held, sx, sy, sz, sv, NC, early};
    unsigned long long key = ~0ull, bits = ~0ull;
    double h = 0.0, w = 0.0;
    hex_element<R, CORO>(gd, DT1, io, a.err, key, bits, h, w);
    ehou += h;
    wpla += w;
  }
  static __device__ __forceinline__ void corner(const R* all, int o, R (&f)[C]) {
    f[0] += all[o]; f[1] += all[8 * TILE + o]; f[2] += all[16 * TILE + o];
  }
  __device__ __forceinline__ void store(const Args& a, bool has) const {
    if (!has) return;
#pragma unroll
    for (int c = 0; c < 6; ++c) a.sig[(size_t)c * a.nelpad + e] = sig_[c];
    a.eint[e] = eint_; a.rho[e] = rho_; a.qvis[e] = qvis_; a.pla[e] = pla_; a.epsd[e] = epsd_;
  }
};

// Shared memory: node planes x y z dx dy dz (FP64) and NODE_R of R (velocities, mass, with
// rotations also those and the inertia), global index (int), owner and code (bytes); per
// patch its corner forces and state planes; per held node its list range and slot range (int2); the lists
template <class R>
inline size_t persist_smem(int node_r, int patch_r, int ncmax, int P, int nlist) {
  const size_t nodes = (size_t)ncmax * (6 * sizeof(double) + node_r * sizeof(R) + sizeof(int) + 2);
  return (nodes + 15) / 16 * 16 + (size_t)P * patch_r * sizeof(R) +      // patch_r: CORNER_R + STATE_R
         2 * (size_t)ncmax * sizeof(int2) + (size_t)nlist * sizeof(int);
}

template <class Kind, class R, int MAXT>
__global__ void __launch_bounds__(MAXT, 1)
cycle_persistent_kernel(typename Kind::Args a, NodeArgs<R> na, PersistArgs pa, int ncycles, int parity0,
                        const float* __restrict__ zw) {
  typedef typename Vec4<R>::T R4;
  constexpr int NT = Kind::NT, C = Kind::C;
  constexpr bool ROT = C == 6;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_abort;
  __shared__ double s_e0[PERSIST_THREADS / 32], s_e1[PERSIST_THREADS / 32];
  __shared__ unsigned long long s_dt[2];        // the CTA's dt key and dt bits minimum of a cycle
  __shared__ PartAcc s_acc;                     // the grid's
  __shared__ __align__(8) unsigned long long s_dtbar;
  __shared__ int s_handed;                      // warps that have handed in, without a spare warp
  const int tid = threadIdx.x;
  const int cta = blockIdx.x, G = gridDim.x;
  const int P = pa.patches_per_cta, NC = pa.ncmax;
  const int sub = tid / NT, lt = tid % NT;
  // ---- shared layout ----
  double* sx = reinterpret_cast<double*>(smem_raw);
  double* sy = sx + NC;
  double* sz = sy + NC;
  double* sdx = sz + NC;
  double* sdy = sdx + NC;
  double* sdz = sdy + NC;
  R* sv = reinterpret_cast<R*>(sdz + NC);      // vx vy vz [rx ry rz] planes of NC
  R* sms = sv + C * NC;
  R* sin_ = sms + NC;                          // ROT: inertia; else the spare fifth plane
  int* sglob = reinterpret_cast<int*>(sv + (size_t)Kind::NODE_R * NC);
  unsigned char* sown = reinterpret_cast<unsigned char*>(sglob + NC);
  unsigned char* scode = sown + NC;
  const size_t nodes = (size_t)NC * (6 * sizeof(double) + Kind::NODE_R * sizeof(R) + sizeof(int) + 2);
  R* sc_all = reinterpret_cast<R*>(smem_raw + (nodes + 15) / 16 * 16);     // corner forces, patch after patch
  R* sp_all = sc_all + (size_t)P * Kind::CORNER_R;                         // state planes, patch after patch
  int2* slist = reinterpret_cast<int2*>(sp_all + (size_t)P * Kind::STATE_R);   // list ranges
  int2* srange = slist + NC;                                                   // slot ranges
  int* swords = reinterpret_cast<int*>(srange + NC);

  // ---- this CTA's patch and elements ----
  const int p = cta * P + sub;
  const bool has_patch = sub < P && p < a.npatch;
  Kind el;
  const bool active = el.load(a, pa, zw, p, has_patch, lt, sc_all + (size_t)sub * Kind::CORNER_R,
                              sp_all + (size_t)sub * Kind::STATE_R);
  const unsigned lanes = __ballot_sync(0xffffffffu, active);      // of this warp, with elements
  // ---- stage the held nodes and their lists ----
  const int n0 = pa.node_ofs[cta], nn = pa.node_ofs[cta + 1] - n0;
  const int nsh = pa.node_nshared[cta];
  const int w0 = pa.list_ofs[n0], nw = pa.list_ofs[n0 + nn] - w0;
  for (int i = tid; i < nn; i += blockDim.x) {
    const int g = pa.node_glob[n0 + i];
    const double4 xx = na.X[g];
    const R4 vv = na.V[g];
    sx[i] = xx.x; sy[i] = xx.y; sz[i] = xx.z;
    sdx[i] = na.DX[g]; sdy[i] = na.DY[g]; sdz[i] = na.DZ[g];
    sv[0 * NC + i] = vv.x; sv[1 * NC + i] = vv.y; sv[2 * NC + i] = vv.z;
    if constexpr (ROT) {
      const R4 rr = na.VR[g];
      sv[3 * NC + i] = rr.x; sv[4 * NC + i] = rr.y; sv[5 * NC + i] = rr.z;
      sin_[i] = rr.w;
    }
    sms[i] = R(xx.w);
    sglob[i] = g;
    sown[i] = pa.owner[n0 + i];
    scode[i] = na.code[g];
    srange[i] = make_int2(na.adsky[g], na.adsky[g + 1]);
    slist[i] = make_int2(pa.list_ofs[n0 + i] - w0, pa.list_ofs[n0 + i + 1] - w0);
  }
  for (int i = tid; i < nw; i += blockDim.x) swords[i] = pa.list[w0 + i];
  // the thread that carries the CTA's time step to the grid and waits for the others': of
  // the last warp, idle in the element phase.  If all warps have elements (six patches of 64
  // shells), the one that hands in last sends it on the way, and the first thread waits after
  // its elements; when that thread sent it too, 47,961 split shells took 9.7 us a cycle, so 8.5.
  // The kernels for 256 threads always have the warp, but with one patch of 256.
  const bool spare = (MAXT < PERSIST_THREADS && NT < MAXT) || (int)blockDim.x > P * NT;
  const bool courier = tid == (spare ? (int)blockDim.x - 32 : 0);
  const bool reports = tid < P * NT;               // in a warp that hands in a minimum (an empty one too)
  // Energies: each thread adds its elements' hourglass energy and plastic work over
  // the launch's cycles; the patch sums them once at the end onto its cumulative
  // partials (the phase kernels sum per cycle, so the two agree to FP64 rounding).
  double cum_ehou_t = 0.0, cum_wpla_t = 0.0;
  if (tid == 0) {
    s_dt[0] = ~0ull; s_dt[1] = ~0ull;
    s_abort = 0;
    s_handed = 0;
    mbar_init_n(&s_dtbar, (unsigned)(P * NT / 32));
  }
  PartTime t = na.time[parity0];
  R4* fs[2] = {a.fslot, reinterpret_cast<R4*>(pa.fslot2)};
  R4* ms_[2] = {const_cast<R4*>(na.mslot), reinterpret_cast<R4*>(pa.mslot2)};
  unsigned* const abort = pa.sync + 1;
  // the slots this CTA writes, in both buffers
  for (int i = tid; i < nsh; i += blockDim.x) {
    const int first = pa.list_ofs[n0 + i], end = pa.list_ofs[n0 + i + 1];
    for (int w = first; w < end; w += 1 + (pa.list[w] & 0xff)) {
      const int s = pa.list[w] >> 8;
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        st_slot(&fs[b][s], no_slot(R(0)), no_slot(R(0)), no_slot(R(0)));
        if constexpr (ROT) st_slot(&ms_[b][s], no_slot(R(0)), no_slot(R(0)), no_slot(R(0)));
      }
    }
  }
  __syncthreads();

  // one patch's partial of a node: its corners from word w on; returns its slot
  auto partial = [&](int& w, R (&f)[C]) {
    const int head = swords[w++];
#pragma unroll
    for (int q = 0; q < C; ++q) f[q] = R(0);
    const int end = w + (head & 0xff);
#pragma unroll 4
    for (; w < end; ++w) Kind::corner(sc_all, swords[w], f);
    return head >> 8;
  };

  for (int c = 0; c < ncycles; ++c) {
    R4 *fslot = fs[c & 1], *mslot = ms_[c & 1];
    R4 *fclear = fs[1 - (c & 1)], *mclear = ms_[1 - (c & 1)];
    // ---------------- element phase ----------------
    PartAcc* const acc = &pa.acc3[c % 3];
    auto send = [&]() {                // the CTA's minimum to the grid, and its arrival
      atomicMin(&acc->dtkey, s_dt[0]);
      atomicMin(&acc->dtbits, s_dt[1]);
      s_dt[0] = ~0ull; s_dt[1] = ~0ull;        // no warp touches them again in this cycle
      if (!(c == 0 && cta == pa.stall_cta)) grid_arrive(&pa.sync[0]);
    };
    auto handed_in = [&]() {           // one thread of a warp, after the warp's minimum
      if (spare) { mbar_arrive(&s_dtbar); return; }
      __threadfence_block();
      if (atomicAdd(&s_handed, 1) != P * NT / 32 - 1) return;
      __threadfence_block();
      s_handed = 0;
      send();
    };
    if (active) {
      auto early = [&](unsigned long long key, unsigned long long bits) {
        const unsigned long long wk = warp_min_u64(key, lanes), wb = warp_min_u64(bits, lanes);
        if ((tid & 31) == __ffs(lanes) - 1) {
          atomicMin(&s_dt[0], wk);
          atomicMin(&s_dt[1], wb);
          handed_in();
        }
      };
      el.element(a, R(t.dt2), sx, sy, sz, sv, NC, early, cum_ehou_t, cum_wpla_t);
    } else if (reports && lanes == 0 && (tid & 31) == 0) {
      handed_in();                       // a warp without elements
    }
    if (courier) {
      bool out = false;
      if (spare) {
        out = !mbar_wait(&s_dtbar, c & 1, STAGE_WAIT_TRIES);
        if (out) give_up(abort, a.err);
        send();
      }
      out = out || grid_wait(&pa.sync[0], (unsigned)(c + 1) * (unsigned)G, abort, a.err);
      s_acc.dtkey = __ldcg(&acc->dtkey);
      s_acc.dtbits = __ldcg(&acc->dtbits);
      if (cta == 0) {      // every CTA arrived here, so all have read the last cycle's: its buffer is cycle c + 2's
        PartAcc r; r.dtkey = ~0ull; r.dtbits = ~0ull;
        pa.acc3[(c + 2) % 3] = r;
      }
      if (out) s_abort = 1;
    }
    __syncthreads();
    if (s_abort) return;
    // ---------------- nodes ----------------
    int ityp, nelt;
    double DT2;
    cycle_dt(s_acc, t, na.growth, na.dtmx, na.split, DT2, ityp, nelt);
    const double DTc1 = t.dt2;
    const double DT12 = 0.5 * (DTc1 + DT2);
    const bool last = c == ncycles - 1;
    auto update = [&](const int i, const R (&f)[C]) {
      const int g = sglob[i];
      double px = sx[i], py = sy[i], pz = sz[i], qx = sdx[i], qy = sdy[i], qz = sdz[i];
      R4 v = mk4(sv[0 * NC + i], sv[1 * NC + i], sv[2 * NC + i], R(0)), w = mk4(R(0), R(0), R(0), R(0));
      R r[3] = {R(0), R(0), R(0)};
      if constexpr (ROT) {
        w = mk4(sv[3 * NC + i], sv[4 * NC + i], sv[5 * NC + i], sin_[i]);
        r[0] = f[3]; r[1] = f[4]; r[2] = f[5];
      }
      double ek = 0.0, ekr = 0.0;
      node_update<R>(na, g, scode[i], ROT, f[0], f[1], f[2], r[0], r[1], r[2], sms[i], DTc1, DT2, DT12, px, py, pz, qx,
                     qy, qz, v, w, ek, ekr, last);        // only the launch's last cycle reports kinetic energy
      sx[i] = px; sy[i] = py; sz[i] = pz; sdx[i] = qx; sdy[i] = qy; sdz[i] = qz;
      sv[0 * NC + i] = v.x; sv[1 * NC + i] = v.y; sv[2 * NC + i] = v.z;
      if constexpr (ROT) { sv[3 * NC + i] = w.x; sv[4 * NC + i] = w.y; sv[5 * NC + i] = w.z; }
      if (last && sown[i]) { pa.ek_node[g] = ek; pa.ekr_node[g] = ekr; }
    };
    // shared nodes: this CTA's patch partials to their slots, and the next cycle's cleared
    const int nwrite = c == 0 && cta == pa.stall_slots ? 0 : nsh;
    for (int i = tid; i < nwrite; i += blockDim.x) {
      const int2 lr = slist[i];
      for (int w = lr.x; w < lr.y;) {
        R f[C];
        const int s = partial(w, f);
        st_slot(&fslot[s], slot_value(f[0]), slot_value(f[1]), slot_value(f[2]));
        if constexpr (ROT) st_slot(&mslot[s], slot_value(f[3]), slot_value(f[4]), slot_value(f[5]));
        st_slot(&fclear[s], no_slot(R(0)), no_slot(R(0)), no_slot(R(0)));
        if constexpr (ROT) st_slot(&mclear[s], no_slot(R(0)), no_slot(R(0)), no_slot(R(0)));
      }
    }
    // the CTA's own nodes, by the threads from the last down, then the shared ones by the
    // threads from the first up, so that few have one of each.  For shells one loop, so that
    // the node update is in the kernel once: in FP64 they spill less for it.  Hexas do not,
    // and ran 5 % faster with the two apart.  Four slots are polled at a time (FP64 shells
    // two, for their registers): two ran the 4,000 hexas in 8.47 us a cycle, eight in 7.94.
#pragma unroll (ROT ? 1 : 2)
    for (int shared = 0; shared < 2; ++shared) {
      const int last_node = shared ? nsh - 1 : nn - 1, first_node = shared ? 0 : nsh;
      const int i0 = shared ? tid : last_node - (int)(blockDim.x - 1 - tid);
      const int dir = shared ? (int)blockDim.x : -(int)blockDim.x;
      for (int i = i0; i >= first_node && i <= last_node; i += dir) {
        R f[C];
#pragma unroll
        for (int q = 0; q < C; ++q) f[q] = R(0);
        if (!shared) {
          const int2 lr = slist[i];
          for (int w = lr.x; w < lr.y;) {
            R h[C];
            const bool first = w == lr.x;
            partial(w, h);
#pragma unroll
            for (int q = 0; q < C; ++q) f[q] = first ? h[q] : f[q] + h[q];
          }
        } else {
          // ASSPAR4: the node's slots in ascending patch order, U at a time
          constexpr int U = ROT && sizeof(R) == 8 ? 2 : 4;
          const int2 rg = srange[i];
          for (int k = rg.x; k < rg.y; k += U) {
            R4 F[U], M[U];
            long long t0 = 0;
            for (int tries = 0;; ++tries) {
              bool all = true;
#pragma unroll
              for (int u = 0; u < U; ++u)
                if (k + u < rg.y) {
                  F[u] = ld_slot(&fslot[k + u]);
                  if constexpr (ROT) M[u] = ld_slot(&mslot[k + u]);
                }
#pragma unroll
              for (int u = 0; u < U; ++u)
                if (k + u < rg.y) {
                  all = all && is_slot(F[u].x) && is_slot(F[u].y) && is_slot(F[u].z);
                  if constexpr (ROT) all = all && is_slot(M[u].x) && is_slot(M[u].y) && is_slot(M[u].z);
                }
              if (all) break;
              if ((tries & 63) == 63) {
                if (!t0) t0 = clock64();
                const bool late = clock64() - t0 > (1ll << 31);       // about a second at the SM clock
                if (late) give_up(abort, a.err);
                if (late || __ldcg(abort)) {
                  // zeros for the slots that did not come: their NaN would raise OR_E_NAN
#pragma unroll
                  for (int u = 0; u < U; ++u) {
                    F[u] = mk4(R(0), R(0), R(0), R(0));
                    if constexpr (ROT) M[u] = F[u];
                  }
                  s_abort = 1;
                  break;
                }
              }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
              if (k + u >= rg.y) break;
              const bool first = k + u == rg.x;
              f[0] = first ? F[u].x : f[0] + F[u].x; f[1] = first ? F[u].y : f[1] + F[u].y;
              f[2] = first ? F[u].z : f[2] + F[u].z;
              if constexpr (ROT) {
                f[3] = first ? M[u].x : f[3] + M[u].x; f[4] = first ? M[u].y : f[4] + M[u].y;
                f[5] = first ? M[u].z : f[5] + M[u].z;
              }
            }
          }
        }
        update(i, f);
      }
    }
    t.tt = t.tt + DT2; t.dt2 = DT2; t.dt2old = DT2; t.dt1 = DTc1; t.dt12 = DT12;
    t.ncycle = t.ncycle + 1; t.ityptst = ityp; t.neltst = nelt; t.pad = 0;
    __syncthreads();
    if (s_abort) return;
  }

  // ---- write back: held nodes by their owner, element state, energies, time ----
  for (int i = tid; i < nn; i += blockDim.x) {
    if (!sown[i]) continue;
    const int g = sglob[i];
    na.X[g] = make_double4(sx[i], sy[i], sz[i], na.X[g].w);
    na.DX[g] = sdx[i]; na.DY[g] = sdy[i]; na.DZ[g] = sdz[i];
    na.V[g] = mk4(sv[0 * NC + i], sv[1 * NC + i], sv[2 * NC + i], R(0));
    if constexpr (ROT) na.VR[g] = mk4(sv[3 * NC + i], sv[4 * NC + i], sv[5 * NC + i], sin_[i]);
  }
  el.store(a, has_patch);
  {   // the group's sums, through the corner forces' memory (read for the last time above)
    double* s_sum = reinterpret_cast<double*>(sc_all) + 2 * (size_t)sub * (NT / 32);
    group_sums<NT>(cum_ehou_t, cum_wpla_t, s_sum, s_sum + NT / 32);
    if (has_patch && lt == 0) {
      a.blk_ehour[p] = a.blk_ehour[p] + cum_ehou_t;
      a.blk_wpla[p] = a.blk_wpla[p] + cum_wpla_t;
    }
  }
  if (cta == 0 && tid == 0) {
    const int fin = (parity0 + ncycles) & 1;
    na.time[fin] = t;
    PartAcc r; r.dtkey = ~0ull; r.dtbits = ~0ull;
    a.acc[fin] = r;
  }
  // kinetic energy per node tile of 128, summed as the node pass sums it
  __syncthreads();
  if (tid == 0) {
    grid_arrive(pa.sync + SYNC_END);
    if (grid_wait(pa.sync + SYNC_END, (unsigned)G, abort, a.err)) s_abort = 1;
  }
  __syncthreads();
  if (s_abort) return;
  for (int tile = cta; tile < pa.ntiles_node; tile += G) {
    double ek = 0.0, ekr = 0.0;
    if (tid < 128) {
      ek = __ldcg(&pa.ek_node[tile * 128 + tid]);
      ekr = __ldcg(&pa.ekr_node[tile * 128 + tid]);
    }
    const int lane = tid & 31, warp = tid >> 5;
    if (tid < 128) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        ek += __shfl_xor_sync(0xffffffffu, ek, o);
        ekr += __shfl_xor_sync(0xffffffffu, ekr, o);
      }
      if (lane == 0) { s_e0[warp] = ek; s_e1[warp] = ekr; }
    }
    __syncthreads();
    if (tid == 0) {
      double s0 = 0.0, s1 = 0.0;
      for (int w = 0; w < 4; ++w) { s0 += s_e0[w]; s1 += s_e1[w]; }
      na.blk_ekin[tile] = s0;
      na.blk_ekinr[tile] = s1;
    }
    __syncthreads();
  }
}

}  // namespace orb
