// On-chip relaxation: whole RK4 steps of one or more grids in one cooperative
// launch, for grids whose state fits in the GPU's registers and shared memory.
//
// The substep kernels (kernels_fused.cu, kernels_march.cu) end every RK4
// substep with a kernel boundary and read every pointwise field from L2 again:
// 6.5 us per substep at 64x64x8 and 10 us at 128x128x16, of which the FP64
// arithmetic needs 0.15 and 1.2 us.  Here a block owns a tile of (i0,i1)
// columns with all their i2 planes for the whole launch:
//   * y_n, the running total and vv of its points stay in registers, the
//     source fields in shared memory, and uu with a 5-point halo in two
//     shared-memory buffers (one read, one written per substep);
//   * only uu crosses block boundaries (and vv of the last 7 planes before
//     the x0max face).  A block stores each new value together with the number
//     of the substep that produced it, in one 16-byte (FP32: 8-byte) store,
//     and its neighbours read value and number with one load and keep what
//     carries the number they wait for: no fence, no flag, no grid barrier,
//     and a block waits only for the neighbours it reads;
//   * twelve warps of a block compute and four fetch: the halos of the next
//     substep arrive while this one is computed.  Both work through the planes
//     in a lower and an upper half and meet at named barriers, so the compute
//     warps start on the lower half while the upper halos are under way;
//   * ghost points across xx0 = 0 and the axis are images of the block's own
//     columns (the tile holds all planes), so inner boundaries cost nothing;
//   * the radiation BC of the x0max face runs in blocks of its own beside the
//     interior blocks, on the same arithmetic as column_rows; the ghost values
//     that a column's next substep reads itself stay in the block;
//   * at substep 1 each block publishes its share of the residual norm, and
//     every block sums all shares in the same order before substep 4, which
//     is the first one that overwrites y_n: three substeps hide the sum.
// FP64 grids and the FP32 correction form run here.  Every point is evaluated
// with the same device functions in the same order as in the substep kernels,
// so the steps are bit-identical to theirs.
// Measured per FP64 RK4 step (substep kernels -> here): 26.0 -> 12.0 us at
// 64x64x8, 26.4 -> 15.7 at 90x75x10, 38.6 -> 23.5 at 128x128x16 (26.6 with all
// warps fetching first and then computing); a 64x64x8 mixed relaxation 58.1 ->
// 25.8 ms.  Bound by the exchange (a store, one L2 round trip and the fetch's
// instructions: most of the 5600 cycles of a substep at 64x64x8) and, from
// 96x96x12 on, by the instruction issue and shared-memory loads of the
// interior blocks and by the radiation blocks' serial recurrence and gathers
// (4400 + 5000 cycles of a substep at 128x128x16).
//
// Waits are bounded: a thread that polls too long raises the launch's error
// flag, every block leaves at its next barrier and the host reports it.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "resident.cuh"

namespace nrpyell {

namespace {

// Slots of an exchanged value, by substep.  A writer runs at most three substeps
// ahead of a reader: neighbouring interior blocks, and a radiation block and the
// face tiles of its rows, read each other; what else a radiation block reads (five
// rows either side, seven columns of tiles at least five wide) lies at most two
// tiles from one of those.
constexpr int kSlots = 8;
// Threads of a block: in an interior block 384 compute (three warpgroups) and
// 128 fetch halos.  The launch's 128 registers per thread are divided 144 : 80.
constexpr int kThreads = 512, kCompute = 384;
constexpr int kComputeRegs = 144, kFetchRegs = 80;
static_assert(kCompute * kComputeRegs + (kThreads - kCompute) * kFetchRegs <= kThreads * 128, "registers of the launch");
constexpr int kMaxBlocks = 160;      // interior blocks of one grid
// radiation rows: 12 points at an odd pitch; planes are padded so that the rows
// of the next plane continue the pattern of banks (13 (z R + row) mod 16)
constexpr int kRadPitch = 13, kRadPad = 14;
constexpr unsigned kPollLimit = 1u << 20;

// ------------------------------------------------- exchange of tagged values

template <typename T>
struct Tagged;
template <>
struct Tagged<double> {
  using Raw = double2;
  static __device__ __forceinline__ void store(Raw* p, double v, unsigned tag) {
    asm volatile("{\n.reg .b128 t;\nmov.b128 t, {%1, %2};\nst.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"((unsigned long long)tag));
  }
  static __device__ __forceinline__ unsigned load(const Raw* p, double& v) {
    long long lo, hi;
    asm volatile("{\n.reg .b128 t;\nld.relaxed.gpu.global.b128 t, [%2];\nmov.b128 {%0, %1}, t;\n}\n"
                 : "=l"(lo), "=l"(hi)
                 : "l"(p));
    v = __longlong_as_double(lo);
    return (unsigned)hi;
  }
};
template <>
struct Tagged<float> {
  using Raw = float2;
  static __device__ __forceinline__ void store(Raw* p, float v, unsigned tag) {
    const unsigned long long x = (unsigned long long)__float_as_uint(v) | ((unsigned long long)tag << 32);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;\n" ::"l"(p), "l"(x));
  }
  static __device__ __forceinline__ unsigned load(const Raw* p, float& v) {
    unsigned long long x;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];\n" : "=l"(x) : "l"(p));
    v = __uint_as_float((unsigned)x);
    return (unsigned)(x >> 32);
  }
};

// Named barriers of an interior block (0 is __syncthreads).
enum { kBarCompute = 1, kBarFree = 2, kBarFull = 4, kBarFetch = 8 };
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) {
  asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "r"(n) : "memory");
}

// ---------------------------------------------------------------- geometry

// Row pitch of the shared uu tile (at least TX + 10 points): the rows of a warp
// fall on different banks.
constexpr int tile_pitch(bool fp64, int tx) { return fp64 ? (tx == 8 ? 24 : 26) : (tx == 8 ? 24 : 48); }

// Columns x TX wide: a warp holds TX points along i0 times 32/TX rows.
template <typename T, int TX>
struct TileGeom {
  static constexpr int RPW = 32 / TX;
  static constexpr int PITCH = tile_pitch(sizeof(T) == 8, TX);
};

__host__ __device__ constexpr int ceil_div(int a, int b) { return (a + b - 1) / b; }

// A value the compiler cannot see through.  Index arithmetic that starts from
// it stays inside the time loop: hoisted out (it does not change from substep
// to substep) it took hundreds of registers and spilled.
__device__ __forceinline__ int opaque(int x) {
  asm volatile("" : "+r"(x));
  return x;
}

__device__ __forceinline__ int split(int t, int n, int parts) { return (int)((long long)t * n / parts); }

// Shared block state: the stop test's outcome, whether a wait gave up, per-warp
// residual partials.
struct BlockState {
  int stop, failed;
  double part[kThreads / 32];
};

// Polls one tagged value until it carries `tag`; 1 when the wait gave up.
template <typename T>
__device__ __forceinline__ int wait_tag(const typename Tagged<T>::Raw* p, unsigned tag, int* err) {
  T v;
  for (unsigned it = 0; it < kPollLimit; it++) {
    if (Tagged<T>::load(p, v) == tag) return 0;
    if ((it & 1023u) == 1023u && *(volatile int*)err) return 1;
  }
  atomicExch(err, 1);
  return 1;
}

// Halo values of a block: entry i comes from exchange offset tab[i].x of the
// version's slot and goes to tab[i].y of the shared buffer.  The table covers
// all planes and is padded to whole units of 32 entries with copies of entry 0
// that go to element 0 of the buffer, a corner that nothing reads.  Warp w
// takes units w, w + nw, ...; up to eight loads per thread are in flight, and a
// batch counts only when every value of the warp carries the version (else one
// lane waits for one missing value and the warp fetches the batch again).  The
// instructions per entry are what this costs: with the offsets computed here
// and values accepted one by one a fetch took twice as long, and with every
// lane polling its own values the poll traffic saturated L2.
template <typename T, int NB, typename D>
__device__ __forceinline__ int fetch(const int2* t, int stride, const typename Tagged<T>::Raw* slot, unsigned ver,
                                     D* dst, int* err) {
  const typename Tagged<T>::Raw* src[NB];
  int to[NB];
#pragma unroll
  for (int j = 0; j < NB; j++) {
    const int2 e = t[j * stride];
    src[j] = slot + e.x;
    to[j] = e.y;
  }
  for (;;) {
    T v[NB];
    unsigned tag[NB], bad = 0;
#pragma unroll
    for (int j = 0; j < NB; j++) tag[j] = Tagged<T>::load(src[j], v[j]);
#pragma unroll
    for (int j = 0; j < NB; j++) bad |= tag[j] ^ ver;
    const unsigned who = __ballot_sync(0xffffffffu, bad != 0);
    if (!who) {
#pragma unroll
      for (int j = 0; j < NB; j++) dst[to[j]] = (D)v[j];
      return 0;
    }
    int failed = 0;
    if ((threadIdx.x & 31) == 31 - __clz(who)) {
      const typename Tagged<T>::Raw* at = src[0];
#pragma unroll
      for (int j = 1; j < NB; j++)
        if (tag[j] != ver) at = src[j];
      failed = wait_tag<T>(at, ver, err);
    }
    if (__any_sync(0xffffffffu, failed)) return 1;
  }
}

// Fetches the units of `tab` with warps w = 0 .. nw - 1; returns 1 when a wait
// gave up.
template <typename T, int NB, typename D>
__device__ __forceinline__ int gather(const ResJob<T>& J, const int2* tab, int units, int w, int nw, unsigned ver,
                                      D* dst) {
  const int warp = opaque(w);
  const typename Tagged<T>::Raw* const slot =
      (const typename Tagged<T>::Raw*)J.xu + (long long)(ver & (kSlots - 1)) * J.xu_slot;
  int* const err = J.err;
  const int2* t = tab + warp * 32 + (threadIdx.x & 31);
  const int stride = nw * 32;
  int n = units > warp ? (units - warp + nw - 1) / nw : 0;
  for (; n >= NB; n -= NB, t += NB * stride)
    if (fetch<T, NB>(t, stride, slot, ver, dst, err)) return 1;
  if constexpr (NB > 4)
    if (n >= 4) {
      if (fetch<T, 4>(t, stride, slot, ver, dst, err)) return 1;
      n -= 4;
      t += 4 * stride;
    }
  switch (n) {
    case 1: return fetch<T, 1>(t, stride, slot, ver, dst, err);
    case 2: return fetch<T, 2>(t, stride, slot, ver, dst, err);
    case 3: return fetch<T, 3>(t, stride, slot, ver, dst, err);
    default: return 0;
  }
}

// One warp, before substep 4 of step n: the residual norm of y_n from all
// interior blocks' shares (summed in the same order by every block) and the
// stop test (finalize_l2's rule).
template <typename T>
__device__ __forceinline__ int stop_test(const ResJob<T>& J, int local, int n, unsigned tag, BlockState* bs) {
  const int lane = opaque(threadIdx.x & 31);
  const int nI = J.n0t * J.n1t;
  const double2* part = J.part + (n & 1) * nI;
  double v[kMaxBlocks / 32], s = 0.0;
  unsigned pending = 0;
#pragma unroll
  for (int j = 0; j < kMaxBlocks / 32; j++)
    if (lane + 32 * j < nI) pending |= 1u << j;
  bool ok = true;
  for (unsigned it = 0; pending && ok; it++) {
    unsigned got[kMaxBlocks / 32];
#pragma unroll
    for (int j = 0; j < kMaxBlocks / 32; j++)
      if (pending >> j & 1u) got[j] = Tagged<double>::load(part + lane + 32 * j, v[j]);
#pragma unroll
    for (int j = 0; j < kMaxBlocks / 32; j++)
      if ((pending >> j & 1u) && got[j] == tag) pending &= ~(1u << j);
    if (pending && (it >= kPollLimit || ((it & 1023u) == 1023u && *(volatile int*)J.err))) {
      if (it >= kPollLimit) atomicExch(J.err, 1);
      ok = false;
    }
  }
#pragma unroll
  for (int j = 0; j < kMaxBlocks / 32; j++)
    if (lane + 32 * j < nI) s += v[j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  ok = __all_sync(0xffffffffu, ok);
  if (lane == 0) {
    bool test = true;
    if (J.check_every > 0) test = n >= 1 && ((n - 1) % J.check_every == 0 || n >= J.max_steps);
    const bool met = test && residual_met(J, s);
    const bool stop = met || n >= J.max_steps;
    bs->stop = stop;
    if (local == 0 && ok) {
      J.sums[n] = s;
      if (met) J.state[2] = 1;
      if (stop)
        J.state[1] = stop_mark(n);
      else
        J.state[0] = n + 1;
    }
  }
  return !ok;
}

// Entries of a block's table: `n` per plane, all planes, in whole units.
__host__ __device__ inline int table_entries(int n, int Nz) { return ceil_div(n * Nz, 32) * 32; }

// ---------------------------------------------------------- interior blocks

template <typename T, bool CORR, int TX, int P2>
__device__ __forceinline__ void interior_block(const ResJob<T>& J, int local, unsigned base, int steps,
                                               unsigned char* smem, BlockState* bs) {
  using G = TileGeom<T, TX>;
  constexpr int PITCH = G::PITCH, RPW = G::RPW;
  using Raw = typename Tagged<T>::Raw;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int Nz = J.Nxx2, N0 = J.N0, Zh = (Nz + 1) / 2;  // planes of the lower half
  const int t0 = local % J.n0t, t1 = local / J.n0t;
  const int x0 = split(t0, J.Nxx0, J.n0t), w = split(t0 + 1, J.Nxx0, J.n0t) - x0;
  const int r0 = split(t1, J.Nxx1, J.n1t), h = split(t1 + 1, J.Nxx1, J.n1t) - r0;
  const int plane = (J.hmax + 2 * NGHOSTS) * PITCH;
  int2* const tab = reinterpret_cast<int2*>(smem);
  T* const buf0 = reinterpret_cast<T*>(smem + sizeof(int2) * (table_entries(10 * (J.hmax + TX), Nz) + 32));
  T* const buf1 = buf0 + (size_t)Nz * plane;
  const bool left = t0 == 0, low = t1 == 0, high = t1 == J.n1t - 1;
  // ---- halo entries: columns left and right, rows below and above; the lower
  // half's planes, then the upper half's, each in whole units
  const int xrow = J.xu_row;
  const int nl = left ? 0 : NGHOSTS * h, nr = NGHOSTS * h, nd = low ? 0 : NGHOSTS * w, nu = high ? 0 : NGHOSTS * w;
  const int nent = nl + nr + nd + nu, units0 = ceil_div(nent * Zh, 32), units1 = ceil_div(nent * (Nz - Zh), 32);
  for (int u = tid; u < (units0 + units1) * 32; u += kThreads) {
    const bool upper = u >= units0 * 32;
    const int i = upper ? u - units0 * 32 : u;
    const bool pad = i >= nent * (upper ? Nz - Zh : Zh);
    const int z = pad ? 0 : (upper ? Zh : 0) + i / nent;
    int q = pad ? 0 : i % nent, jx, jr;
    if (q < nl) {
      jx = q % NGHOSTS - NGHOSTS;
      jr = q / NGHOSTS;
    } else if ((q -= nl) < nr) {
      jx = w + q % NGHOSTS;
      jr = q / NGHOSTS;
    } else if ((q -= nr) < nd) {
      jx = q % w;
      jr = q / w - NGHOSTS;
    } else {
      q -= nd;
      jx = q % w;
      jr = h + q / w;
    }
    // padding: the half's first entry, to a corner of the tile
    const int zp = pad && upper ? Zh : z;
    tab[u] = make_int2((r0 + jr) * xrow + x0 + jx + zp * J.xu_plane,
                       pad ? 0 : (jr + NGHOSTS) * PITCH + jx + NGHOSTS + z * plane);
  }
  // ---- uu with its halo from y_n (corners of the tile are never read)
  {
    const int tw = w + 2 * NGHOSTS, th = h + 2 * NGHOSTS;
    for (int e = tid; e < tw * th * Nz; e += kThreads) {
      const int xx = e % tw, q = e / tw, rr = q % th, z = q / th;
      int jx = xx - NGHOSTS, jr = rr - NGHOSTS;
      if ((jx < 0 || jx >= w) && (jr < 0 || jr >= h)) continue;
      jx += x0;
      jr += r0;
      int zs = z;
      bool flip = false;
      if (jx < 0) {
        jx = -1 - jx;
        flip = true;
      }
      if (jr < 0) {
        jr = -1 - jr;
        flip = !flip;
      } else if (jr >= J.Nxx1) {
        jr = 2 * J.Nxx1 - 1 - jr;
        flip = !flip;
      }
      if (flip) {
        zs += J.half2;
        if (zs >= Nz) zs -= Nz;
      }
      buf0[z * plane + rr * PITCH + xx] =
          __ldcg(J.y + (jx + NGHOSTS) + (long long)N0 * (jr + NGHOSTS) + J.N01 * (zs + NGHOSTS));
    }
  }
  __syncthreads();

  if (warp >= kCompute / 32) {
    // ---- the fetching warps: the halo of every version after the first, half
    // by half, into the buffer that version is read from
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kFetchRegs));
    const int gw = warp - kCompute / 32, ngw = (kThreads - kCompute) / 32;
    const int n0 = J.n_start;
    bool failed = false;
    for (int i = 1; i < 4 * steps; i++) {
      const unsigned ver = base + i;
      const int par = i & 1;
      T* const dst = par ? buf1 : buf0;
      // the substep that read this buffer's previous version is done
      if (i >= 2) bar_sync(kBarFree + par, kThreads);
      if ((i & 3) == 3) {  // substep 4 comes: the stop test first
        if (gw == ngw - 1 && !failed) failed = stop_test<T>(J, local, n0 + (i >> 2), ver - 2, bs);
        if (failed && lane == 0) bs->failed = 1;
        bar_sync(kBarFetch, kThreads - kCompute);
        if (lane == 0 && gw == 0 && bs->failed) bs->stop = 1;
        bar_sync(kBarFetch, kThreads - kCompute);
        if (bs->stop) {
          bar_arrive(kBarFull + par, kThreads);
          break;
        }
      }
      // a wait that gave up ends the launch at the next stop test; until then
      // nothing is waited for
      if (!failed) failed = gather<T, 8>(J, tab, units0, gw, ngw, ver, dst);
      bar_arrive(kBarFull + par, kThreads);
      if (!failed) failed = gather<T, 8>(J, tab + units0 * 32, units1, gw, ngw, ver, dst);
      bar_arrive(kBarFull + 2 + par, kThreads);
    }
    return;
  }

  // ---- the computing warps: a thread's column and its P2 planes of either half
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kComputeRegs));
  constexpr int P = 2 * P2, NF = CORR ? 5 : 3;
  T* const fld = buf1 + (size_t)Nz * plane + tid;  // source fields of the thread's points, [P][NF][kCompute]
  const int nrg = (J.hmax + RPW - 1) / RPW, zg = warp / nrg;
  const int x = lane % TX, row = (warp % nrg) * RPW + lane / TX, zlo = zg * P2;
  const bool col_ok = x < w && row < h && zlo < Zh;
  const long long gcol = (x0 + x + NGHOSTS) + (long long)N0 * (r0 + row + NGHOSTS);
  const int scol = (row + NGHOSTS) * PITCH + x + NGHOSTS;
  // plane of point p (p < P2: lower half), or -1
  auto plane_of = [&](int p) -> int {
    const int k = zlo + (p < P2 ? p : p - P2);
    return p < P2 ? (k < Zh ? k : -1) : (k < Nz - Zh ? Zh + k : -1);
  };
  T yu[P], yv[P], au[P], av[P], vv[P];
  T C22 = 0, C00 = 0, C11 = 0, C1 = 0, C0 = 0, Cc = 0;
#pragma unroll
  for (int p = 0; p < P; p++) {
    yu[p] = yv[p] = au[p] = av[p] = vv[p] = (T)0;
    const int z = plane_of(p);
    if (col_ok && z >= 0) {
      const long long g = gcol + J.N01 * (z + NGHOSTS);
      yu[p] = __ldcg(J.y + g);
      yv[p] = __ldcg(J.y + J.Ntot + g);
      fld[(p * NF + 0) * kCompute] = __ldg(J.aux + ADD_TIMES_AUUGF * J.Ntot + g);
      fld[(p * NF + 1) * kCompute] = __ldg(J.aux + PSI_BACKGROUNDGF * J.Ntot + g);
      fld[(p * NF + 2) * kCompute] = __ldg(J.aux + WAVESPEEDGF * J.Ntot + g);
      if constexpr (CORR) {
        fld[(p * NF + 3) * kCompute] = __ldg(J.R0 + g);
        fld[(p * NF + 4) * kCompute] = __ldg(J.R0 + J.Ntot + g);
      }
      vv[p] = yv[p];
    }
  }
  if (col_ok) {
    C22 = __ldg(J.coef + gcol);
    C00 = __ldg(J.coef + J.N01 + gcol);
    C11 = __ldg(J.coef + 2 * J.N01 + gcol);
    C1 = __ldg(J.coef + 3 * J.N01 + gcol);
    C0 = __ldg(J.coef + 4 * J.N01 + gcol);
    Cc = __ldg(J.coef + 5 * J.N01 + gcol);
  }
  const bool img0 = left && x < NGHOSTS, imgd = low && row < NGHOSTS, imgu = high && row >= h - NGHOSTS;
  const bool image = img0 || imgd || imgu;
  const bool pub_v = x0 + x >= J.Nxx0 - 7;
  const int xg = (r0 + row) * xrow + x0 + x;                              // exchange offset of the column, plane 0
  const int vg = J.xv0 + (r0 + row) * 12 + (x0 + x - (J.Nxx0 - 7));
  const T dt = J.dt, eta = J.eta;
  const int xu_plane = J.xu_plane, xv_plane = J.xv_plane, nzp = Nz * plane, himg = J.half2 * plane;
  const long long xu_slot = J.xu_slot;
  double r2 = 0.0;

  // one substep of the lower (H = 0) or upper half
  auto substep = [&](auto st, auto half, const T* __restrict__ cur, T* __restrict__ nxt, unsigned ver) {
    constexpr int STAGE = decltype(st)::value, H = decltype(half)::value;
    if (STAGE == 1 && H == 0) r2 = 0.0;
    const int zb = opaque(H ? Zh + zlo : zlo), zend = H ? Nz : Zh;
    if (col_ok && zb < zend) {
      double wl2 = 0.0;
      if (STAGE == 1) wl2 = __ldg(J.w + gcol);
      int o = zb * plane;  // offset of the plane
      const int oend = zend * plane, sc = opaque(scol);
      // uu along i2: planes zb-5 .. zb+P2+4, wrapped (those past a partial last
      // chunk are loaded but not used)
      T q[P2 + 10];
      {
        int oq = o - NGHOSTS * plane;
        if (oq < 0) oq += nzp;
#pragma unroll
        for (int j = 0; j < P2 + 10; j++) {
          q[j] = cur[sc + oq];
          oq += plane;
          if (oq >= nzp) oq -= nzp;
        }
      }
      const T* f = fld + opaque(H * P2 * NF * kCompute);
      Raw* xu = (Raw*)J.xu + (long long)((ver + 1) & (kSlots - 1)) * xu_slot;
      Raw* xv = xu + (vg + zb * xv_plane);
      xu += xg + zb * xu_plane;
#pragma unroll
      for (int p = 0; p < P2; p++) {
        if (o < oend) {
          const T* c = cur + sc + o;
          T s0 = 0, s1 = 0, s00 = 0, s11 = 0, s22 = 0;
#pragma unroll
          for (int k = 1; k <= 5; k++) {
            const T am = c[-k], ap = c[k];
            const T bm = c[-k * PITCH], bp = c[k * PITCH];
            s0 = fma(W<T>::d(k), ap - am, s0);
            s1 = fma(W<T>::d(k), bp - bm, s1);
            s00 = fma(W<T>::e(k), ap + am, s00);
            s11 = fma(W<T>::e(k), bp + bm, s11);
          }
#pragma unroll
          for (int k = 1; k <= 5; k++) s22 = fma(W<T>::e(k), q[p + 5 + k] + q[p + 5 - k], s22);
          T ku, kv, br;
          const T* fp = f + p * NF * kCompute;
          constexpr int FS = kCompute;
          const int i = H * P2 + p;
          if constexpr (CORR) {
            T ju, jv;
            point_rhs_correction<T>(q[p + 5], vv[i], fp[0], fp[FS], fp[2 * FS], C22, C00, C11, C1, C0, Cc, s0, s1, s00,
                                    s11, s22, eta, fp[3 * FS], fp[4 * FS], ku, kv, br, ju, jv);
          } else {
            point_rhs<T>(q[p + 5], vv[i], fp[0], fp[FS], fp[2 * FS], C22, C00, C11, C1, C0, Cc, s0, s1, s00, s11, s22,
                         eta, ku, kv, br);
          }
          T ou, ov;
          rk_combine<T, STAGE>(ku, yu[i], au[i], ou, dt);
          rk_combine<T, STAGE>(kv, yv[i], av[i], ov, dt);
          vv[i] = ov;
          if (STAGE == 4) {
            yu[i] = ou;
            yv[i] = ov;
          }
          Tagged<T>::store(xu, ou, ver + 1);
          if (pub_v) Tagged<T>::store(xv, ov, ver + 1);
          T* n = nxt + sc + o;
          *n = ou;
          if (image) {  // images across xx0 = 0 and the axis: mirrored, half a turn on
            T* ni = n + (o + himg >= nzp ? himg - nzp : himg);
            if (img0) ni[-1 - 2 * x] = ou;
            if (imgd) ni[-(1 + 2 * row) * PITCH] = ou;
            if (imgu) ni[(2 * (h - row) - 1) * PITCH] = ou;
          }
          if (STAGE == 1) {
            const double bb = (double)br;
            r2 += bb * bb * wl2;
          }
        }
        o += plane;
        xu += xu_plane;
        xv += xv_plane;
      }
    }
    if (STAGE == 1 && H == 1) {
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) r2 += __shfl_down_sync(0xffffffffu, r2, s);
      if (lane == 0) bs->part[warp] = r2;
    }
  };
  // substep `st` of version base + i: its halves as their halos arrive, then
  // every computing warp's values are written and the buffer read is free
  auto full_substep = [&](auto st, int i) {
    const int par = i & 1;
    const T* cur = par ? buf1 : buf0;
    T* nxt = par ? buf0 : buf1;
    if (i > 0) bar_sync(kBarFull + par, kThreads);
    if (decltype(st)::value == 4 && bs->stop) return true;
    substep(st, std::integral_constant<int, 0>(), cur, nxt, base + i);
    if (i > 0) bar_sync(kBarFull + 2 + par, kThreads);
    substep(st, std::integral_constant<int, 1>(), cur, nxt, base + i);
    bar_sync(kBarCompute, kCompute);
    bar_arrive(kBarFree + par, kThreads);
    return false;
  };
  const int n0 = J.n_start;
  for (int k = 0; k < steps; k++) {
    full_substep(std::integral_constant<int, 1>(), 4 * k);
    if (warp == 0) {  // the block's share of the residual norm
      double s = lane < kCompute / 32 ? bs->part[lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (lane == 0)
        Tagged<double>::store(J.part + ((n0 + k) & 1) * (J.n0t * J.n1t) + local, s, base + 4 * k + 1);
    }
    full_substep(std::integral_constant<int, 2>(), 4 * k + 1);
    full_substep(std::integral_constant<int, 3>(), 4 * k + 2);
    if (full_substep(std::integral_constant<int, 4>(), 4 * k + 3)) break;
  }
  if (col_ok && !bs->failed) {
#pragma unroll
    for (int p = 0; p < P; p++) {
      const int z = plane_of(p);
      if (z >= 0) {
        const long long g = gcol + J.N01 * (z + NGHOSTS);
        J.y[g] = yu[p];
        J.y[J.Ntot + g] = yv[p];
      }
    }
  }
}

// --------------------------------------------------------- radiation blocks
// Rows r0 .. r0+R-1 of the x0max face, all planes, both gridfunctions, with
// column_rows' arithmetic.  What the layer recurrence needs of a column, the
// radial derivatives at the last interior plane and the five layers and the
// RHS of the last interior point, is spread over the warps; after a barrier one
// thread per column and gridfunction runs the recurrence.

// Shared layout of a radiation block, in doubles after the entry table.  What a
// thread reads of a table stands together, at compile-time offsets (odd strides
// keep the banks apart).
constexpr int kCfStride = 7, kFpStride = 5, kGeoStride = 31;
struct RadLayout {
  int F, X, Y, kl, cf, fp, geo, w, total;
};
__host__ __device__ inline RadLayout rad_layout(int R, int Nz) {
  RadLayout l;
  const int RZ = R * Nz;
  l.F = 0;                                                // [2][Nz][R + 10][13] (+ 14) uu, vv
  l.X = l.F + 2 * Nz * ((R + 2 * NGHOSTS) * kRadPitch + kRadPad);     // [5][2 RZ] drf + f / r at layers -1 .. 3
  l.Y = l.X + 5 * 2 * RZ;                                 // [5][2 RZ] drf + f (1/r) at layers 0 .. 4
  l.kl = l.Y + 5 * 2 * RZ;                                // [2 RZ] RHS of the last interior point
  l.cf = l.kl + 2 * RZ;                                   // [R][6] metric weights of the last interior point
  l.fp = l.cf + kCfStride * R;                            // [RZ][3, correction form 5] its pointwise fields
  l.geo = l.fp + kFpStride * RZ;                          // [R][5][6] r, dxx0/dr, dxx1/dr, 1/r, r^3
  l.w = (l.geo + kGeoStride * R + 1) / 2 * 2;             // [6][12] weights along x0
  l.total = l.w + 72;
  return l;
}
// Entries of a plane: the last 7 interior points of the block's rows (their
// ghost points stay in the block) and 6 points of the rows around them.
__host__ __device__ inline int rad_entries(int R) { return 2 * (7 * R + 6 * 2 * NGHOSTS); }

// Points jj0 .. jj0 + K - 1 of one column (q of its 2 RZ): f the column's row in
// F, g its geometry, w the weights.  K points share the column's 12 values
// along x0, and a warp's K is uniform.
template <int K>
__device__ __forceinline__ void radiation_points(const double* f, const double* g, const double* w, int jj0, int q,
                                                 int n, double invdx0, double invdx1, double* X, double* Y) {
  double v[12];
#pragma unroll
  for (int m = 0; m < 12; m++) v[m] = f[m];
#pragma unroll
  for (int i = 0; i < K; i++) {
    const int jj = jj0 + i;
    const double2* const wj = reinterpret_cast<const double2*>(w) + 6 * jj;
    double wt[12], u[12];
#pragma unroll
    for (int m = 0; m < 6; m++) {
      const double2 t = wj[m];
      wt[2 * m] = t.x;
      wt[2 * m + 1] = t.y;
    }
    // the stencil of point 0 starts at value 0, the others' at value 1
#pragma unroll
    for (int m = 0; m < 11; m++) u[m] = jj == 0 ? v[m] : v[m + 1];
    const double d0 = radiation_sum_x0(wt, u);
    const double* const f1 = f + 6 + jj;
#pragma unroll
    for (int m = 0; m < 11; m++) u[m] = (m == 5) ? 0.0 : f1[(m - 5) * kRadPitch];
    const double d1 = radiation_sum_x1<true>(u);
    const double drf = radiation_drf(d0, d1, invdx0, invdx1, g[6 + jj], g[12 + jj]);
    const double fv = f1[0];
    if (jj < NGHOSTS) X[jj * n + q] = radiation_outgoing_neighbour(drf, fv, g[jj]);
    if (jj > 0) Y[(jj - 1) * n + q] = radiation_outgoing_point(drf, fv, g[18 + jj]);
  }
}

template <typename T, bool CORR>
__device__ __forceinline__ void radiation_block(const ResJob<T>& J, int local, unsigned base, int steps,
                                                unsigned char* smem, BlockState* bs) {
  using Raw = typename Tagged<T>::Raw;
  const int tid = threadIdx.x, warp = tid >> 5, NT = blockDim.x;
  const int Nz = J.Nxx2, N0 = J.N0;
  const int rb = local - J.n0t * J.n1t;
  const int r0 = split(rb, J.Nxx1, J.nrad), R = split(rb + 1, J.Nxx1, J.nrad) - r0;
  const int RZ = R * Nz, rows = R + 2 * NGHOSTS;
  const int plane = rows * kRadPitch + kRadPad, gplane = plane * Nz;  // F[g][z]: rows of 13, then the padding
  const int nent = rad_entries(R), units = ceil_div(nent * Nz, 32);
  int2* const tab = reinterpret_cast<int2*>(smem);
  double* const base_s = reinterpret_cast<double*>(smem + sizeof(int2) * 32 * units);
  const RadLayout lay = rad_layout(R, Nz);
  double* const F = base_s + lay.F;
  double* const X = base_s + lay.X;
  double* const Y = base_s + lay.Y;
  double* const kl = base_s + lay.kl;
  double* const cf = base_s + lay.cf;
  double* const fp = base_s + lay.fp;
  double* const geo = base_s + lay.geo;
  double* const wx0 = base_s + lay.w;
  // ---- the entries, and the same points from y_n (ghost rows across the axis:
  // half a turn on)
  const int xrow = J.xu_row;
  for (int i = tid; i < units * 32; i += NT) {
    const bool pad = i >= nent * Nz;
    const int z = pad ? 0 : i / nent, e = pad ? 0 : i % nent, g = e / (nent / 2);
    int q = e % (nent / 2), jr, c;
    if (q < 7 * R) {
      jr = q / 7;
      c = q % 7;
    } else {
      q -= 7 * R;
      c = 6 + q % 6;
      q /= 6;
      jr = q < NGHOSTS ? q - NGHOSTS : R + q - NGHOSTS;
    }
    int j1 = r0 + jr, zs = z;
    if (j1 < 0 || j1 >= J.Nxx1) {
      j1 = j1 < 0 ? -1 - j1 : 2 * J.Nxx1 - 1 - j1;
      zs = z + J.half2 >= Nz ? z + J.half2 - Nz : z + J.half2;
    }
    const int to = g * gplane + z * plane + (jr + NGHOSTS) * kRadPitch + c;
    tab[i] = make_int2(g ? J.xv0 + zs * J.xv_plane + j1 * 12 + c : zs * J.xu_plane + j1 * xrow + J.Nxx0 - 7 + c,
                       pad ? 0 : to);
    if (!pad)
      F[to] = (double)__ldcg(J.y + g * J.Ntot + (J.Nxx0 - 7 + c + NGHOSTS) + (long long)N0 * (j1 + NGHOSTS) +
                             J.N01 * (zs + NGHOSTS));
  }
  for (int e = tid; e < 72; e += NT) {
    const int jj = e / 12;
    wx0[e] = e % 12 < 11 ? c_fd1w[((jj <= 1) ? -1 : -jj) + 5][e % 12] : 0.0;
  }
  for (int e = tid; e < 6 * R; e += NT) {
    const int jj = e / R, row = e % R, i1 = r0 + row + NGHOSTS;
    double* const g = geo + row * kGeoStride + jj;
    const double r = __ldg(J.colgeo + jj * J.N1 + i1);
    g[0] = r;
    g[6] = __ldg(J.colgeo + (6 + jj) * J.N1 + i1);
    g[12] = __ldg(J.colgeo + (12 + jj) * J.N1 + i1);
    g[18] = 1.0 / r;
    g[24] = radiation_r3(r);
  }
  const long long last = NGHOSTS + J.Nxx0 - 1;
  for (int e = tid; e < 6 * R; e += NT)
    cf[(e % R) * kCfStride + e / R] =
        (double)__ldg(J.coef + (e / R) * J.N01 + last + (long long)N0 * (r0 + e % R + NGHOSTS));
  for (int e = tid; e < (CORR ? 5 : 3) * RZ; e += NT) {
    const int f = e / RZ, c = e % RZ, row = c % R, z = c / R;
    const long long g = last + (long long)N0 * (r0 + row + NGHOSTS) + J.N01 * (z + NGHOSTS);
    const T* src = f == 0 ? J.aux + ADD_TIMES_AUUGF * J.Ntot
                 : f == 1 ? J.aux + PSI_BACKGROUNDGF * J.Ntot
                 : f == 2 ? J.aux + WAVESPEEDGF * J.Ntot
                 : f == 3 ? J.R0 : J.R0 + J.Ntot;
    fp[c * kFpStride + f] = (double)__ldg(src + g);
  }
  // ---- the thread's column of ghost points
  const bool live = tid < 2 * RZ;
  const int cg = live ? tid / RZ : 0, cc = live ? tid % RZ : 0, crow = cc % R, cz = cc / R;
  const long long gidx = cg * J.Ntot + (N0 - NGHOSTS) + (long long)N0 * (r0 + crow + NGHOSTS) + J.N01 * (cz + NGHOSTS);
  const double cw = (double)J.cOB[cg];
  Raw* const to0 = (Raw*)J.xu + (cg ? J.xv0 + (r0 + crow) * 12 + 7 + cz * J.xv_plane
                                    : (r0 + crow) * xrow + J.Nxx0 + cz * J.xu_plane);
  const long long slot = J.xu_slot;
  const T dt = J.dt, eta = J.eta;
  const double invdx0 = J.invdx0, invdx1 = J.invdx1;
  T y[NGHOSTS], acc[NGHOSTS];
  double base_rhs[NGHOSTS];
#pragma unroll
  for (int L = 0; L < NGHOSTS; L++) {
    y[L] = live ? __ldcg(J.y + gidx + L) : (T)0;
    acc[L] = (T)0;
    base_rhs[L] = (CORR && live) ? (double)__ldg(J.R0 + gidx + L) : 0.0;
  }
  double* const own = F + cg * gplane + cz * plane + (crow + NGHOSTS) * kRadPitch + 7;  // its ghost points in F
  if (live)
    for (int L = 0; L < NGHOSTS; L++) own[L] = (double)y[L];
  // a warp's derivative task: K = 1, 2, 3 or 6 points of 32 of both
  // gridfunctions' columns; the RHS of the last interior points goes to the
  // warps left, in rounds that take about twice a point's time: the K with the
  // shortest longer one
  const int nw = NT >> 5, n_rhs = ceil_div(RZ, 32), n_col = ceil_div(2 * RZ, 32);
  int K = 6;
  {
    int best = 1 << 30;
    for (int k = 6; k >= 1; k = k == 6 ? 3 : k - 1) {
      const int left = nw - n_col * (6 / k);
      const int t = left > 0 ? max(k, 2 * ceil_div(n_rhs, left)) : left == 0 ? k + 2 * ceil_div(n_rhs, nw) : 1 << 30;
      if (t <= best) {
        best = t;
        K = k;
      }
    }
  }
  const int n_drf = n_col * (6 / K), rest = nw - n_drf;
  const int jj0 = warp / n_col * K, drf_q = (warp % n_col) * 32 + (tid & 31);
  const bool drf_on = warp < n_drf && drf_q < 2 * RZ;
  const int drf_c = drf_q >= RZ ? drf_q - RZ : drf_q, drf_row = drf_c % R;
  const int drf_f = (drf_q >= RZ ? gplane : 0) + drf_c / R * plane + (drf_row + NGHOSTS) * kRadPitch;
  const int rhs_step = rest > 0 ? rest : nw, rhs_first = rest <= 0 ? warp : warp >= n_drf ? warp - n_drf : n_rhs;

  auto substep = [&](auto st, unsigned ver) {
    constexpr int STAGE = decltype(st)::value;
    if (drf_on) {
      const double* const f = F + opaque(drf_f);
      const double* const g = geo + opaque(drf_row * kGeoStride);
      const int j = opaque(jj0), q = opaque(drf_q);
      if (K == 1)
        radiation_points<1>(f, g, wx0, j, q, 2 * RZ, invdx0, invdx1, X, Y);
      else if (K == 2)
        radiation_points<2>(f, g, wx0, j, q, 2 * RZ, invdx0, invdx1, X, Y);
      else if (K == 3)
        radiation_points<3>(f, g, wx0, j, q, 2 * RZ, invdx0, invdx1, X, Y);
      else
        radiation_points<6>(f, g, wx0, j, q, 2 * RZ, invdx0, invdx1, X, Y);
    }
    for (int task = opaque(rhs_first); task < n_rhs; task += rhs_step) {
      const int c = task * 32 + opaque(tid & 31);
      if (c < RZ) {
        const int z = c / R, row = c - z * R;
        const double* const f = F + z * plane + (row + NGHOSTS) * kRadPitch;
        T s0 = 0, s1 = 0, s00 = 0, s11 = 0, s22 = 0;
#pragma unroll
        for (int k = 1; k <= 5; k++) {
          const T am = (T)f[6 - k], ap = (T)f[6 + k];
          const T bm = (T)f[6 - k * kRadPitch], bp = (T)f[6 + k * kRadPitch];
          s0 = fma(W<T>::d(k), ap - am, s0);
          s1 = fma(W<T>::d(k), bp - bm, s1);
          s00 = fma(W<T>::e(k), ap + am, s00);
          s11 = fma(W<T>::e(k), bp + bm, s11);
        }
#pragma unroll
        for (int k = 1; k <= 5; k++) {
          const int up = (z + k >= Nz ? k - Nz : k) * plane, dn = (z - k < 0 ? Nz - k : -k) * plane;
          s22 = fma(W<T>::e(k), (T)f[6 + up] + (T)f[6 + dn], s22);
        }
        T ku, kv, br;
        const T vv = (T)f[gplane + 6];
        const double* const m = cf + row * kCfStride;
        const double* const p = fp + c * kFpStride;
        if constexpr (CORR) {
          T ju, jv;
          point_rhs_correction<T>((T)f[6], vv, (T)p[0], (T)p[1], (T)p[2], (T)m[0], (T)m[1], (T)m[2], (T)m[3], (T)m[4],
                                  (T)m[5], s0, s1, s00, s11, s22, eta, (T)p[3], (T)p[4], ku, kv, br, ju, jv);
          ku = ju;
          kv = jv;
        } else {
          point_rhs<T>((T)f[6], vv, (T)p[0], (T)p[1], (T)p[2], (T)m[0], (T)m[1], (T)m[2], (T)m[3], (T)m[4], (T)m[5],
                       s0, s1, s00, s11, s22, eta, ku, kv, br);
        }
        kl[c] = (double)ku;
        kl[RZ + c] = (double)kv;
      }
    }
    __syncthreads();
    if (live) {
      const int t = opaque(tid);
      const double* const g = geo + opaque(crow * kGeoStride);
      double k = kl[t];
      Raw* to = to0 + (long long)((ver + 1) & (kSlots - 1)) * slot;
      double mine[NGHOSTS];
#pragma unroll
      for (int L = 0; L < NGHOSTS; L++) {
        k = radiation_layer(cw, k, X[L * 2 * RZ + t], Y[L * 2 * RZ + t], g[24 + L], g[19 + L]);
        const double kfull = CORR ? k + base_rhs[L] : k;
        T ou;
        rk_combine<T, STAGE>((T)kfull, y[L], acc[L], ou, dt);
        if (STAGE == 4) y[L] = ou;
        Tagged<T>::store(to + L, ou, ver + 1);
        mine[L] = (double)ou;
      }
      // after the recurrence, whose loads the compiler would keep behind these
      // (this substep's reads of F are done: the barrier above)
#pragma unroll
      for (int L = 0; L < NGHOSTS; L++) own[L] = mine[L];
    }
  };

  unsigned ver = base;
  const int n0 = J.n_start;
  for (int k = 0; k < steps; k++) {
    const int n = n0 + k;
    if (__syncthreads_or(k > 0 ? gather<T, 4>(J, tab, units, warp, NT >> 5, ver, F) : 0)) return;
    substep(std::integral_constant<int, 1>(), ver);
    ver++;
    if (__syncthreads_or(gather<T, 4>(J, tab, units, warp, NT >> 5, ver, F))) return;
    substep(std::integral_constant<int, 2>(), ver);
    ver++;
    if (__syncthreads_or(gather<T, 4>(J, tab, units, warp, NT >> 5, ver, F))) return;
    substep(std::integral_constant<int, 3>(), ver);
    ver++;
    int failed = warp == (NT >> 5) - 1 ? stop_test<T>(J, local, n, ver - 2, bs) : 0;
    failed |= gather<T, 4>(J, tab, units, warp, NT >> 5, ver, F);
    if (__syncthreads_or(failed)) return;
    if (bs->stop) break;
    substep(std::integral_constant<int, 4>(), ver);
    ver++;
  }
  if (live) {
#pragma unroll
    for (int L = 0; L < NGHOSTS; L++) J.y[gidx + L] = y[L];
  }
}

// Up to `steps` RK4 steps of every job from step `first` on; block b belongs to
// the last job with cta0 <= b.  Exchanged values of this launch carry tags base + 1 ..
// base + 4 steps.
template <typename T, bool CORR, int TX, int P2>
__global__ void __launch_bounds__(kThreads, 1)
    k_relax_resident(const ResJob<T>* __restrict__ jobs, int njobs, unsigned base, int steps, int first) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ BlockState bs;
  __shared__ ResJob<T> J;
  int j = 0;
  while (j + 1 < njobs && (int)blockIdx.x >= jobs[j + 1].cta0) j++;
  if (threadIdx.x == 0) {
    J = jobs[j];
    J.n_start = first;
    bs.stop = stopped_before(*(volatile int*)(J.state + 1), first);
    bs.failed = 0;
  }
  __syncthreads();
  if (bs.stop) return;
  const int local = (int)blockIdx.x - J.cta0;
  if (local < J.n0t * J.n1t)
    interior_block<T, CORR, TX, P2>(J, local, base, steps, smem, &bs);
  else
    radiation_block<T, CORR>(J, local, base, steps, smem, &bs);
}

// history[i]: weighted sum of squares -> log10 L2 (finalize_l2's form)
__global__ void k_history_log10(double* history, double volume, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) history[i] = log10(1e-16 + sqrt(history[i] / volume));
}

// ------------------------------------------------------------------- host

int device_attr(cudaDeviceAttr a) {
  int dev = 0, v = 0;
  NRPYELL_CUDA(cudaGetDevice(&dev));
  NRPYELL_CUDA(cudaDeviceGetAttribute(&v, a, dev));
  return v;
}

constexpr int kTX[] = {8, 16};
constexpr int kP[] = {1, 2, 3};  // planes of a thread per half

template <typename T>
using ResKernel = void (*)(const ResJob<T>*, int, unsigned, int, int);

template <typename T>
ResKernel<T> resident_kernel(int tx, int p) {
  constexpr bool CORR = sizeof(T) == 4;
#define NRPYELL_RES(TX, P) \
  if (tx == TX && p == P) return k_relax_resident<T, CORR, TX, P>;
  NRPYELL_RES(8, 1) NRPYELL_RES(8, 2) NRPYELL_RES(8, 3)
  NRPYELL_RES(16, 1) NRPYELL_RES(16, 2) NRPYELL_RES(16, 3)
#undef NRPYELL_RES
  return nullptr;
}

// Device memory that only grows.
struct ResidentArea {
  size_t bytes = 0;
  unsigned char* mem = nullptr;
};

// Work memory of the on-chip driver, kept between calls until
// nrpyell_release_tables.  Values are told from older ones by their tags alone,
// so a word that is read as a tag must never have held anything else since it
// was cleared: the exchange slots of FP64 (value and tag in 16 bytes), those of
// FP32 (8 bytes) and the residual shares have an area each, in which every
// layout has its tags at the same places.
struct ResidentWork {
  ResidentArea slots[2], shares;  // slots: FP64, FP32
  ResidentArea jobs;
  int* err = nullptr;
  int* pinned = nullptr;          // polled states of two launches
  size_t pinned_ints = 0;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  unsigned version = 0;           // last tag used in slots and shares
};
ResidentWork g_res;

size_t align_up(size_t n) { return (n + 255) / 256 * 256; }

bool grow(ResidentArea* a, size_t bytes) {
  if (a->bytes >= bytes) return true;
  NRPYELL_CUDA(cudaStreamSynchronize(stream()));
  cudaFree(a->mem);
  *a = ResidentArea();
  NRPYELL_CUDA(dev_alloc(&a->mem, bytes));
  if (!status_ok()) return false;
  NRPYELL_CUDA(cudaMemsetAsync(a->mem, 0, bytes, stream()));
  a->bytes = bytes;
  return status_ok();
}

bool ensure_resident(bool fp64, size_t slot_bytes, size_t share_bytes, size_t jobs_bytes, size_t pinned_ints) {
  if (!g_res.err) {
    NRPYELL_CUDA(dev_alloc(&g_res.err, sizeof(int)));
    NRPYELL_CUDA(cudaMemsetAsync(g_res.err, 0, sizeof(int), stream()));
    for (cudaEvent_t& e : g_res.ev) NRPYELL_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  }
  if (!grow(&g_res.slots[fp64 ? 0 : 1], slot_bytes) || !grow(&g_res.shares, share_bytes) ||
      !grow(&g_res.jobs, jobs_bytes))
    return false;
  if (g_res.pinned_ints < pinned_ints) {
    NRPYELL_CUDA(cudaStreamSynchronize(stream()));
    cudaFreeHost(g_res.pinned);
    g_res.pinned = nullptr;
    g_res.pinned_ints = 0;
    NRPYELL_CUDA(cudaMallocHost(&g_res.pinned, sizeof(int) * pinned_ints));
    if (!status_ok()) return false;
    g_res.pinned_ints = pinned_ints;
  }
  return status_ok();
}

// RK4 steps of one launch: long enough that loading and storing the state
// (a few us) does not show, short enough that a launch ends within
// milliseconds.
constexpr int kStepsPerLaunch = 512;

}  // namespace

void release_resident() {
  for (ResidentArea* a : {&g_res.slots[0], &g_res.slots[1], &g_res.shares, &g_res.jobs}) cudaFree(a->mem);
  cudaFree(g_res.err);
  cudaFreeHost(g_res.pinned);
  for (cudaEvent_t e : g_res.ev)
    if (e) cudaEventDestroy(e);
  g_res = ResidentWork();
}

// The layout with the shortest estimated substep, the longer of an interior and
// a radiation block's.
template <typename T>
ResPlan resident_plan(const Dims& d, int max_blocks) {
  ResPlan best;
  memset(&best, 0, sizeof(best));
  if (d.Nxx0 < 12 || d.Nxx1 < NGHOSTS || d.Nxx2 < NGHOSTS || d.Nxx2 % 2 || d.N0 != d.Nxx0 + 2 * NGHOSTS ||
      d.N1 != d.Nxx1 + 2 * NGHOSTS || d.N2 != d.Nxx2 + 2 * NGHOSTS || d.Ntot >= (1LL << 27))
    return best;
  const bool fp64 = sizeof(T) == 8;
  const int Nz = d.Nxx2, nf = fp64 ? 3 : 5;
  const size_t limit = (size_t)device_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin) - 1024;
  double best_cost = 1e300;
  for (int tx : kTX) {
    const int n0t = ceil_div(d.Nxx0, tx), rpw = 32 / tx;
    if (d.Nxx0 / n0t < NGHOSTS) continue;
    for (int n1t = 1; n1t <= d.Nxx1 / NGHOSTS && n0t * n1t < max_blocks; n1t++) {
      const int hmax = ceil_div(d.Nxx1, n1t), nrg = ceil_div(hmax, rpw);
      // radiation blocks: as many as are left, but not more than rows
      const int nrad = std::min(max_blocks - n0t * n1t, d.Nxx1);
      const int R = ceil_div(d.Nxx1, nrad);
      if (n0t * n1t > kMaxBlocks) continue;
      for (int p : kP) {
        if (nrg * ceil_div((Nz + 1) / 2, p) > kCompute / 32 || 2 * R * Nz > kThreads) continue;
        const size_t s_int = sizeof(int2) * (table_entries(10 * (hmax + tx), Nz) + 32) +
                             sizeof(T) * ((size_t)2 * Nz * (hmax + 2 * NGHOSTS) * tile_pitch(fp64, tx) + (size_t)nf * 2 * p * kCompute);
        const size_t s_rad = sizeof(int2) * table_entries(rad_entries(R), Nz) + sizeof(double) * (size_t)rad_layout(R, Nz).total;
        const size_t smem = std::max(s_int, s_rad);
        if (smem > limit) continue;
        // cycles: the block's warps share the pipes (interior: shared-memory
        // wavefronts, two per FP64 load of the 24 + 10 / p a point takes), its
        // fetches run beside that; a radiation block fetches, then computes
        const double pts = (double)std::min(tx, d.Nxx0) * hmax * Nz;
        const double c_int = 1200.0 + 500.0 * p + pts / 32.0 * (fp64 ? 2.0 : 1.0) * (28.0 + 10.0 / p);
        const double fetch = 800.0 + 300.0 * ceil_div(table_entries(10 * (hmax + tx), Nz), 8 * (kThreads - kCompute));
        const double c_rad = 1800.0 + 500.0 * ceil_div(2 * ceil_div(2 * R * Nz, 32), kThreads / 32) +
                             700.0 * ceil_div(table_entries(rad_entries(R), Nz), 4 * kThreads) +
                             8.0 * table_entries(rad_entries(R), Nz) / 32.0;
        const double cost = std::max(std::max(c_int, fetch), c_rad) + 0.1 * (c_int + fetch + c_rad);
        if (cost < best_cost) {
          best_cost = cost;
          best = {tx, p, kThreads, n0t, n1t, nrad, hmax, n0t * n1t + nrad, smem, cost};
        }
      }
    }
  }
  return best;
}
template ResPlan resident_plan<double>(const Dims&, int);
template ResPlan resident_plan<float>(const Dims&, int);

template <typename T>
bool resident_ok(const Dims& d) {
  return g_forced_tile < 0 && resident_plan<T>(d, sm_count()).blocks > 0;
}
template bool resident_ok<double>(const Dims&);
template bool resident_ok<float>(const Dims&);

int sm_count() { return device_attr(cudaDevAttrMultiProcessorCount); }

// More grids at once leave each fewer blocks, but their exchanges overlap.
template <typename T>
int resident_team(const Dims& d, int available) {
  int best = 0;
  double best_cost = 0.0;
  const int sms = sm_count();
  for (int m = 1; m <= std::min(available, 16); m++) {
    const ResPlan p = resident_plan<T>(d, sms / m);
    if (p.blocks == 0) continue;
    if (best == 0 || p.cost / m < best_cost) {
      best = m;
      best_cost = p.cost / m;
    }
  }
  return best;
}
template int resident_team<double>(const Dims&, int);
template int resident_team<float>(const Dims&, int);

template <typename T>
bool relax_resident(const std::vector<ResGrid>& grids, std::vector<RelaxResult>* results) {
  const int n = (int)grids.size();
  const int sms = sm_count();
  std::vector<ResJob<T>> jobs(n);
  size_t slot_bytes = 0, share_bytes = 0;
  std::vector<size_t> slot_off(n), share_off(n);
  ResPlan plan = resident_plan<T>(grids[0].d, sms / n);
  if (plan.blocks == 0) {
    NRPYELL_FAIL("relax_resident: the grid does not fit");
    return false;
  }
  int blocks = 0, max_steps = 0;
  using Raw = typename Tagged<T>::Raw;
  for (int i = 0; i < n; i++) {
    const ResGrid& g = grids[i];
    const Dims& d = g.d;
    ResJob<T>& J = jobs[i];
    memset(&J, 0, sizeof(J));
    J.cta0 = blocks;
    blocks += plan.blocks;
    J.n0t = plan.n0t;
    J.n1t = plan.n1t;
    J.nrad = plan.nrad;
    J.hmax = plan.hmax;
    J.Nxx0 = d.Nxx0;
    J.Nxx1 = d.Nxx1;
    J.Nxx2 = d.Nxx2;
    J.half2 = d.Nxx2 / 2;
    J.N0 = d.N0;
    J.N1 = d.N1;
    J.N01 = (long long)d.N0 * d.N1;
    J.Ntot = d.Ntot;
    J.y = (T*)g.b.y;
    J.aux = (const T*)g.b.aux;
    J.R0 = (const T*)g.b.R0;
    J.coef = sizeof(T) == 8 ? (const T*)g.rt->coef : (const T*)g.rt->coef32;
    J.colgeo = g.bt->colgeo;
    J.w = g.lt->w;
    J.xu_row = (d.Nxx0 + NGHOSTS + 1) / 2 * 2;  // rows start on a 32-byte sector
    J.xu_plane = d.Nxx1 * J.xu_row;
    J.xv_plane = d.Nxx1 * 12;
    J.xv0 = J.xu_plane * d.Nxx2;
    J.xu_slot = (long long)J.xv0 + J.xv_plane * d.Nxx2;
    slot_off[i] = slot_bytes;
    slot_bytes += align_up(sizeof(Raw) * kSlots * J.xu_slot);
    share_off[i] = share_bytes;
    share_bytes += align_up(sizeof(double2) * 2 * J.n0t * J.n1t);
    J.state = g.state;
    J.sums = g.history;
    J.volume = g.lt->volume;
    J.log10_tol = g.rp.log10_tol;
    // log10(1e-16 + sqrt(s / volume)) against the tolerance: decided by the
    // sum alone more than 1e-9 away from it.  Not where the volume is 0 (no
    // point within the integration radius: the norm is NaN and never meets a
    // tolerance) or the sum at the tolerance is no normal number.
    const double t = g.rp.log10_tol, vol = g.lt->volume;
    J.sum_met = J.sum_not_met = NAN;
    if (t > -15.0) {
      const double root = pow(10.0, t) - 1e-16, at = vol * root * root;
      if (at > 1e-300 && at < 1e300) {
        J.sum_met = at * (1.0 - 1e-9);
        J.sum_not_met = at * (1.0 + 1e-9);
      }
    } else if (t < -17.0) {
      J.sum_not_met = 0.0;
    }
    J.max_steps = g.rp.max_steps;
    J.check_every = g.rp.check_every;
    J.dt = (T)g.rp.dt;
    J.eta = (T)g.rp.eta;
    J.cOB[0] = (T)g.rp.cOB[0];
    J.cOB[1] = (T)g.rp.cOB[1];
    J.invdx0 = g.rt->invdx[0];
    J.invdx1 = g.rt->invdx[1];
    max_steps = std::max(max_steps, g.rp.max_steps);
  }
  const int stride = 4 * n;  // ints per polled launch
  constexpr bool fp64 = sizeof(T) == 8;
  if (!ensure_resident(fp64, slot_bytes, share_bytes, sizeof(ResJob<T>) * n, 2 * (stride + 1))) return false;
  for (int i = 0; i < n; i++) {
    jobs[i].xu = g_res.slots[fp64 ? 0 : 1].mem + slot_off[i];
    jobs[i].part = (double2*)(g_res.shares.mem + share_off[i]);
    jobs[i].err = g_res.err;
    NRPYELL_CUDA(cudaMemsetAsync(grids[i].state, 0, sizeof(int) * 4, stream()));
  }
  NRPYELL_CUDA(cudaMemcpyAsync(g_res.jobs.mem, jobs.data(), sizeof(ResJob<T>) * n, cudaMemcpyHostToDevice, stream()));
  ResKernel<T> kern = resident_kernel<T>(plan.tx, plan.p);
  NRPYELL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)plan.smem));
  if (!status_ok()) return false;
  const ResJob<T>* jobs_dev = (const ResJob<T>*)g_res.jobs.mem;
  int njobs = n;
  // max_steps + 1 residuals are evaluated at most; the states of a launch are
  // read while the next one runs
  long long left = (long long)max_steps + 1;
  for (long long k = 0; left > 0; k++) {
    int steps = (int)std::min<long long>(kStepsPerLaunch, left), first = (int)(kStepsPerLaunch * k);
    left -= steps;
    if (g_res.version > 0xf0000000u) {  // tags are about to wrap: start again from cleared slots
      for (const ResidentArea* a : {&g_res.slots[0], &g_res.slots[1], &g_res.shares})
        if (a->bytes) NRPYELL_CUDA(cudaMemsetAsync(a->mem, 0, a->bytes, stream()));
      g_res.version = 0;
    }
    unsigned base = g_res.version;
    g_res.version += 4 * steps;
    void* args[] = {(void*)&jobs_dev, (void*)&njobs, (void*)&base, (void*)&steps, (void*)&first};
    NRPYELL_CUDA(cudaLaunchCooperativeKernel((const void*)kern, dim3(blocks), dim3(plan.threads), args, plan.smem,
                                             stream()));
    count_launch();
    if (!status_ok()) return false;
    const int slot = (int)(k & 1);
    int* st = g_res.pinned + slot * (stride + 1);
    for (int i = 0; i < n; i++)
      NRPYELL_CUDA(cudaMemcpyAsync(st + 4 * i, grids[i].state, sizeof(int) * 4, cudaMemcpyDeviceToHost, stream()));
    NRPYELL_CUDA(cudaMemcpyAsync(st + stride, g_res.err, sizeof(int), cudaMemcpyDeviceToHost, stream()));
    NRPYELL_CUDA(cudaEventRecord(g_res.ev[slot], stream()));
    if (k > 0) {
      NRPYELL_CUDA(cudaEventSynchronize(g_res.ev[1 - slot]));
      const int* s1 = g_res.pinned + (1 - slot) * (stride + 1);
      bool all = true;
      for (int i = 0; i < n; i++) all = all && s1[4 * i + 1];
      if (all || s1[stride]) break;
    }
    if (!status_ok()) return false;
  }
  NRPYELL_CUDA(cudaStreamSynchronize(stream()));
  std::vector<int> st(4 * n);
  int err = 0;
  for (int i = 0; i < n; i++)
    NRPYELL_CUDA(cudaMemcpy(&st[4 * i], grids[i].state, sizeof(int) * 4, cudaMemcpyDeviceToHost));
  NRPYELL_CUDA(cudaMemcpy(&err, g_res.err, sizeof(int), cudaMemcpyDeviceToHost));
  if (err) {
    NRPYELL_CUDA(cudaMemsetAsync(g_res.err, 0, sizeof(int), stream()));
    NRPYELL_FAIL("on-chip relaxation: a bounded wait for a neighbouring block gave up");
  }
  if (!status_ok()) return false;
  results->assign(n, RelaxResult());
  for (int i = 0; i < n; i++) {
    const int steps = st[4 * i];
    NRPYELL_LAUNCH(k_history_log10, (steps + 256) / 256, 256, 0, grids[i].history, grids[i].lt->volume, steps + 1);
    (*results)[i].steps = steps;
    (*results)[i].converged = st[4 * i + 2] != 0;
    NRPYELL_CUDA(cudaMemcpyAsync(&(*results)[i].last_log10_l2, grids[i].history + steps, sizeof(double),
                                 cudaMemcpyDeviceToHost, stream()));
  }
  NRPYELL_CUDA(cudaStreamSynchronize(stream()));
  return status_ok();
}
template bool relax_resident<double>(const std::vector<ResGrid>&, std::vector<RelaxResult>*);
template bool relax_resident<float>(const std::vector<ResGrid>&, std::vector<RelaxResult>*);

}  // namespace nrpyell
