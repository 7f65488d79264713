// H.psi stencil pass over 16 x 16 cell tiles with the z history in tensor
// memory (sm_100a, warp-specialised).
//
// Same arithmetic and pass modes as stencil_blk.cu.  What bounds that form is
// the shared-memory pipe: 9 values read per output (2 x 2 cells per thread,
// nine running z sums per cell in registers leave no room for more) and a halo
// of 2.5 cells copied per output cell.  Here a thread owns 4 x 4 cells of one
// 8-byte element (FP64 one real lane, FP32 one complex state), which reads
// 1 + 8/4 + 8/4 = 5 values per output, and the halo of a 16 x 16 tile costs 2
// cells per cell.  The z direction needs no running sums in registers: for
// every cell the thread keeps, in its own lanes of the SM's tensor memory,
//   C(k-4 .. k-1)  the cell's values of the last four planes,
//   P(k-4 .. k-1)  the partial sums of the last four output planes: the
//                  in-plane arms, the potential and the z arms from below,
// and at plane k
//   out(k-4) = P(k-4) + sum_{j=0..3} w(4-j) C(k-j),
//   P(k)     = in-plane arms + potential + sum_{j=1..4} w(-j) C(k-j):
// five tensor-memory reads and two writes per output (rings indexed by
// k mod 4: no unrolling over the ring).  2 rings x 4 planes x 256 cells x 128
// bytes fill the 256 KB.  The planes above and below the output range need
// their own cells only, without the in-plane halo.
//
// Four producer warps gather the planes through the load map into a ring of
// three stages (zero-filling 16-byte cp.async, the map entries two planes
// ahead) and make the centre weights, once per cell; eight consumer warps
// compute.  A stage changes hands through a full barrier (every producer
// thread's copies) and an empty barrier (every consumer warp, after its last
// read of the stage); each wait is bounded and records HPSI_ERR_TIMEOUT in
// p.err.  The register split leaves the consumers 208 registers; the hand-over
// waits for local stores, so that spills in the loop over the planes cost 10-60 %.
// The apply forms have none, the FP64 Horner forms 16 bytes, the grouped kernels 16 to
// 24, with phases 76 to 120.
//
// Measured (B200, CUDA events; the blocked pass of stencil_blk.cu before):
// R = 12 sphere, 904,089 points, 128 states: apply 1.472 -> 0.984 ms FP64 (3.77
// TB/s of psi read once and H psi written once), 0.731 -> 0.517 FP32; Horner pass
// 1.688 -> 1.282 and 0.832 -> 0.664; 64^3 box, 32 states, FP64 0.114 -> 0.073 ms;
// 48^3, 16 states 0.042 -> 0.024.  On 64 planes of 16 x 16 tiles (one CTA per
// SM) the counters read: issue slots 61 %, shared-memory pipe 50 %, FP64 pipe 44 %
// busy, and an SM takes 3,700 cycles a plane step where the FP64 pipe alone needs
// 1,600: what bounds it now is the latency of two computing warps per scheduler.
// Tried and not kept: one persistent CTA per SM over a static unit list (15 %
// slower: it loses the neighbouring tiles' L2 reuse and the hardware's balancing),
// waits that sleep in hardware, loads of tensor memory that wait in one
// statement (both within 3 %).
//
// Reference semantics: X(nl_operator_operate_batch)
// (src/grid/nl_operator_inc.F90:21-130), the local potential
// (src/hamiltonian/hamiltonian_elec_base_inc.F90:233-242) and the Taylor
// axpys (src/electrons/exponential.F90:738-746).
#include "stencil_blk_impl.cuh"

namespace hpsi {

using namespace blk;

namespace {

constexpr int TM_TX = 16, TM_TY = 16, TM_HAL = 4;
constexpr int TM_R = 4;                               // cells per thread along x and y
constexpr int TM_CELLB = 128;                         // bytes of one cell chunk
constexpr int TM_BAND = TM_TX * (TM_TY + 2 * TM_HAL); // halo rows over the tile's columns
constexpr int TM_SIDE = 2 * TM_HAL * TM_TY;           // cells left and right of the tile
constexpr int TM_SC = TM_BAND + TM_SIDE;              // star cells of a plane
constexpr int TM_NC = 256, TM_NP = 128;               // consumer, producer threads
// registers a thread: at launch (the whole CTA's share), after the split
constexpr int TM_LREG = 168, TM_CREG = 208, TM_PREG = 88;
// (the grouped pass, whose arguments are indexed by system, needs more registers
// in its consumers)
constexpr int TM_GCREG = 216, TM_GPREG = 72;
static_assert(TM_NC * TM_CREG + TM_NP * TM_PREG <= (TM_NC + TM_NP) * TM_LREG, "registers of the split");
static_assert(TM_NC * TM_GCREG + TM_NP * TM_GPREG <= (TM_NC + TM_NP) * TM_LREG, "registers of the grouped split");
constexpr int TM_NBUF = 3;
constexpr size_t TM_OV = size_t(TM_SC) * TM_CELLB;              // centre weights of the plane
constexpr size_t TM_STAGE = TM_OV + TM_TX * TM_TY * sizeof(double);
constexpr size_t TM_OBS = TM_NBUF * TM_STAGE;                   // observable sums of the consumers
constexpr size_t TM_OBSB = size_t(TM_NC) * 3 * sizeof(double);
constexpr size_t TM_MAP = TM_OBS + TM_OBSB;                     // load map entries of the producers
constexpr size_t TM_PH = TM_MAP + 3 * TM_SC * sizeof(int);       // (rows, two planes of entries), phases of a plane's images
// output rows four planes below, in a ring of their own: they are read after the
// stage has been handed back.  Four slots: a plane's rows are overwritten by those
// of the fourth plane after it, whose copies wait for every warp to hand back the
// next plane's stage, that is to be done with this plane
constexpr size_t TM_ROWB = TM_TX * TM_TY * sizeof(int);
constexpr size_t TM_OROW = TM_PH + size_t(TM_SC) * 16;
constexpr size_t TM_BAR = TM_OROW + 4 * TM_ROWB;
constexpr size_t TM_BYTES = TM_BAR + 2 * TM_NBUF * 8 + 16;
static_assert(TM_BYTES <= 232448, "shared memory per CTA");
static_assert(TM_STAGE % 128 == 0 && TM_BAR % 16 == 0, "alignment");

// tensor memory: 32 columns (16 cells x 8 bytes) per slot
__device__ __forceinline__ void tm_load(uint32_t addr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr));
}
// the loaded registers pass through the wait, so that no use moves above it
__device__ __forceinline__ void tm_wait_load(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                 "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]),
                 "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29])
               :
               : "memory");
  asm volatile("" : "+r"(r[30]), "+r"(r[31]) : : "memory");
}
__device__ __forceinline__ void tm_store(uint32_t addr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};\n" ::"r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
      "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
      "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tm_wait_store() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

__device__ __forceinline__ void unpack(const uint32_t (&r)[32], double (&c)[16]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) c[i] = __hiloint2double(int(r[2 * i + 1]), int(r[2 * i]));
}
__device__ __forceinline__ void unpack(const uint32_t (&r)[32], float2 (&c)[16]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) c[i] = make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}
__device__ __forceinline__ void pack(const double (&c)[16], uint32_t (&r)[32]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    r[2 * i] = uint32_t(__double2loint(c[i]));
    r[2 * i + 1] = uint32_t(__double2hiint(c[i]));
  }
}
__device__ __forceinline__ void pack(const float2 (&c)[16], uint32_t (&r)[32]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    r[2 * i] = __float_as_uint(c[i].x);
    r[2 * i + 1] = __float_as_uint(c[i].y);
  }
}
__device__ __forceinline__ double escale(double w, double v) { return w * v; }
__device__ __forceinline__ float2 escale(float w, float2 v) { return make_float2(w * v.x, w * v.y); }

// Position in the ring of stages, kept across the work units of a CTA.
struct TmemRing {
  int slot = 0;
  unsigned phase = 0;
  unsigned n = 0;     // planes so far (rows ring)
  bool dead = false;  // a wait has given up: no further waits
  __device__ __forceinline__ int *rows(unsigned char *smem) const {
    return reinterpret_cast<int *>(smem + TM_OROW + (n & 3u) * TM_ROWB);
  }
  __device__ __forceinline__ void next() {
    ++n;
    if (++slot == TM_NBUF) {
      slot = 0;
      phase ^= 1u;
    }
  }
  // PAUSE: producers pause between polls, which would take issue slots from
  // the consumers on the same schedulers
  template <bool PAUSE>
  __device__ __forceinline__ void wait(uint64_t *bar, unsigned parity, int *err) {
    if (dead) return;
    unsigned n = 0;
    while (!mbar_try_wait(bar, parity)) {
      if (++n == TMA_WAIT_LIMIT) {
        dead = true;
        if (err) atomicExch(err, HPSI_ERR_TIMEOUT);
        return;
      }
      if constexpr (PAUSE) __nanosleep(64);
    }
  }
};
// full barrier of a stage, or its empty barrier
template <bool EMPTY>
__device__ __forceinline__ uint64_t *smem_bar(unsigned char *smem, int b) {
  return reinterpret_cast<uint64_t *>(smem + TM_BAR) + (EMPTY ? TM_NBUF : 0) + b;
}

// Producer side of one work unit (tile column over a z range, one state chunk).
// TMA: a run of eight cells of a halo row that are eight consecutive rows of
// the batch (bit of p.seg_mask; segments of the tile's columns only) arrives as
// one box copy of 8 rows x 128 bytes on the stage's full barrier.
// PH: the pass has Bloch phases.
template <typename T, bool TMA, bool PH>
__device__ __forceinline__ void tmem_produce(const PassArgs &p, const int ih, const int chunk, unsigned char *smem,
                                             TmemRing &ring, const CUtensorMap *tm = nullptr) {
  constexpr int HAL = TM_HAL;
  constexpr int SL = TM_CELLB / int(sizeof(T));  // reals per cell chunk
  const CellBox &B = p.box;
  const int4 it = p.items[ih];
  const int cx0 = HAL + it.x * TM_TX, cy0 = HAL + it.y * TM_TY;
  const int zs = it.z, ze = it.w;
  const int zbeg = zs - HAL, nplanes = ze - zs + 2 * HAL;
  const int tid = threadIdx.x, lane = tid & 31;
  const int left = p.lanes - chunk * SL;  // reals of the batch from this chunk on (the last chunk may be partial)
  const int col = chunk * SL;
  const long long planeN = (long long)B.NX * B.NY;
  // warp pw copies star cells 128 pw .. 128 pw + 127 (band rows 8 pw .. for
  // pw < 3, the side cells for pw = 3); lane i holds the map entries of the
  // four x-consecutive cells 4 i .. 4 i + 3 of them
  const int pt = tid - TM_NC, pw = pt >> 5;
  const int c0 = 128 * pw + 4 * lane;
  int my, mx;
  if (pw < 3) {
    my = c0 / TM_TX;
    mx = HAL + c0 % TM_TX;
  } else {
    const int s = c0 - TM_BAND;
    my = HAL + s / (2 * HAL);
    mx = (s & 4) ? HAL + TM_TX : 0;
  }
  const int *map = p.cell_src + (long long)(cy0 - HAL + my) * B.NX + cx0 - HAL + mx;
  const int piece = lane & 7, sub = lane >> 3;
  constexpr int EPP = 16 / int(sizeof(T));
  // pieces past the batch width are zero-filled
  const bool pok = piece * EPP < left;
  const int csize = pok ? 16 : 0;
  const T *in_base = static_cast<const T *>(p.in) + (pok ? col + piece * EPP : 0);
  const char *in_bytes = reinterpret_cast<const char *>(in_base);
  const unsigned in_rb = unsigned(2 * p.in_ld) * unsigned(sizeof(T));
  // centre weights (weight + potential + field): 128 pairs of cells; output
  // rows: 64 pieces of four cells
  const int vx = cx0 + (2 * pt) % TM_TX, vy = cy0 + (2 * pt) / TM_TX;
  const double2 *v_at = p.v_cell ? reinterpret_cast<const double2 *>(p.v_cell + (long long)vy * B.NX + vx) : nullptr;
  const long long r_src = (long long)(cy0 + (4 * pt) / TM_TX) * B.NX + cx0 + (4 * pt) % TM_TX;
  const double fscale = p.fld_scale_dev ? *p.fld_scale_dev : 1.0;
  const double fz = p.fld[2] * fscale * B.h[2], fx = fscale * p.fld[0] * B.h[0], fy = fscale * p.fld[1] * B.h[1];
  const double fxy = fx * double(vx + B.lo[0]) + fy * double(vy + B.lo[1]);
  const bool has_field = fz != 0.0 || fx != 0.0 || fy != 0.0;
  auto v_load = [&](int q) {
    return v_at && q >= zs && q < ze ? __ldg(v_at + (long long)q * (planeN / 2)) : make_double2(0.0, 0.0);
  };
  // Bloch phases: an entry <= -2 names a boundary point, whose image row is
  // copied like any other row; the copy is multiplied by the point's phase in
  // shared memory once it has landed, one plane after it was issued, before the
  // stage is handed over (`ent`: the plane's entries, double-buffered)
  int4 *mapw = reinterpret_cast<int4 *>(smem + TM_MAP) + 32 * pw;  // this warp's rows of the plane
  [[maybe_unused]] int4 *ent = mapw + TM_SC / 4;
  auto image = [&](int e) { return e >= -1 ? e : __ldg(p.per_inner - (e + 2)); };
  [[maybe_unused]] auto images4 = [&](const int4 &e) { return PH ? make_int4(image(e.x), image(e.y), image(e.z), image(e.w)) : e; };
  // phases of this warp's images, staged before the plane is finished
  using C = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
  [[maybe_unused]] C *phw = reinterpret_cast<C *>(smem + TM_PH) + 128 * pw;
  [[maybe_unused]] auto phase_of = [&](int e) {
    C c;
    c.x = 1;
    c.y = 0;
    return e >= -1 ? c : __ldg(static_cast<const C *>(p.phase_corr) - ((long long)e + 2));
  };
  [[maybe_unused]] int pslot = -1, pq0 = 0, pq1 = 0, pent = 0;  // plane waiting for its phases
  [[maybe_unused]] auto finish = [&]() {
    unsigned char *d0 = smem + size_t(pslot) * TM_STAGE + (size_t(128 * pw) + 4 * sub) * TM_CELLB + piece * 16;
    const int4 *pe = ent + pent * (TM_SC / 4);
    if (pq1 > pq0) {
      const int4 e = pe[lane];
      const C c0 = phase_of(e.x), c1 = phase_of(e.y), c2 = phase_of(e.z), c3 = phase_of(e.w);
      __syncwarp();
      phw[4 * lane] = c0;
      phw[4 * lane + 1] = c1;
      phw[4 * lane + 2] = c2;
      phw[4 * lane + 3] = c3;
      __syncwarp();
    }
    for (int g = pq0; g < pq1; ++g) {
      const int4 m4 = pe[4 * g + sub];
      const int src[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (src[j] >= -1 || !pok) continue;
        T *e = reinterpret_cast<T *>(d0 + size_t(16 * g + j) * TM_CELLB);
        const C ph = phw[16 * g + 4 * sub + j];
#pragma unroll
        for (int i = 0; i < EPP; i += 2) {
          const T xr = e[i], xi = e[i + 1];
          e[i] = xr * ph.x - xi * ph.y;
          e[i + 1] = xr * ph.y + xi * ph.x;
        }
      }
    }
    mbar_arrive(smem_bar<false>(smem, pslot));
    mbar_arrive(smem_bar<false>(smem, pslot));
  };

  auto entries = [&](int q) { return *reinterpret_cast<const int4 *>(map + (long long)q * planeN); };
  // The loads of the next planes: an arrival (release) waits for the thread's
  // loads in flight.  In the first planes they are issued after it, so that the
  // ring fills at once; later before it, which holds the next plane's copies back
  // until the consumers are past their shared-memory loads (R = 12 sphere, 128
  // states, FP64: 0.98 ms; issued after it throughout: 1.14 ms, and in the small
  // boxes of 6-plane units 0.026 -> 0.024 ms).
  int4 cur = entries(zbeg), nxt = nplanes > 1 ? entries(zbeg + 1) : cur;
  int4 rows = images4(cur);
  double2 v = v_load(zbeg), vnxt = v_load(zbeg + 1);
  auto advance = [&](int k) {
    cur = nxt;
    rows = images4(cur);
    v = vnxt;
    if (k + 2 < nplanes) {
      nxt = entries(zbeg + k + 2);
      vnxt = v_load(zbeg + k + 2);
    }
  };
  for (int k = 0; k < nplanes; ++k) {
    const int q = zbeg + k;
    const bool inner = q >= zs && q < ze;  // the in-plane halo is read for output planes only
    // rounds of this warp that hold cells of the tile itself (band rows 4..19)
    const int q0 = inner ? 0 : pw == 0 ? 4 : pw == 3 ? 8 : 0;
    const int q1 = inner ? 8 : pw == 2 ? 4 : 8;
    __syncwarp();  // the plane before has read its entries
    mapw[lane] = PH ? rows : cur;
    [[maybe_unused]] bool images = false;  // whether the plane's rounds hold an image (uniform in the warp)
    if constexpr (PH) {
      ent[(k & 1) * (TM_SC / 4) + lane] = cur;
      images = __any_sync(0xffffffffu, lane >= 4 * q0 && lane < 4 * q1 &&
                                           (cur.x < -1 || cur.y < -1 || cur.z < -1 || cur.w < -1));
    }
    __syncwarp();
    const double2 vk = v;
    if (k >= TM_NBUF) advance(k);
    const int b = ring.slot;
    ring.wait<true>(smem_bar<true>(smem, b), ring.phase ^ 1u, p.err);  // the first round passes at once
    unsigned char *st = smem + size_t(b) * TM_STAGE;
    unsigned char *dst = st + (size_t(128 * pw) + 4 * sub) * TM_CELLB + piece * 16;
    [[maybe_unused]] unsigned boxes = 0;  // bits 2 g, 2 g + 1: the two segments of row g of this warp
    if constexpr (TMA) {
      const unsigned long long m = __ldg(p.seg_mask + (size_t(it.y) * p.seg_tiles_x + it.x) * B.NZ + q);
      boxes = pw < 3 && q1 > q0 ? unsigned(m >> (16 * pw)) & ((0xffffu >> (16 - 2 * (q1 - q0))) << (2 * q0)) : 0u;
      // the bytes of the boxes; the warp's plain arrivals all come after its stores of
      // centre weights (a release: the asynchronous arrivals order copies only)
      if (lane == 0 && boxes) mbar_expect_tx(smem_bar<false>(smem, b), unsigned(__popc(boxes)) * 8u * TM_CELLB);
      __syncwarp();
      if (lane < 16 && ((boxes >> lane) & 1u))
        tma_load_rows(st + (size_t(128 * pw) + 8 * lane) * TM_CELLB, tm, col, mapw[2 * lane].x, smem_bar<false>(smem, b));
    }
#pragma unroll 2
    for (int g = q0; g < q1; ++g) {
      if constexpr (TMA)
        if ((boxes >> (2 * g + (sub >> 1))) & 1u) continue;  // these cells arrive with their segment's box
      const int4 m4 = mapw[4 * g + sub];
      const int src[4] = {m4.x, m4.y, m4.z, m4.w};
      unsigned char *d = dst + size_t(16 * g) * TM_CELLB;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        cp_async16_zfill(d + j * TM_CELLB, in_bytes + size_t(unsigned(max(src[j], 0))) * in_rb, src[j] >= 0 ? csize : 0);
    }
    if (inner) {
      double2 c = vk;
      if (has_field) {
        const double f = fxy + fz * double(q + B.lo[2]);
        c.x += f;
        c.y += f + fx;
      }
      T *cw = reinterpret_cast<T *>(st + TM_OV) + 2 * pt;
      const T w0 = wsel_t<T>(p.wx, p.wxf, 4);
      cw[0] = w0 + static_cast<T>(c.x);
      cw[1] = w0 + static_cast<T>(c.y);
    }
    if (pt < 64 && q - HAL >= zs)
      cp_async16(ring.rows(smem) + 4 * pt, p.cell_row + (long long)(q - HAL) * planeN + r_src);
    if constexpr (PH) {
      cp_async_commit();
      if (pslot >= 0) {
        cp_async_wait<1>();
        finish();
      }
      pslot = b;
      pq0 = images ? q0 : 0;
      pq1 = images ? q1 : 0;
      pent = k & 1;
    } else {
      cp_async_arrive_noinc(smem_bar<false>(smem, b));
      mbar_arrive(smem_bar<false>(smem, b));
    }
    ring.next();
    if (k < TM_NBUF) advance(k);
  }
  if constexpr (PH) {
    if (pslot >= 0) {
      cp_async_wait<0>();
      finish();
    }
  }
}

// Consumer side of one work unit.
// CROSS: Horner pass on real lanes with a purely imaginary factor: the lane
// that holds one part of H psi writes the other part of the output, so the
// lanes exchange nothing.
// pw: the arguments that hold the weights (at a fixed parameter address).
// RHO: also the density of the outputs, per row and chunk (p.rho_part).
template <typename T, bool HORNER, bool OBS, bool CROSS, bool RHO>
__device__ __forceinline__ void tmem_consume(const PassArgs &p, const PassArgs &pw, const int ih, const int chunk,
                                             unsigned char *smem, const uint32_t tm_base, TmemRing &ring) {
  constexpr bool CPLX = sizeof(T) == 4;
  constexpr bool X0 = HORNER || OBS;
  using E = typename BlkElem<T, CPLX>::E;
  static_assert(sizeof(E) == 8, "8-byte elements");
  static_assert(!CROSS || (HORNER && !OBS && !CPLX), "real lanes only");
  constexpr int SL = TM_CELLB / int(sizeof(T));  // reals per cell chunk
  constexpr int SLE = TM_CELLB / 8;              // elements per cell chunk
  constexpr int HAL = TM_HAL, R = TM_R;
  const CellBox &B = p.box;
  const int4 it = p.items[ih];
  const int cx0 = HAL + it.x * TM_TX, cy0 = HAL + it.y * TM_TY;
  const int zs = it.z, ze = it.w;
  const int zbeg = zs - HAL, nplanes = ze - zs + 2 * HAL;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int left = p.lanes - chunk * SL;  // reals of the batch from this chunk on (the last chunk may be partial)
  const int l = lane & 15;
  // the two warps of a scheduler (w, w + 4) take opposite halves of the tile
  // in x: on a partly filled tile the work spreads over the schedulers (7 %
  // fewer plane steps on the busiest one, R = 12 sphere)
  const int g = 2 * (warp ^ (warp >> 2)) + (lane >> 4);
  const int bx = (g & 3) * R, by = (g >> 2) * R;
  const uint32_t tm = tm_base + (uint32_t(32 * (warp & 3)) << 16) + uint32_t(256 * (warp >> 2));
  const T are = static_cast<T>(p.a_re), aim = static_cast<T>(p.a_im);
  const bool odd = !CPLX && (l & 1) != 0;
  const T caim = odd ? -aim : aim;
  const int oelem = chunk * SLE + (CROSS ? (l ^ 1) : l);
  const bool lok = l * (8 / int(sizeof(T))) < left;  // both parts of a state lie on the same side of the width
  // outputs of lanes past the width count as outside the mesh
  const unsigned rows_np = lok ? unsigned(p.np) : 0u;
  char *out_bytes = static_cast<char *>(p.out) + size_t(oelem) * 8;
  const unsigned out_rb = unsigned(2 * p.out_ld) * unsigned(sizeof(T));
  const char *x0_at = static_cast<const char *>(p.psi0) + (lok ? size_t(oelem) * 8 : 0);
  const unsigned x0_rb = unsigned(2 * p.psi0_ld) * unsigned(sizeof(T));
  // density weight of this lane's state
  [[maybe_unused]] const double wrho = RHO && lok ? p.rho_w[chunk * (SL / 2) + (CPLX ? l : l / 2)] : 0.0;
  double se = 0.0, sn = 0.0, sd = 0.0;
  const double dxy00 = OBS ? p.obs_pol[0] * B.h[0] * double(cx0 + bx + B.lo[0]) +
                                 p.obs_pol[1] * B.h[1] * double(cy0 + by + B.lo[1])
                           : 0.0;

  // z range of the inner points under the warp's cells: it computes the
  // output planes [ws, we) and reads the planes up to four beyond them
  int ws = 1 << 30, we = -(1 << 30);
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int cx = 0; cx < R; ++cx) {
      const int2 cz = __ldg(p.col_z + (long long)(cy0 + by + r) * B.NX + cx0 + bx + cx);
      ws = min(ws, cz.x);
      we = max(we, cz.y + 1);
    }
  ws = max(zs, __reduce_min_sync(0xffffffffu, ws));
  we = min(ze, __reduce_max_sync(0xffffffffu, we));

  // byte offsets in a stage: own cells, left and right neighbours (in the
  // band, or the side cells at the tile's edge)
  const int own = ((by + HAL) * TM_TX + bx) * TM_CELLB + l * 8;
  const int lefto = bx == 0 ? (TM_BAND + by * 2 * HAL) * TM_CELLB + l * 8 : own - HAL * TM_CELLB;
  const int lstep = (bx == 0 ? 2 * HAL : TM_TX) * TM_CELLB;
  const int righto = bx + R == TM_TX ? (TM_BAND + by * 2 * HAL + HAL) * TM_CELLB + l * 8 : own + R * TM_CELLB;
  const int rstep = (bx + R == TM_TX ? 2 * HAL : TM_TX) * TM_CELLB;

#pragma unroll 1
  for (int k = 0; k < nplanes; ++k) {
    const int b = ring.slot;
    const int pz = zbeg + k;
    ring.wait<false>(smem_bar<false>(smem, b), ring.phase, p.err);
    const unsigned char *st = smem + size_t(b) * TM_STAGE;
    const int *rows = ring.rows(smem);
    const bool need = pz >= ws - HAL && pz < we + HAL;  // warp-uniform
    const bool work = need && pz >= ws;
    const bool emit = work && pz - HAL >= ws;  // output plane pz - 4 completes here
    E c[16], a[16];                            // C(k), P(k)
    E x0[16];
    if (need) {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int cx = 0; cx < R; ++cx)
          c[r * R + cx] = *reinterpret_cast<const E *>(st + own + (r * TM_TX + cx) * TM_CELLB);
    }
    if (emit) {
      // rows of the output plane
            if constexpr (X0) {
        // lane i of a cell group fetches cell i's psi0 line to L2: it is read
        // after the in-plane arms (a load in flight across the hand-over of
        // the stage would delay it)
        const int mine = rows[(by + (l >> 2)) * TM_TX + bx + (l & 3)];
        if (unsigned(mine) < unsigned(p.np))
          asm volatile("prefetch.global.L2 [%0];\n" ::"l"(static_cast<const char *>(p.psi0) + size_t(chunk) * TM_CELLB +
                                                         size_t(unsigned(mine)) * x0_rb));
      }
    }
    if (work) {
#pragma unroll
      for (int i = 0; i < 16; ++i) a[i] = ezero<E>();
      if (pz < we) {
        // the arms inside the 4 x 4 block
#pragma unroll
        for (int i = 0; i < R * R; ++i)
          a[i] = escale(wsel_t<T>(pw.wx, pw.wxf, (i & 1) ? 3 : 5), c[i ^ 1]);
#pragma unroll
        for (int d = 1; d < R; ++d)
#pragma unroll
          for (int i = 0; i < R; ++i)
#pragma unroll
            for (int j = 0; j + d < R; ++j) {
              // cells j and j + d of a row / column i
              if (d > 1 || j % 2 == 1) {  // (the others came first)
                a[i * R + j] = fmae(wsel_t<T>(pw.wx, pw.wxf, 4 + d), c[i * R + j + d], a[i * R + j]);
                a[i * R + j + d] = fmae(wsel_t<T>(pw.wx, pw.wxf, 4 - d), c[i * R + j], a[i * R + j + d]);
              }
              a[j * R + i] = fmae(wsel_t<T>(pw.wy, pw.wyf, 4 + d), c[(j + d) * R + i], a[j * R + i]);
              a[(j + d) * R + i] = fmae(wsel_t<T>(pw.wy, pw.wyf, 4 - d), c[j * R + i], a[(j + d) * R + i]);
            }
        // y arms from above and below the block
#pragma unroll
        for (int i = 0; i < HAL; ++i)
#pragma unroll
          for (int cx = 0; cx < R; ++cx) {
            const E lo = *reinterpret_cast<const E *>(st + own + ((i - HAL) * TM_TX + cx) * TM_CELLB);
            const E hi = *reinterpret_cast<const E *>(st + own + ((i + R) * TM_TX + cx) * TM_CELLB);
#pragma unroll
            for (int r = 0; r < R; ++r) {
              if (i - HAL - r >= -HAL)
                a[r * R + cx] = fmae(wsel_t<T>(pw.wy, pw.wyf, i - r), lo, a[r * R + cx]);
              if (i + R - r <= HAL)
                a[r * R + cx] = fmae(wsel_t<T>(pw.wy, pw.wyf, i + R - r + 4), hi, a[r * R + cx]);
            }
          }
        // x arms from left and right of the block
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int i = 0; i < HAL; ++i) {
            const E lo = *reinterpret_cast<const E *>(st + lefto + r * lstep + i * TM_CELLB);
            const E hi = *reinterpret_cast<const E *>(st + righto + r * rstep + i * TM_CELLB);
#pragma unroll
            for (int cx = 0; cx < R; ++cx) {
              if (i - HAL - cx >= -HAL)
                a[r * R + cx] = fmae(wsel_t<T>(pw.wx, pw.wxf, i - cx), lo, a[r * R + cx]);
              if (i + R - cx <= HAL)
                a[r * R + cx] = fmae(wsel_t<T>(pw.wx, pw.wxf, i + R - cx + 4), hi, a[r * R + cx]);
            }
          }
        // the centre after the in-plane arms: it cancels most of their sum, so the
        // z arms are added to a small number (FP32 rounding error of H psi 1.6e-7,
        // with the centre first 2.1e-7)
        const T *cw = reinterpret_cast<const T *>(st + TM_OV) + by * TM_TX + bx;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          T w[R];
          if constexpr (CPLX) {
            const float4 t = *reinterpret_cast<const float4 *>(cw + r * TM_TX);
            w[0] = t.x, w[1] = t.y, w[2] = t.z, w[3] = t.w;
          } else {
            const double2 t = *reinterpret_cast<const double2 *>(cw + r * TM_TX);
            const double2 u = *reinterpret_cast<const double2 *>(cw + r * TM_TX + 2);
            w[0] = t.x, w[1] = t.y, w[2] = u.x, w[3] = u.y;
          }
#pragma unroll
          for (int cx = 0; cx < R; ++cx) a[r * R + cx] = fmae(w[cx], c[r * R + cx], a[r * R + cx]);
        }
      }

    }
    // the stage has been read: it is handed back before the z arms, so that the
    // producers' copies overlap the z arms and not the next plane's loads from
    // shared memory
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_bar<true>(smem, b));

    const uint32_t slot = uint32_t(k & 3) * 32u;
    uint32_t buf[32], buf2[32];
    tm_wait_store();  // of the plane before
    if (work) {
      if constexpr (X0) {
        if (emit) {
          // rows outside the mesh read row 0 (not used)
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int4 v = *reinterpret_cast<const int4 *>(rows + (by + r) * TM_TX + bx);
            const int row[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < R; ++i)
              x0[r * R + i] = *reinterpret_cast<const E *>(
                  x0_at + size_t(unsigned(row[i]) < rows_np ? unsigned(row[i]) : 0u) * x0_rb);
          }
        }
      }
      // z arms: C(k-1 .. k-4) feed P(k) and, with C(k), out(k-4); each load
      // is in flight during the sums of the one before
      E o[16], u[16];
      tm_load(tm + 128u + slot, buf);                   // P(k-4)
      tm_load(tm + uint32_t((k - 1) & 3) * 32u, buf2);  // C(k-1)
      tm_wait_load(buf);
      tm_wait_load(buf2);
      unpack(buf, o);
#pragma unroll
      for (int i = 0; i < 16; ++i) o[i] = fmae(wsel_t<T>(pw.wz, pw.wzf, 8), c[i], o[i]);
      auto zarm = [&](auto Jc, const E (&v)[16]) {
        constexpr int J = decltype(Jc)::value;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          a[i] = fmae(wsel_t<T>(pw.wz, pw.wzf, 4 - J), v[i], a[i]);
          if (J < HAL) o[i] = fmae(wsel_t<T>(pw.wz, pw.wzf, 8 - J), v[i], o[i]);
        }
      };
      tm_load(tm + uint32_t((k - 2) & 3) * 32u, buf);
      unpack(buf2, u);
      zarm(std::integral_constant<int, 1>{}, u);
      tm_wait_load(buf);
      tm_load(tm + uint32_t((k - 3) & 3) * 32u, buf2);
      unpack(buf, u);
      zarm(std::integral_constant<int, 2>{}, u);
      tm_wait_load(buf2);
      tm_load(tm + slot, buf);  // C(k-4)
      unpack(buf2, u);
      zarm(std::integral_constant<int, 3>{}, u);
      tm_wait_load(buf);
      unpack(buf, u);
      zarm(std::integral_constant<int, 4>{}, u);
      // the slots of C(k-4) and P(k-4) take plane k
      pack(c, buf);
      tm_store(tm + slot, buf);
      pack(a, buf2);
      tm_store(tm + 128u + slot, buf2);
      if (emit) {
        [[maybe_unused]] double rc[16];  // this lane's share of the cells' density
        double pe = 0.0, pn = 0.0, pd = 0.0;
        int4 rv;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (i % R == 0) rv = *reinterpret_cast<const int4 *>(rows + (by + i / R) * TM_TX + bx);
          const int row = i % R == 0 ? rv.x : i % R == 1 ? rv.y : i % R == 2 ? rv.z : rv.w;
          const E h = o[i];
          E val = h;
          if constexpr (HORNER) {
            if constexpr (CPLX) {
              val.x = x0[i].x + are * h.x - aim * h.y;
              val.y = x0[i].y + are * h.y + aim * h.x;
            } else if constexpr (CROSS) {
              val = fma(caim, h, x0[i]);
            } else {
              const T hp = __shfl_xor_sync(0xffffffffu, h, 1);  // the other part of this state
              val = odd ? x0[i] + are * h + aim * hp : x0[i] + are * h - aim * hp;
            }
          }
          const bool ok = unsigned(row) < rows_np;
          if constexpr (RHO) {
            if constexpr (CPLX)
              rc[i] = ok ? wrho * (double(val.x) * double(val.x) + double(val.y) * double(val.y)) : 0.0;
            else
              rc[i] = ok ? wrho * double(val) * double(val) : 0.0;
          }
          if (ok) {
            if constexpr (OBS) {
              double eh, n2;
              if constexpr (CPLX) {
                eh = double(x0[i].x) * double(h.x) + double(x0[i].y) * double(h.y);
                n2 = double(x0[i].x) * double(x0[i].x) + double(x0[i].y) * double(x0[i].y);
              } else {
                eh = double(x0[i]) * double(h);
                n2 = double(x0[i]) * double(x0[i]);
              }
              pe += eh;
              pn += n2;
              pd += n2 * (double(i % R) * (p.obs_pol[0] * B.h[0]) + double(i / R) * (p.obs_pol[1] * B.h[1]));
            }
            *reinterpret_cast<E *>(out_bytes + size_t(unsigned(row)) * out_rb) = val;
          }
        }
        if constexpr (RHO) {
          // sums over the 16 lanes of the chunk: a transposing butterfly halves
          // the cells a lane holds at each step; lane l ends with one cell's total
          int cell = 0;
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const int half = 8 >> t, off = 8 >> t;
            const bool hi = (l & off) != 0;
#pragma unroll
            for (int j = 0; j < half; ++j) {
              const double send = hi ? rc[j] : rc[j + half];
              const double keep = hi ? rc[j + half] : rc[j];
              rc[j] = keep + __shfl_xor_sync(0xffffffffu, send, off);
            }
            if (hi) cell += half;
          }
          const int row = rows[(by + cell / R) * TM_TX + bx + cell % R];
          if (unsigned(row) < unsigned(p.np)) p.rho_part[(long long)chunk * p.np + row] = rc[0];
        }
        if constexpr (OBS) {
          se += pe;
          sn += pn;
          sd += pn * (dxy00 + p.obs_pol[2] * B.h[2] * double(pz - HAL + B.lo[2])) + pd;
        }
      }
    } else if (need) {
      pack(c, buf);
      tm_store(tm + slot, buf);
    }
    ring.next();
  }
  tm_wait_store();

  if constexpr (OBS) {
    double *red = reinterpret_cast<double *>(smem + TM_OBS);
    red[tid * 3] = se;
    red[tid * 3 + 1] = sn;
    red[tid * 3 + 2] = sd;
    asm volatile("bar.sync 1, 256;\n" ::: "memory");
    if (tid < SL / 2 && 2 * tid < left) {
      constexpr int LW = CPLX ? 1 : 2;  // elements per state
      Kahan s[3] = {{0, 0}, {0, 0}, {0, 0}};
      for (int t = LW * tid; t < TM_NC; t += SLE)
        for (int q = 0; q < LW; ++q)
#pragma unroll
          for (int i = 0; i < 3; ++i) kadd(s[i], red[(t + q) * 3 + i]);
      double *ob = p.obs + ((long long)ih * p.obs_ld + chunk * (SL / 2) + tid) * 6;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        ob[2 * i] = s[i].s;
        ob[2 * i + 1] = s[i].c;
      }
    }
  }
}

// Shared set-up and end of a CTA: tensor memory, barriers, register split.
__device__ __forceinline__ uint32_t tmem_begin(unsigned char *smem) {
  uint32_t *tm_addr = reinterpret_cast<uint32_t *>(smem + TM_BAR + 2 * TM_NBUF * 8);
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(
                     static_cast<unsigned>(__cvta_generic_to_shared(tm_addr)))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (threadIdx.x == 0) {
    for (int b = 0; b < TM_NBUF; ++b) {
      mbar_init(smem_bar<false>(smem, b), 2 * TM_NP);
      mbar_init(smem_bar<true>(smem, b), TM_NC / 32);
    }
    mbar_init_fence();
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  return *tm_addr;
}
__device__ __forceinline__ void tmem_end(uint32_t tm_base) {
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(tm_base));
  }
}

// grid: nitems * chunks
template <typename T, bool HORNER, bool OBS, bool CROSS, bool RHO, bool TMA, bool PH>
__global__ void __launch_bounds__(TM_NC + TM_NP, 1) pass_tmem_kernel(const __grid_constant__ PassArgs p,
                                                                    const __grid_constant__ CUtensorMap tm) {
  extern __shared__ __align__(128) unsigned char smem[];
  const uint32_t tm_base = tmem_begin(smem);
  const int ih = blockIdx.x / p.chunks, chunk = blockIdx.x % p.chunks;
  TmemRing ring;
  if (threadIdx.x >= TM_NC) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(TM_PREG));
    tmem_produce<T, TMA, PH>(p, ih, chunk, smem, ring, &tm);
    // the copies have landed before the CTA ends
    cp_async_commit();
    cp_async_wait<0>();
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(TM_CREG));
    tmem_consume<T, HORNER, OBS, CROSS, RHO>(p, p, ih, chunk, smem, tm_base, ring);
  }
  tmem_end(tm_base);
}

// Many systems in one launch (Horner passes): CTA i takes the units
// first[i] .. first[i + 1] - 1 of the list; the producers run on into the next
// unit while the consumers finish one.
// WEQ: every system has the weights of the first (equal spacings): they are
// read at a fixed parameter address instead of through the system's index.
template <typename T, bool PH, bool WEQ>
__global__ void __launch_bounds__(TM_NC + TM_NP, 1) pass_tmem_group_kernel(const __grid_constant__ GroupArgs g) {
  extern __shared__ __align__(128) unsigned char smem[];
  const uint32_t tm_base = tmem_begin(smem);
  const int u0 = g.first[blockIdx.x], u1 = g.first[blockIdx.x + 1];
  TmemRing ring;
  if (threadIdx.x >= TM_NC) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(TM_GPREG));
    for (int u = u0; u < u1; ++u) {
      const int4 W = g.units[u];  // {system, item, chunk, -}
      tmem_produce<T, false, PH>(g.sys[W.x], W.y, W.z, smem, ring);
    }
    cp_async_commit();
    cp_async_wait<0>();
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(TM_GCREG));
    for (int u = u0; u < u1; ++u) {
      const int4 W = g.units[u];
      tmem_consume<T, true, false, sizeof(T) == 8, false>(g.sys[W.x], WEQ ? g.sys[0] : g.sys[W.x], W.y, W.z, smem,
                                                            tm_base, ring);
    }
  }
  tmem_end(tm_base);
}

template <class K>
cudaError_t tmem_kernel_setup(K kern, int &regs) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(TM_BYTES));
  cudaFuncAttributes fa;
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, kern);
  if (e == cudaSuccess) regs = fa.numRegs;
  return e;
}
hpsi_status tmem_regs_ok(int regs) {
  if (regs >= TM_LREG) return HPSI_OK;
  // the consumers' larger share would never be granted
  set_error("launch_pass_tmem: compiled with too few registers for the split");
  return HPSI_ERR_UNSUPPORTED;
}

template <typename T, bool HORNER, bool OBS, bool CROSS, bool RHO, bool TMA, bool PH>
hpsi_status launch_tmem_mode(const PassArgs &a, const CUtensorMap *tm, cudaStream_t st) {
  auto kern = pass_tmem_kernel<T, HORNER, OBS, CROSS, RHO, TMA, PH>;
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  static int regs = 0;
  std::call_once(once, [&] { attr = tmem_kernel_setup(kern, regs); });
  HPSI_TRY_CUDA(attr);
  if (hpsi_status r = tmem_regs_ok(regs)) return r;
  if (!blk_strides_ok<T>(a)) return HPSI_ERR_ARG;
  CUtensorMap none;
  std::memset(&none, 0, sizeof(none));
  kern<<<unsigned(a.nitems) * unsigned(a.chunks), TM_NC + TM_NP, TM_BYTES, st>>>(a, tm ? *tm : none);
  HPSI_CHECK_LAUNCH();
  return HPSI_OK;
}

template <typename T, bool TMA, bool PH>
hpsi_status launch_tmem_f(const PassArgs &a, const CUtensorMap *tm, cudaStream_t st) {
  constexpr bool REAL = sizeof(T) == 8;
  const bool horner = a.mode == PASS_HORNER, obs = a.obs != nullptr, rho = a.rho_part != nullptr;
  if (rho) {
    if (!horner || obs) {
      set_error("launch_pass_tmem: the density is fused into Horner passes without observables only");
      return HPSI_ERR_UNSUPPORTED;
    }
    if (REAL && a.a_re == 0.0) return launch_tmem_mode<T, true, false, REAL, true, TMA, PH>(a, tm, st);
    return launch_tmem_mode<T, true, false, false, true, TMA, PH>(a, tm, st);
  }
  if (horner && obs) return launch_tmem_mode<T, true, true, false, false, TMA, PH>(a, tm, st);
  if (horner && REAL && a.a_re == 0.0) return launch_tmem_mode<T, true, false, REAL, false, TMA, PH>(a, tm, st);
  if (horner) return launch_tmem_mode<T, true, false, false, false, TMA, PH>(a, tm, st);
  if (obs) return launch_tmem_mode<T, false, true, false, false, TMA, PH>(a, tm, st);
  return launch_tmem_mode<T, false, false, false, false, TMA, PH>(a, tm, st);
}

template <typename T, bool PH, bool WEQ>
hpsi_status launch_tmem_group_f(const GroupArgs &g, int grid, cudaStream_t st) {
  auto kern = pass_tmem_group_kernel<T, PH, WEQ>;
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  static int regs = 0;
  std::call_once(once, [&] { attr = tmem_kernel_setup(kern, regs); });
  HPSI_TRY_CUDA(attr);
  if (hpsi_status r = tmem_regs_ok(regs)) return r;
  kern<<<grid, TM_NC + TM_NP, TM_BYTES, st>>>(g);
  HPSI_CHECK_LAUNCH();
  return HPSI_OK;
}

}  // namespace

template <typename T>
hpsi_status launch_pass_tmem_group(const GroupArgs &g, int grid, cudaStream_t st) {
  if (g.nunits == 0) return HPSI_OK;
  bool phased = false, weq = true;
  for (int s = 0; s < GROUP_MAX && g.sys[s].in != nullptr; ++s) {
    if (!blk_strides_ok<T>(g.sys[s])) return HPSI_ERR_ARG;
    phased = phased || g.sys[s].phase_corr != nullptr;
    weq = weq && std::memcmp(g.sys[s].wx, g.sys[0].wx, sizeof(g.sys[0].wx)) == 0 &&
          std::memcmp(g.sys[s].wy, g.sys[0].wy, sizeof(g.sys[0].wy)) == 0 &&
          std::memcmp(g.sys[s].wz, g.sys[0].wz, sizeof(g.sys[0].wz)) == 0;
    if (g.sys[s].a_re != 0.0 && sizeof(T) == 8) {
      set_error("launch_pass_tmem_group: purely imaginary Horner factors only");
      return HPSI_ERR_UNSUPPORTED;
    }
  }
  if (phased) return launch_tmem_group_f<T, true, false>(g, grid, st);
  return weq ? launch_tmem_group_f<T, false, true>(g, grid, st) : launch_tmem_group_f<T, false, false>(g, grid, st);
}
template hpsi_status launch_pass_tmem_group<double>(const GroupArgs &, int, cudaStream_t);
template hpsi_status launch_pass_tmem_group<float>(const GroupArgs &, int, cudaStream_t);

template <typename T>
hpsi_status launch_pass_tmem(const PassArgs &a, const CUtensorMap *tm, cudaStream_t st) {
  if (a.nitems == 0) return HPSI_OK;
  if (tm && (!a.seg_mask || a.phase_corr)) {
    set_error("launch_pass_tmem: TMA fill without its segment masks, or with Bloch phases");
    return HPSI_ERR_ARG;
  }
  if (a.phase_corr) return launch_tmem_f<T, false, true>(a, nullptr, st);
  return tm ? launch_tmem_f<T, true, false>(a, tm, st) : launch_tmem_f<T, false, false>(a, tm, st);
}
template hpsi_status launch_pass_tmem<double>(const PassArgs &, const CUtensorMap *, cudaStream_t);
template hpsi_status launch_pass_tmem<float>(const PassArgs &, const CUtensorMap *, cudaStream_t);

}  // namespace hpsi
