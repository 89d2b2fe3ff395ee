// The wide kernel's first way with a row: one pass over it, where the row is such that one pass can serve it. (Included by sample_wide.cuh inside its namespace, once per
// instance.)
//
// One pass sums the mass of everything (S) with the fast exponential relative to an anchor near the row maximum. With a top-p
// cut, a sample of the row places the cut in a window of logit values; the window's own logits go to lists, and the cut is
// decided exactly among them. What lies above the window is certainly kept: its mass is summed beside S (P1_MID), or, where few
// logits lie below the window, they are listed too and the rest of S is what is kept (P1_LOW: a quarter fewer instructions
// in a loop that is bound by their issue where an SM has four rows). The sample only chooses the window: whether the cut really
// lies inside is checked on the sums of the whole row, and a row whose window failed (or that the sample cannot place:
// a few heavy tokens, NaN, a wide window) takes two passes (sample_wide.cuh). Rows without a cut need neither sample
// nor window. Long ones whose maximum lies where a first look expects it are flat, many tokens share the mass, and the fast
// exponential serves them (P1_ALL); short ones, and those in which a logit turns up more than 2 above that, get exact sums
// (P1_EXACT), which cost twice the instructions. (us, flat rows, and rows with 16 peaks of 8 on a sigma of 2, the latter by exact sums and as two passes
// over the row: 512 x 151,936 f32 68, 91, 210, bf16 52, 88, 161; 256 x 50,257 f32 23, 29, 51.)
//
// The lists. A window of 1 to 2 % of the logits puts one into a tenth of the lane-steps, so nearly every warp-step has a lane
// that must list something, and slots from a shared counter cost every warp some ninety issue slots a step. So a lane has a
// buffer of its own: a predicated store and a predicated addition per logit, no branch, no counter, consecutive lanes in
// consecutive banks. At the end of a piece (of every turn of the ring, where the window is wide) the warp moves what its lanes hold to its list, a vote per round. What is listed is
// the logit alone: its piece is known, and the few indices that the cut's ties need are found by looking at one piece again.
//
// The loads. Four CTAs' shared memory leaves some 28 KB of L1 per SM, too little for 64 KB of register loads on their way
// (512 rows of 151,936 f32, loads alone: 65 us; 51 with L1 free), and the loop's loads share their scoreboards with its
// exponentials. So sample and row come by asynchronous copies to shared memory, which take no L1 (53); asking L2
// for lines further ahead made the pass slower. Everything uniform lies in shared memory and the pass has nothing on its stack: the stacks of a former
// version wrote 59 MB to HBM per 311 MB read. (The code around it still spills some values, once a row.)
//
// Error budget of the fast sums against exp(d) in f64, d = x/T - max rounded to f32 as upstream. With a cut the argument of
// 2^t is one FMA, x/T log2 e - C: ex2.approx 2.4e-7, three f32 additions per step before the f64 accumulators 1.8e-7, and per
// unit of |x/T - anchor| the roundings of t, of log2 e and of upstream's d, 1.4e-7 together: W1_EPS_FIXED + W1_EPS_PER_D * (largest |d|
// that carries mass). (C is the anchor times log2 e, rounded: the anchor that this stands for is what the sums are taken
// back from.) The anchor must lie within 2 of the maximum. The quick sums without a cut take the same roundings, one more of x/T - C.
constexpr int P1_ALL = 0, P1_EXACT = 1, P1_LOW = 2, P1_MID = 3;
constexpr int W1_SAMPLE = (W_NT >= 512) ? 16384 : 8192;        // logits of the sample
constexpr int W1_MIN_CUT = 4 * W1_SAMPLE + 64;                 // rows shorter than this are not sampled
constexpr int W1_SBINS = 1024;           // its histogram's buckets
constexpr float W1_MAX_WINDOW = 3328.0f; // logits of a window that takes more than the usual sample and buffers (wide_place_window)
constexpr float W1_PER_VISIT = 1.5f;     // logits that a lane's buffer gets, on average, before it is emptied: the most
constexpr double W1_EPS_FIXED = 4.5e-7;
constexpr double W1_EPS_PER_D = 2.0e-7;
constexpr int W1X_ENTRIES = 256, W1X_COPIES = 16;   // table of the exact exponential: 2^(j/256), a copy per pair of banks
constexpr float W1X_FAR = 88.0f;         // the sums' base may lie this far below the maximum
constexpr double W1X_STRETCH = 1.0 + 2.376e-12;   // what it takes the exponential of is stretched by this
static_assert(W1_SBINS % W_NT == 0 && W1_BINS == W_NT && W1_SAMPLE * 4 + W1_SBINS * 4 <= W1_OFF_BINS && W1X_ENTRIES * W1X_COPIES * 8 <= W1_OFF_RING, "a thread's share of the buckets; the sample and its buckets lie where lists and ring will be, the table where lists and buffers are not");
static_assert(W_MAX_PPW <= 32 && W_NW <= 32 && W_MAX_PIECES <= W1_BINS && W1_OFF_MASS + W_NW * W1_WCAP * 8 <= W1_OFF_BINS, "memory of the selection");

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }
__device__ __forceinline__ float ex2_approx(float t) { float e; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(t)); return e; }
__device__ __forceinline__ float set_ge(float a, float b) { float r; asm("set.ge.f32.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b)); return r; }   // 1.0f or 0.0f

// x / T in IEEE f32 round-to-nearest by q0 = x y, r = fma(-q0, T, x), q = fma(r, y, q0) with y = RN(1/T) (Markstein's correction):
// the correctly rounded quotient whenever T's significand is not all ones and nothing over- or underflows
// (the caller takes this form for 2^-20 <= T <= 2^20 only and clamps x at -1e30: whatever lies below has
// mass 0 either way).
__device__ __forceinline__ f32x2_t div2_fast(f32x2_t X, float T, float y) {
  const f32x2_t Y = pk2(y, y);
  const f32x2_t Q0 = mul2(X, Y);
  const f32x2_t R = fma2(Q0, pk2(-T, -T), X);
  return fma2(R, Y, Q0);
}
// Rows without a cut: quick sums first for rows of at least so many steps per warp whose first look spans no more than this, in units of x / T. Short
// rows gain little (592 x 12,000 f32: 27 us exact, 32 in two passes). A wide span goes with tokens far above the rest, which a first look
// does not see: the quick sums would be for nothing in most such rows.
constexpr int W1_QUICK_STEPS = 8;
constexpr float W1_QUICK_RANGE = 6.0f;
constexpr float P1_L2E = 1.4426950408889634f;

struct P1Consts {
  float C, Tm, yT;         // the anchor times log2 e (without a cut: what the sums are relative to, in units of x / T); temperature and its rounded reciprocal
  float xlow;              // P1_EXACT: logits below have no mass
  uint32_t tab;            // P1_EXACT: shared-memory address of this lane's copy of the table
  float xA;                // above the window: x >= xA
  float xmid, xhalf;       // |x - xmid| <= xhalf is a superset of the window
  uint32_t buf, buf_end;   // shared-memory addresses of this lane's buffer: its first slot, and the one that leaves room for four logits
};
struct P1Acc {
  double tot, tot2;        // all mass of the running piece (P1_MID: all mass so far); P1_EXACT: in two parts
  double kep;              // P1_MID: mass above the window of the running piece
  double stot;             // all mass of the pieces done
  float vmax;              // NaN-propagating running maximum
  uint32_t at;             // the lane's next slot
};

// Eight logits of a lane of a row without a cut: exp(x/T - C) as f64. Table and short polynomial (Tang's scheme): with n the integer nearest to
// s 256/ln2, s = n ln2/256 + r, exp = 2^(n/256) (1 + r + r^2/2 + r^3/6). ln2/256 is H + L with H of nine bits, so n H is exact up to
// |s| = W1X_FAR and r is rounded once; 1 + ... is applied in f64. The error is at most 1.2e-10 (two roundings at |r| <= 2^-9.5), besides
// that L's 24 bits make it exp(s W1X_STRETCH): the way back from C to the maximum is stretched too, and what is left is 2.4e-12 per
// unit below the maximum. s = x/T - C is exact for what carries mass: C is 0 while the row's first look stays within 32 of 0, else
// the next multiple of 32 on the side of 0. The table's exponent fields are reduced by j << 12, so that adding n << 12 leaves n div 256 there.
// (Bound by the number of instructions: the conversion of r (1 + ...) to f64 done by shifts is slower, 92 against 87 us for 512 x 151,936 bf16.)
template <bool TONE>
__device__ __forceinline__ void p1_body_exact(const float* x, const P1Consts& k, P1Acc& a) {
  a.vmax = max3nan(a.vmax, x[0], x[1]); a.vmax = max3nan(a.vmax, x[2], x[3]);
  a.vmax = max3nan(a.vmax, x[4], x[5]); a.vmax = max3nan(a.vmax, x[6], x[7]);
  constexpr float INV = 369.32993f, MAGIC = 12582912.0f, H = 355.0f / 131072.0f, L = -0x1.bd0106p-21f;
#pragma unroll
  for (int c = 0; c < 4; c++) {
    f32x2_t S_ = pk2(fmaxf(x[2 * c], k.xlow), fmaxf(x[2 * c + 1], k.xlow));
    if (!TONE) S_ = div2_fast(S_, k.Tm, k.yT);
    S_ = add2(S_, pk2(-k.C, -k.C));
    const f32x2_t F = fma2(S_, pk2(INV, INV), pk2(MAGIC, MAGIC));
    const f32x2_t N = add2(F, pk2(-MAGIC, -MAGIC));
    f32x2_t R = fma2(N, pk2(-H, -H), S_);
    R = fma2(N, pk2(-L, -L), R);
    const f32x2_t W = fma2(fma2(R, pk2(1.0f / 6.0f, 1.0f / 6.0f), pk2(0.5f, 0.5f)), mul2(R, R), R);
    float f[2], w[2];
    upk2(F, f[0], f[1]);
    upk2(W, w[0], w[1]);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t n = __float_as_uint(f[h]);
      const double t = lds_f64(k.tab + (n & (W1X_ENTRIES - 1)) * (W1X_COPIES * 8));
      const double E = __hiloint2double(__double2hiint(t) + static_cast<int>(n << 12), __double2loint(t));
      double& sum = h ? a.tot2 : a.tot;
      sum += fma(E, static_cast<double>(w[h]), E);
    }
  }
}
// Eight logits of a lane by ex2.approx; masked logits are -Inf and add 0. Three f32 additions per sum, then f64. With a cut, logits near
// the window go to the lane's buffer.
template <int VEC, bool TONE, int MODE>
__device__ __forceinline__ void p1_body(const float* x, const P1Consts& k, P1Acc& a) {
  constexpr bool CUT = MODE == P1_LOW || MODE == P1_MID;
  if (MODE == P1_EXACT) { p1_body_exact<TONE>(x, k, a); return; }
  a.vmax = max3nan(a.vmax, x[0], x[1]); a.vmax = max3nan(a.vmax, x[2], x[3]);
  a.vmax = max3nan(a.vmax, x[4], x[5]); a.vmax = max3nan(a.vmax, x[6], x[7]);
  f32x2_t E[4], KK[2];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const f32x2_t X = pk2(x[2 * c], x[2 * c + 1]);
    f32x2_t S_ = X;
    if (!TONE) S_ = div2_fast(pk2(fmaxf(x[2 * c], -1e30f), fmaxf(x[2 * c + 1], -1e30f)), k.Tm, k.yT);
    float t0, t1;
    if (CUT) upk2(fma2(S_, pk2(P1_L2E, P1_L2E), pk2(-k.C, -k.C)), t0, t1);
    else upk2(mul2(add2(S_, pk2(-k.C, -k.C)), pk2(P1_L2E, P1_L2E)), t0, t1);
    E[c] = pk2(ex2_approx(t0), ex2_approx(t1));
    if (MODE == P1_MID) {
      const f32x2_t M = pk2(set_ge(x[2 * c], k.xA), set_ge(x[2 * c + 1], k.xA));
      if ((c & 1) == 0) KK[c >> 1] = mul2(E[c], M); else KK[c >> 1] = fma2(E[c], M, KK[c >> 1]);
    }
    if (!CUT) continue;
    float z0, z1;
    upk2(add2(X, pk2(-k.xmid, -k.xmid)), z0, z1);
#pragma unroll
    for (int h = 0; h < 2; h++)
      asm volatile("{\n\t.reg .pred p;\n\tsetp.le.f32 p, %2, %3;\n\t@p st.shared.f32 [%0], %1;\n\t@p add.u32 %0, %0, %4;\n\t}"
                   : "+r"(a.at) : "f"(x[2 * c + h]), "f"(fabsf(h ? z1 : z0)), "f"(k.xhalf), "n"(W_NT * 4));
    if (c & 1) a.at = min(a.at, k.buf_end);                     // a full buffer stays full: the row takes two passes
  }
  { float p, q; upk2(add2(add2(E[0], E[1]), add2(E[2], E[3])), p, q); a.tot += static_cast<double>(p + q); }
  if (MODE == P1_MID) {
    float p, q;
    upk2(add2(KK[0], KK[1]), p, q);
    a.kep += static_cast<double>(p + q);
  }
}
// Logits of a lane-step (first vector gv) that lie outside the row become -Inf.
template <int VEC>
__device__ __forceinline__ void p1_mask(float* x, int gv, int nvec, int shift, int V) {
#pragma unroll
  for (int c = 0; c < 8; c++) {
    const int g = gv + 32 * (c / VEC), i = g * VEC - shift + (c % VEC);
    if (!(g < nvec && i >= 0 && i < V)) x[c] = -INFINITY;
  }
}
// The pass. Leaves in shared memory: part[warp * ppw + piece], the mass of each piece (P1_MID: of its logits above the window), relative to the anchor or base; the warps' lists, and in from[warp][piece] where a piece begins in its warp's;
// per warp kw (sum of its pieces), sc.d0 (all mass), sc.i0 (order key of the maximum), sc.i1 (1: a NaN, 2: a list that did
// not hold all).
template <typename T, bool TONE, int MODE, bool OFTEN = false>
__device__ __noinline__ void wide_onepass_stream(unsigned char* dyn, WideShared& sh) {
  constexpr int VEC = Elem<T>::VEC, EPI = 8 / VEC, SV = 32 * EPI;
  constexpr uint32_t STAGE = EPI * W_NT * 16;                  // ring: EPI vectors per thread and stage
  constexpr int NQ = W1_RING_BYTES / STAGE;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nvec = sh.nvec, shift = sh.shift, ppw = sh.ppw;
  const int first = warp * sh.span, end = min(nvec, first + sh.span);
  const int nst = (end > first) ? (end - first + SV - 1) / SV : 0;
  // steps [clean_lo, clean_hi) hold no logit outside the row: all their vectors exist, none is the row's first or last
  const int clean_lo = (first == 0) ? 1 : 0, clean_hi = min(nst, (nvec - 1 - first) / SV);
  P1Consts k;
  constexpr bool CUT = MODE == P1_LOW || MODE == P1_MID;
  k.C = CUT ? sh.as * P1_L2E : (MODE == P1_EXACT ? sh.base : sh.as); k.Tm = sh.Tm; k.yT = TONE ? 1.0f : __frcp_rn(sh.Tm);
  k.xlow = (sh.base - 700.0f) * sh.Tm;
  k.tab = smem_addr(dyn + W1_OFF_TAB) + 8u * (lane & (W1X_COPIES - 1));
  k.xA = sh.xA;
  k.xmid = 0.5f * sh.xA + 0.5f * sh.xB;
  k.xhalf = (0.5f * sh.xA - 0.5f * sh.xB) * 1.000001f + 1e-30f + 2.4e-7f * fabsf(k.xmid);
  k.buf = smem_addr(dyn + W1_OFF_BUF) + static_cast<uint32_t>(tid) * 4u;
  k.buf_end = k.buf + (W1_SLOTS - 4) * W_NT * 4u;
  double* part_w = reinterpret_cast<double*>(dyn + W_OFF_PART) + warp * ppw;
  float* list = reinterpret_cast<float*>(dyn + W1_OFF_LIST) + warp * W1_WCAP;
  int* from = reinterpret_cast<int*>(dyn + W1_OFF_FROM) + warp * (W_MAX_PPW + 1);
  int listed = 0;                                              // by the warp, so far
  bool full = false;
  if (lane == 0) from[0] = 0;
  P1Acc a;
  a.tot = 0.0; a.tot2 = 0.0; a.kep = 0.0; a.stot = 0.0; a.vmax = -INFINITY; a.at = k.buf;
  // The ring: a thread copies the vectors it will take itself, and waits for its own copies only. A vector past the row's
  // end is replaced by the row's last one (masked below).
  const uint4* src = sh.vbase + first + lane;
  const int omax = nvec - 1 - first - lane;                    // of the offsets from src (negative: none of the warp's steps runs then)
  const uint32_t ring = smem_addr(dyn + W1_OFF_RING) + static_cast<uint32_t>(tid) * 16u;
  const uint4* ring_at = reinterpret_cast<const uint4*>(dyn + W1_OFF_RING) + tid;
  volatile int* far = &sh.far;
  constexpr int VISIT = OFTEN ? NQ : W_G;                      // steps from one emptying of the buffers to the next
  auto empty_buffers = [&]() {
    full |= a.at >= k.buf_end;
    const int n = static_cast<int>((a.at - k.buf) / (W_NT * 4u));
    for (int r = 0;; r++) {
      const unsigned have = __ballot_sync(FULL, r < n);
      if (have == 0u) break;
      const int slot = listed + __popc(have & ((1u << lane) - 1u));
      if (r < n && slot < W1_WCAP) {
        float v;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(k.buf + static_cast<uint32_t>(r) * (W_NT * 4u)));
        list[slot] = v;
      }
      listed += __popc(have);
    }
    a.at = k.buf;
  };
  auto piece_end = [&](int st) {
    if (CUT && lane == 0) from[st / W_G + 1] = min(listed, W1_WCAP);
    double t = a.kep;
    if (MODE == P1_MID) a.kep = 0.0;
    else { t = (MODE == P1_EXACT) ? a.tot + a.tot2 : a.tot; a.stot += t; a.tot = a.tot2 = 0.0; }
    double kw = warp_sum_d(t);
    if (MODE == P1_EXACT && kw < 1e-270) kw = 0.0;               // -Inf throughout (each counts as exp(-700))
    if (lane == 0) part_w[st / W_G] = kw;
  };
  auto step = [&](int st, int slot, auto&& refill, bool clean) {
    cp_wait<NQ - 1>();
    float x[8];
    Elem<T>::unpack(ring_at[slot * EPI * W_NT], x);
    if (EPI == 2) Elem<T>::unpack(ring_at[slot * EPI * W_NT + W_NT], x + 4 * (EPI - 1));
    refill();                                                  // into the slot just read
    cp_commit();
    if (!clean) p1_mask<VEC>(x, first + st * SV + lane, nvec, shift, sh.V);
    p1_body<VEC, TONE, MODE>(x, k, a);
  };
  auto put = [&](int slot, const uint4* p0, const uint4* p1) {
    cp_async16(ring + slot * STAGE, p0);
    if (EPI == 2) cp_async16(ring + slot * STAGE + W_NT * 16u, p1);
  };
  auto put_any = [&](int slot, int q) { if (q < nst) put(slot, src + min(q * SV, omax), src + min(q * SV + 32, omax)); };
#pragma unroll
  for (int q = 0; q < NQ; q++) { put_any(q, q); cp_commit(); }
  // Pieces, or the parts of a piece between two emptyings, that hold no step at the row's edges and whose refills are clean too run without a
  // mask, a clamp or a test; either is a multiple of the ring's NQ steps.
  static_assert(W_G % NQ == 0, "a piece begins at the ring's first slot");
  int st = 0;
#pragma unroll 1
  while (st < nst) {
    if (st >= clean_lo && st + VISIT + NQ <= clean_hi) {
      const uint4* p = src + (st + NQ) * SV;
#pragma unroll 1
      for (int j = 0; j < VISIT; j += NQ, p += NQ * SV) {
#pragma unroll
        for (int q = 0; q < NQ; q++) step(st, q, [&]() { put(q, p + q * SV, p + q * SV + 32); }, true);
      }
      st += VISIT;
    } else {
#pragma unroll 1
      for (int j = 0; j < VISIT && st < nst; j++, st++)
        step(st, j % NQ, [&]() { put_any(j % NQ, st + NQ); }, st >= clean_lo && st < clean_hi);
    }
    if (CUT) empty_buffers();
    if (OFTEN && st % W_G != 0 && st < nst) continue;
    piece_end(st - 1);
    if (MODE == P1_ALL) {                                      // a logit far above the anchor: the row's sums will be exact ones
      if (__any_sync(FULL, a.vmax > k.xA || *far != 0)) {
        if (lane == 0) *far = 1;
        break;
      }
    }
  }
  cp_wait<0>();
  if (lane == 0) {
    for (int q = (nst + W_G - 1) / W_G; q < ppw; q++) {        // pieces past the row's end
      from[q + 1] = min(listed, W1_WCAP);
      part_w[q] = 0.0;
    }
  }
  __syncwarp();
  const double kw = warp_sum_d((lane < ppw) ? part_w[lane] : 0.0);
  const double S = warp_sum_d(MODE == P1_MID ? a.tot : a.stot);
  const uint32_t wmax = __reduce_max_sync(FULL, okey(a.vmax));
  const int odd = (__any_sync(FULL, a.vmax != a.vmax) ? 1 : 0) | ((CUT && (listed > W1_WCAP || __any_sync(FULL, full))) ? 2 : 0);
  if (lane == 0) { sh.kw[warp] = kw; sh.sc.d0[warp] = S; sh.sc.i0[warp] = static_cast<int>(wmax); sh.sc.i1[warp] = odd; }
  __syncthreads();
}

template <typename T, bool TONE, int MODE>
__device__ __forceinline__ void pass_with_cut(unsigned char* dyn, WideShared& sh) {
  if (sh.placed & HOW_OFTEN) wide_onepass_stream<T, TONE, MODE, true>(dyn, sh);
  else wide_onepass_stream<T, TONE, MODE>(dyn, sh);
}

// Places the window of a row with a cut: sh.as, xA, xB, placed and eps. 0, or why the row takes two passes, or WHY_AGAIN: twice the sample may do,
// and the next call (`again`) adds its other half to the buckets.
template <typename T>
__device__ __noinline__ int wide_place_window(unsigned char* dyn, WideShared& sh, const double plim, const bool again) {
  constexpr int VEC = Elem<T>::VEC;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float Tm = sh.Tm;
  const int V = sh.V;
  // ---- the sample: 64-byte pieces spread evenly over the row, none of them at its edges; a thread looks at what it copied itself
  constexpr int J = W1_SAMPLE / (W_NT * VEC), PIECES = W_NT * J / 4;
  const int have = (sh.nvec - 2) / 4;                                     // whole pieces between the row's first and last vector
  {
    const uint4* src = sh.vbase + 1 + (tid & 3);
    const uint32_t dst = smem_addr(dyn) + static_cast<uint32_t>(tid) * 16u;
#pragma unroll
    for (int j = 0; j < J; j++) {                                         // (the other half's pieces lie between the first's)
      const uint32_t at = 2u * static_cast<uint32_t>((j * W_NT + tid) >> 2) + (again ? 1u : 0u);
      const int piece = static_cast<int>(static_cast<uint32_t>((static_cast<uint64_t>(at) * static_cast<uint32_t>(have)) / (2u * PIECES)));
      cp_async16(dst + j * W_NT * 16, src + piece * 4);
    }
    cp_commit();
  }
  uint32_t* bins = reinterpret_cast<uint32_t*>(dyn + W1_SAMPLE * 4);
  if (!again) for (int j = tid; j < W1_SBINS; j += W_NT) bins[j] = 0u;
  auto each = [&](auto&& fn) {
#pragma unroll 2
    for (int j = 0; j < J; j++) {
      float x[VEC];
      Elem<T>::unpack(reinterpret_cast<const uint4*>(dyn)[j * W_NT + tid], x);
#pragma unroll
      for (int c = 0; c < VEC; c++) fn(x[c]);
    }
  };
  cp_wait<0>();
  float smax = again ? sh.xA : -INFINITY, smin = again ? sh.xB : INFINITY;
  if (!again) {
    each([&](float x) { smax = maxnan(smax, x); smin = fminf(smin, x); });
    uint32_t hi = okey(smax), lo = ~okey(smin), nan = (smax != smax) ? 1u : 0u;
    bu::max_u3<W_NW>(hi, lo, nan, sh.sc, tid);                            // (its barriers also publish the cleared bins)
    if (nan) return WHY_NOT_FINITE;
    smax = okey_to_float(hi);
    smin = okey_to_float(~lo);
  }
  const float as = scale_t(smax, Tm);
  if (!(fabsf(smax) < 1e30f) || !(fabsf(as) < 1e30f)) return WHY_NOT_FINITE;
  // ---- a count histogram of its upper 24 units of x / T (what lies lower has no mass to speak of, and shares the last bucket)
  const float range = fmaxf(fminf(smax - smin, 24.0f * Tm), 1e-6f * fmaxf(fabsf(smax), Tm));
  const float scale = static_cast<float>(W1_SBINS - 1) / range;
  // (a logit of the second half may lie above smax: the pass finds out how far)
  const int sampled = again ? 2 * W1_SAMPLE : W1_SAMPLE;
  each([&](float x) { atomicAdd(&bins[static_cast<int>(fmaxf(fminf((smax - x) * scale, static_cast<float>(W1_SBINS - 1)), 0.0f))], 1u); });
  if (tid == 0) { sh.bc[0] = 0; sh.bc[1] = 0; }
  __syncthreads();
  // ---- the window: where the sample's mass passes plim, give or take 4.5 standard errors of a mass fraction
  // estimated from weighted logits (Var = ((1-p)^2 sum of squared weights above the cut + p^2 of those below) / (sum of
  // weights)^2). Placing it is a matter of speed, not of correctness (the pass checks it on the whole row): f32 does.
  constexpr int PER = W1_SBINS / W_NT;
  const float wl2 = range / (Tm * static_cast<float>(W1_SBINS - 1)) * 1.4426950408889634f;   // bucket width in units of log2
  int cnt[PER] = {}, n = 0;
  float mass = 0.0f, sq = 0.0f;
  const float ratio = ex2_approx(-wl2), e0 = ex2_approx(-(static_cast<float>(tid * PER) + 0.5f) * wl2);
  auto weight = [&](int j, float e) { return (tid * PER + j == W1_SBINS - 1) ? 0.0f : static_cast<float>(cnt[j]) * e; };
  {
    float e = e0;
#pragma unroll
    for (int j = 0; j < PER; j++) {
      cnt[j] = static_cast<int>(bins[tid * PER + j]);
      const float c = weight(j, e);
      n += cnt[j]; mass += c; sq = fmaf(c, e, sq);
      e *= ratio;
    }
  }
  float im = mass, iq = sq;
  int in = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float a = __shfl_up_sync(FULL, im, o), b = __shfl_up_sync(FULL, iq, o);
    const int c = __shfl_up_sync(FULL, in, o);
    if (lane >= o) { im += a; iq += b; in += c; }
  }
  float* wm = reinterpret_cast<float*>(sh.sc.d0);
  float* wq = reinterpret_cast<float*>(sh.sc.d1);
  if (lane == 31) { wm[warp] = im; wq[warp] = iq; sh.sc.i0[warp] = in; }
  if (tid == 0) wq[W_NW] = 0.0f;
  __syncthreads();
  float tot_m = 0.0f, tot_q = 0.0f;
  im -= mass; iq -= sq; in -= n;                                          // exclusive
#pragma unroll
  for (int w = 0; w < W_NW; w++) {
    const float a = wm[w], b = wq[w];
    if (w < warp) { im += a; iq += b; in += sh.sc.i0[w]; }
    tot_m += a; tot_q += b;
  }
  if (!(tot_m * 2.4e-3f >= 1.0f)) return WHY_HEAVY;                             // heavy tokens (one above 1/400 of the mass): not for a sample to place
  const float pl = static_cast<float>(plim), lim = pl * tot_m;
  // Where a limit is passed: in the last thread whose prefix lies below it, found as a maximum. (A thread's own end and the next one's prefix are rounded
  // differently, and a limit between the two is passed by neither: one row in 17,000 got a window from the row's first bucket that way.)
  auto last_below = [&](int mine, int* slot) {
    const int top = __reduce_max_sync(FULL, mine);
    if (lane == 0) atomicMax(slot, top);
  };
  last_below(im < lim ? __float_as_int(iq + sq) : 0, reinterpret_cast<int*>(wq + W_NW));
  __syncthreads();
  const float q_above = wq[W_NW], q1 = 1.0f - pl;
  const float fpc = 1.0f - static_cast<float>(sampled) / static_cast<float>(V);
  const float delta = 4.5f * sqrtf(fmaxf(q1 * q1 * q_above + pl * pl * (tot_q - q_above), 0.0f) * fpc) + 2.0f;   // in units of mass: two top tokens more
  const float m_lo = lim - delta, m_hi = lim + delta;
  {
    float e = e0, acc = im;
    int c = in, lo = 0, hi = 0;                                           // bucket << 16 | logits of the sample above it, or through it
#pragma unroll
    for (int j = 0; j < PER; j++) {
      const int at = (tid * PER + j) << 16;
      if (acc < m_lo) lo = at | c;
      c += cnt[j];
      if (acc < m_hi) hi = at | c;
      acc += weight(j, e);
      e *= ratio;
    }
    last_below(lo, &sh.bc[0]);
    last_below(hi, &sh.bc[1]);
  }
  __syncthreads();
  static_assert(2 * W1_SAMPLE < 65536, "counts of the sample in 16 bits");
  const int from_bin = sh.bc[0] >> 16, above = sh.bc[0] & 0xffff, to_bin = sh.bc[1] >> 16, through = sh.bc[1] & 0xffff;
  const int b1 = max(from_bin - 1, 0), b2 = min(to_bin + 1, W1_SBINS - 1);   // a bucket of slack for the f32 sums
  // How many logits of the row will be listed: as many as the sample's share of the window says, and of the buckets of slack as many as
  // the window's have on average. The lists hold 4.5 standard deviations more, of the sample's count and of a warp's part; a lane's buffer, which
  // counts as full at 12, is expected to get W1_PER_VISIT at most before it is emptied (full then: one lane in 4 x 10^7, one row of 151,936
  // logits in 15,000). A list that does not hold all costs a pass: one such row made 512 rows of 151,936 (p = 0.98) take 188 us for 115.
  // A window that reaches down to where no mass is saves instructions.
  const float to_row = static_cast<float>(V) / static_cast<float>(sampled), to_warp = to_row * static_cast<float>(sh.span) / static_cast<float>(sh.nvec);
  auto fits = [&](float logits, int visits) {
    const float per_warp = logits * to_warp;
    return per_warp + 4.5f * sqrtf(per_warp * (1.0f + to_warp)) <= static_cast<float>(W1_WCAP) && logits * to_row <= W1_PER_VISIT * static_cast<float>(visits);
  };
  const float seen = static_cast<float>(max(through - above, 0)), per_bucket = seen / static_cast<float>(max(to_bin - from_bin + 1, 1));
  const float n_low = static_cast<float>(sampled - above) + per_bucket, n_mid = seen + 2.0f * per_bucket;
  // how often a lane empties its buffer: once a piece, or once for each turn of the ring
  const int seldom = W_NT * max(sh.nvec / (W_NT * (8 / VEC) * W_G), 1), turns = V / (W1_RING_BYTES / (W_NT * static_cast<int>(sizeof(T))));
  bool low = fits(n_low, seldom), often = false;
  if (!low && !fits(n_mid, seldom)) {
    // Wider windows are listed where an eighth of the row as sample, with the error of a plain share, leaves W1_MAX_WINDOW logits or fewer between
    // the bounds. Beyond that the rows keep the exactness of the two-pass sums, which they always had (3e-10 against 4e-8).
    // (us, flat f32 rows in two passes | one: 512 x 50,257, p = 0.95: 115 | 67; 512 x 100,003, 0.97: 164 | 88; 512 x 151,936, 0.98: 210 | 112;
    // 128 x 100,003, 0.97: 76 | 44.)
    const float by_eighth = tot_m * (5.0f * sqrtf(pl * fabsf(q1) * 8.0f / static_cast<float>(V)) + 32.0f / static_cast<float>(V));
    if (seen * to_row * by_eighth > W1_MAX_WINDOW * delta) return WHY_WINDOW;
    often = true;
    low = fits(n_low, turns);
    if (!low && !fits(n_mid, turns)) {
      // Twice the sample makes the window narrower by sqrt(2), but for its slack: where that will do, and the sample is less than an eighth of
      // the row, its other half too (10 us of 512 rows of 151,936 f32, for which two passes take 100 longer)
      if (again || to_row <= 8.0f || !fits(0.78f * seen + 2.0f * per_bucket, turns)) return WHY_WINDOW;
      if (tid == 0) { sh.xA = smax; sh.xB = smin; }
      return WHY_AGAIN;
    }
  }
  const float xA = smax - static_cast<float>(b1) / scale;
  const float xB = (low || b2 == W1_SBINS - 1) ? smax - 40.0f * Tm : smax - static_cast<float>(b2 + 1) / scale;
  if (!(xA > xB)) return WHY_EMPTY_WINDOW;
  if (tid == 0) {
    sh.as = as; sh.xA = xA; sh.xB = xB; sh.placed = (low ? HOW_LOW : 0) | (often ? HOW_OFTEN : 0) | (again ? HOW_TWICE : 0);
    sh.eps = W1_EPS_FIXED + W1_EPS_PER_D * fmin(9.7, static_cast<double>(range / Tm) + 2.0);
  }
  return 0;
}

// One row. 0, or why it takes two passes (nothing of it has been written then).
template <typename T>
__device__ __noinline__ int wide_onepass_row(const BatchArgs& BA, const int64_t row_id, unsigned char* dyn, WideShared& sh) {
  const KernelArgs& A = BA.k;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int VEC = Elem<T>::VEC, SV = 32 * (8 / VEC), PV = W_G * SV;
  bu::Scratch& sc = sh.sc;
  const double* s_tab = sh.tab;
  const RowCfg cfg = A.cfgs[row_id];
  const float Tm = cfg.temperature;
  const int mode = cfg.topp_mode;
  const double plim = (mode == 0) ? static_cast<double>(cfg.top_p) * 1.5 : static_cast<double>(cfg.top_p);
  // mode A prunes only while the mass exceeds 1.5p; the mass starts at 1 up to ~1e-11 of rounding
  // and 1.5*float(p) is never that close to 1
  const bool cut_on = cfg.top_p > 0.0f && cfg.top_p < 1.0f && !(mode == 0 && plim >= 1.0);
  const bool t_is_one = (Tm == 1.0f);
  // Rows with a cut shorter than four samples take two passes, and are told before anything is done for them. In the 1024-thread instance a sample that
  // then finds nothing to place costs 128 rows of 50,257 f32 8 us of 50, and rows peaked like a language model's are of that kind.
  if (cut_on && A.V < W1_MIN_CUT) return WHY_SHORT;
  bool quick = false;                      // without a cut: the sums by ex2.approx, if the maximum turns out where it is expected
  if (!t_is_one && !(Tm >= 9.5367431640625e-7f && Tm <= 1048576.0f && (__float_as_uint(Tm) & 0x7fffffu) != 0x7fffffu)) return WHY_TEMPERATURE;
  {
    RowView<T> rv;
    rv.init(static_cast<const T*>(A.logits) + row_id * A.row_stride, A.V);
    const int span = (((rv.nvec + W_NW - 1) / W_NW + SV - 1) / SV) * SV;   // a warp's part of the row, in whole steps
    if (span / SV > W_MAX_STEPS) return WHY_LONG;
    if (tid == 0) {
      sh.vbase = rv.vbase; sh.V = rv.V; sh.shift = rv.shift; sh.nvec = rv.nvec;
      sh.span = span; sh.ppw = (span / SV + W_G - 1) / W_G;
      sh.Tm = Tm; sh.xA = 0.0f; sh.xB = 0.0f; sh.base = 0.0f;
    }
    if (!cut_on) {
      // ---- a first look: the warps' first steps. The row's maximum is expected an eighth of their range above theirs.
      float smax = -INFINITY, smin = INFINITY;
#pragma unroll
      for (int h = 0; h < 8 / VEC; h++) {
        const int g = warp * span + 32 * h + lane;
        if (g < rv.nvec) rv.visit(g, [&](float xv, int) { smax = maxnan(smax, xv); smin = fminf(smin, xv); });
      }
      uint32_t top = okey(smax), nan = (smax != smax) ? 1u : 0u, inv = ~okey(smin);
      bu::max_u3<W_NW>(top, nan, inv, sc, tid);
      if (nan) return WHY_NOT_FINITE;
      smax = okey_to_float(top);
      smin = okey_to_float(~inv);
      const float as = scale_t(smax + 0.125f * (smax - smin), Tm);
      quick = rv.nvec >= W1_QUICK_STEPS * W_NW * SV && (smax - smin) / Tm <= W1_QUICK_RANGE && fabsf(as) < 1e30f;
      if (tid == 0) { sh.as = quick ? as : scale_t(smax, Tm); sh.xA = (as + 2.0f) * Tm; sh.far = 0; }
    }
  }
  __syncthreads();
  if (cut_on) {
    int why = wide_place_window<T>(dyn, sh, plim, false);
    if (why == WHY_AGAIN) {
      __syncthreads();                                         // (what the first call left in shared memory has been read)
      why = wide_place_window<T>(dyn, sh, plim, true);
    }
    if (why) return why;
  }
  __syncthreads();
  const bool low = cut_on && (sh.placed & HOW_LOW) != 0;
  const bool mine = lane < W_NW;
  bool exact = false;
  if (low) {
    if (t_is_one) pass_with_cut<T, true, P1_LOW>(dyn, sh); else pass_with_cut<T, false, P1_LOW>(dyn, sh);
  } else if (cut_on) {
    if (t_is_one) pass_with_cut<T, true, P1_MID>(dyn, sh); else pass_with_cut<T, false, P1_MID>(dyn, sh);
  } else {
    float b = sh.as;
    if (quick) {
      if (t_is_one) wide_onepass_stream<T, true, P1_ALL>(dyn, sh); else wide_onepass_stream<T, false, P1_ALL>(dyn, sh);
      if (__reduce_or_sync(FULL, mine ? sc.i1[lane] : 0)) return WHY_NAN;
      b = scale_t(okey_to_float(__reduce_max_sync(FULL, mine ? static_cast<uint32_t>(sc.i0[lane]) : 0u)), Tm);   // the largest so far
    }
    exact = !quick || sh.far || !(fabsf(b - sh.as) <= 2.0f);
    if (exact) {
      if (!(fabsf(b) <= 1e6f)) return WHY_ANCHOR;              // (further out base - 700 is no f32)
      if (tid == 0) sh.base = 32.0f * truncf(b * 0.03125f);
      double* tab = reinterpret_cast<double*>(dyn + W1_OFF_TAB);
      for (int j = tid; j < W1X_ENTRIES * W1X_COPIES; j += W_NT) {
        const int e = j / W1X_COPIES;
        const double t = s_tab[e];
        tab[j] = __hiloint2double(__double2hiint(t) - (e << 12), __double2loint(t));
      }
      __syncthreads();
      if (t_is_one) wide_onepass_stream<T, true, P1_EXACT>(dyn, sh); else wide_onepass_stream<T, false, P1_EXACT>(dyn, sh);
    }
  }
  // ---- the row's sums and maximum
  const float m = scale_t(okey_to_float(__reduce_max_sync(FULL, mine ? static_cast<uint32_t>(sc.i0[lane]) : 0u)), Tm);
  const int any = __reduce_or_sync(FULL, mine ? sc.i1[lane] : 0);
  double S = warp_sum_d(mine ? sc.d0[lane] : 0.0);
  double Ktot = warp_sum_d(mine ? sh.kw[lane] : 0.0);
  if ((any & 1) || !(fabsf(m) < INFINITY)) return WHY_NAN;                    // the two-pass form reports such rows
  if (any & 2) return WHY_LIST;
  // with a cut the anchor is the sample's maximum: it must be close to the row's for the heavy logits to keep the error budget
  if (exact ? !(m - sh.base <= W1X_FAR) : !(fabsf(m - sh.as) <= 2.0f)) return WHY_ANCHOR;
  if (!(S > 0.0) || !(S < 1e300)) return WHY_SUM;
  // everything so far is relative to exp(anchor); from here on to exp(max)
  const double anchor = cut_on ? static_cast<double>(sh.as * P1_L2E) / static_cast<double>(P1_L2E) : static_cast<double>(exact ? sh.base : sh.as);
  const double cf = exp((anchor - static_cast<double>(m)) * (exact ? W1X_STRETCH : 1.0));
  S *= cf;
  Ktot *= cf;
  if (!(S > 0.0)) return WHY_SUM;
  const int ppw = sh.ppw, span = sh.span;
  const float xA = sh.xA, xB = sh.xB;
  const int* from = reinterpret_cast<const int*>(dyn + W1_OFF_FROM);
  const double* part = reinterpret_cast<const double*>(dyn + W_OFF_PART);
  uint32_t* bins = reinterpret_cast<uint32_t*>(dyn + W1_OFF_BINS);
  uint32_t flags = FLAG_GENERAL_PATH;
  RowView<T> rv;
  rv.vbase = sh.vbase; rv.V = sh.V; rv.shift = sh.shift; rv.nvec = sh.nvec;

  // ---- the cut. The order of the kept set is by d, equal ones by index: a class of equal d is kept, dropped, or divided
  // by an index.
  unsigned long long cut_key = 0ull;       // window entries are kept when key < cut_key, or == with cut_incl
  int cut_incl = 0;
  float dstar = INFINITY;
  double estar = 0.0, zw = 0.0;            // mass of one member of the cut's class; lane w: what the window adds to warp w's part
  bool one_class = false;                  // the candidates are a long run of equal d
  bool by_piece = false, ties_in = false;  // kept members of the class: counted per piece in bins[], or all of them
  if (cut_on) {
    const double lim = plim * S;
    auto crossed = [&](double g) -> bool { return mode == 0 ? (g > lim) : (g >= lim); };
    float* list = reinterpret_cast<float*>(dyn + W1_OFF_LIST) + warp * W1_WCAP;   // every warp works on its own list
    double* mass = reinterpret_cast<double*>(dyn + W1_OFF_MASS) + warp * W1_WCAP;
    from += warp * (W_MAX_PPW + 1);
    const int cnt = from[ppw];
    const float dA = scale_t(xA, Tm) - m, dB = scale_t(xB, Tm) - m;
    float dhi = dA, dlo = dB, scale = static_cast<float>(W1_BINS) / (dA - dB);
    auto bucket = [&](float d) { return static_cast<int>(fminf((dhi - d) * scale, static_cast<float>(W1_BINS - 1))); };
    bins[tid] = 0u;
    if (tid == 0) { sh.bc[0] = W1_BINS; sh.bc[1] = W1_BINS - 1; sh.cnt = 0; }
    __syncthreads();
    // logits -> d, in place (1: not in the window, the lists hold a little more), their masses, and their counts by bucket of d
    double inside = 0.0;
    for (int j = lane; j < cnt; j += 32) {
      const float x = list[j];
      const float d = (x >= xB && x < xA) ? scale_t(x, Tm) - m : 1.0f;
      list[j] = d;
      if (d <= 0.0f) {
        const double e = exp_safe(d, s_tab);
        mass[j] = e;
        inside += e;
        atomicAdd(&bins[bucket(d)], 1u);
      }
    }
    if (low) {                                               // what is not listed is kept
      inside = bu::sum_d<W_NW>(inside, sc, tid);             // (its barriers also publish the counts)
      Ktot = S - inside;
    } else {
      __syncthreads();
    }
    // the cut must lie below the window's upper end by more than the error of the sums
    if (!(Ktot < lim - (1e-12 + 2.0 * plim * fabs(1.0 - plim) * sh.eps + 1e-9) * S)) return WHY_CUT_ABOVE;
    double gbase = Ktot;                                     // mass of everything above dhi
    double zsum = 0.0;                                       // this lane's window mass above the crossing's buckets
    int nc = 0;
    for (int round = 0;; round++) {                          // uniform
      // The bucket of the crossing, from bounds of the mass through each bucket (a bucket's members lie between its edges): the
      // first that can cross, and the first that must. The slack covers the f32 sums and edges.
      {
        const float need = static_cast<float>(lim - gbase), width = 1.0f / scale;
        const float c = static_cast<float>(bins[tid]);
        const float top = dhi - static_cast<float>(tid) * width;
        float hi = c * ex2_approx(top * 1.44269504f) * (1.0f + 2e-5f), lo = c * ex2_approx((top - width) * 1.44269504f) * (1.0f - 2e-5f);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const float a = __shfl_up_sync(FULL, hi, o), b = __shfl_up_sync(FULL, lo, o);
          if (lane >= o) { hi += a; lo += b; }
        }
        float* wh = reinterpret_cast<float*>(sc.u);          // (not sc.d0: a warp may still be reading sum_d's there)
        float* wl = reinterpret_cast<float*>(sc.d1);
        if (lane == 31) { wh[warp] = hi; wl[warp] = lo; }
        __syncthreads();
#pragma unroll
        for (int w = 0; w < W_NW; w++) if (w < warp) { hi += wh[w]; lo += wl[w]; }
        const unsigned may = __ballot_sync(FULL, hi >= need && c > 0.0f), must = __ballot_sync(FULL, lo >= need && c > 0.0f);
        if (lane == 0 && may) atomicMin(&sh.bc[0], warp * 32 + __ffs(may) - 1);
        if (lane == 0 && must) atomicMin(&sh.bc[1], warp * 32 + __ffs(must) - 1);
        __syncthreads();
      }
      const int b1 = sh.bc[0], b2 = max(sh.bc[1], b1);
      if (b1 == W1_BINS) return WHY_CUT_BELOW;                          // the window ends before the cut
      // what lies above the crossing's buckets is kept; what lies in them is looked at one by one
      double sure = 0.0;
      float cmax = -INFINITY, cmin = 1.0f;
      float* cd = reinterpret_cast<float*>(bins);            // the candidates: d, the warp they come from (the buckets have been read)
      int* cl = reinterpret_cast<int*>(bins) + 32;
      for (int j = lane; j < cnt; j += 32) {
        const float d = list[j];
        if (d <= dhi && d >= dlo) {
          const int b = bucket(d);
          if (b < b1) sure += mass[j];
          else if (b <= b2) {
            cmin = (cmin > 0.0f) ? d : fminf(cmin, d); cmax = fmaxf(cmax, d);
            const int slot = atomicAdd(&sh.cnt, 1);
            if (slot < 32) { cd[slot] = d; cl[slot] = warp; }
          }
        }
      }
      zsum += sure;
      gbase += bu::sum_d<W_NW>(sure, sc, tid);
      nc = sh.cnt;
      if (nc <= 32) break;
      uint32_t kmax = dkey_of(cmin), inv = ~dkey_of(cmax), none = 0u;      // (dkey falls as d rises)
      if (cmin > 0.0f) { kmax = 0u; inv = 0u; }                            // none here
      bu::max_u3<W_NW>(kmax, inv, none, sc, tid);
      const float was_hi = dhi, was_lo = dlo;
      dhi = -__uint_as_float(~inv); dlo = -__uint_as_float(kmax);
      if (dhi == dlo) { one_class = true; break; }           // a long run of equal d
      if (round == 7) return WHY_CUT_BELOW;
      if (dhi == was_hi && dlo == was_lo) {
        // The cut lies within the bounds' slack of where a long run of equal d ends: nothing came off either end. The upper run by
        // itself, exactly (bf16 rows met this once in four thousand, and took two passes after all).
        int run = 0;
        float next = -INFINITY;
        for (int j = lane; j < cnt; j += 32) {
          const float d = list[j];
          if (d == dhi) run++;
          else if (d < dhi && d >= dlo) next = fmaxf(next, d);
        }
        const double e = exp_safe(dhi, s_tab);
        nc = bu::sum_i<W_NW>(run, sc, tid);
        if (crossed(gbase + nc * e)) { one_class = true; break; }
        zsum += run * e;
        gbase += nc * e;
        uint32_t up = (next > -INFINITY) ? ~dkey_of(next) : 0u, none1 = 0u, none2 = 0u;
        bu::max_u3<W_NW>(up, none1, none2, sc, tid);
        dhi = -__uint_as_float(~up);
      }
      scale = fminf(static_cast<float>(W1_BINS) / (dhi - dlo), 1e30f);
      bins[tid] = 0u;
      if (tid == 0) { sh.bc[0] = W1_BINS; sh.bc[1] = W1_BINS - 1; sh.cnt = 0; }
      __syncthreads();
      for (int j = lane; j < cnt; j += 32) {
        const float d = list[j];
        if (d <= dhi && d >= dlo) atomicAdd(&bins[bucket(d)], 1u);
      }
      __syncthreads();
    }
    // ---- the class of the crossing: its d, the mass above it, its size. Every warp finds it by itself, a candidate per lane.
    double gb = gbase;
    int neq = nc;
    const float d_l = (!one_class && lane < nc) ? reinterpret_cast<const float*>(bins)[lane] : -INFINITY;
    const int from_l = (!one_class && lane < nc) ? reinterpret_cast<const int*>(bins)[32 + lane] : -1;
    const double e_l = (d_l <= 0.0f && lane < nc) ? exp_safe(d_l, s_tab) : 0.0;
    if (one_class) {
      dstar = dhi;
    } else {
      double g = gbase;
      int eq = 0;
      for (int i = 0; i < nc; i++) {
        const float o = __shfl_sync(FULL, d_l, i);
        const double oe = __shfl_sync(FULL, e_l, i);
        g += (o > d_l) ? oe : 0.0;
        eq += (o == d_l) ? 1 : 0;
      }
      const bool cr = lane < nc && crossed(g + eq * e_l);
      const uint32_t best = __reduce_min_sync(FULL, cr ? dkey_of(d_l) : 0xffffffffu);
      if (best == 0xffffffffu) return WHY_CUT_BELOW;                    // rounding: nothing in the window crosses
      const int who = __ffs(__ballot_sync(FULL, cr && dkey_of(d_l) == best)) - 1;
      dstar = -__uint_as_float(best);
      gb = __shfl_sync(FULL, g, who);
      neq = __shfl_sync(FULL, eq, who);
    }
    // Several logits can share one d: a class that also has members outside the window is decided on the whole row
    if (dstar == dA || dstar == scale_t(nextafterf(xB, -INFINITY), Tm) - m) return WHY_CUT_BELOW;
    // the first member whose mass crosses (mode B keeps through it, mode A everything before it)
    estar = exp_safe(dstar, s_tab);
    if (!crossed(gb + neq * estar)) return WHY_CUT_BELOW;
    int r = 1;
    if (neq > 1) {
      r = static_cast<int>(fmin(fmax(ceil((lim - gb) / estar), 1.0), static_cast<double>(neq)));
      while (r > 1 && crossed(gb + (r - 1) * estar)) r--;
      while (r < neq && !crossed(gb + r * estar)) r++;
    }
    const double etol = (1e-12 + 2.0 * plim * fabs(1.0 - plim) * sh.eps) * S;
    if (fabs(gb + r * estar - lim) <= etol || fabs(gb + (r - 1) * estar - lim) <= etol) flags |= FLAG_TOPP_EDGE;
    if (mode == 1 && r < neq) flags |= FLAG_TIE_CUT;         // the cut separates equal probabilities
    const int kept = (mode == 0) ? r - 1 : r;
    const unsigned long long dk = static_cast<unsigned long long>(dkey_of(dstar)) << 32;
    ties_in = kept == neq;
    cut_key = ties_in ? (dk | 0xffffffffull) : dk;
    cut_incl = ties_in ? 1 : 0;
    by_piece = kept > 0 && (one_class || !ties_in);
    // ---- what the window adds to each warp's part of the row (lane w: warp w); where that already holds all of the window's mass, less
    // all of it
    if (low) for (int j = lane; j < cnt; j += 32) zsum -= (list[j] <= 0.0f) ? mass[j] : 0.0;
    zsum = warp_sum_d(zsum);
    __syncthreads();                                         // (the candidates have been read)
    if (lane == 0) sh.zw[warp] = zsum;
    if (by_piece) {
      // members per piece, then which of them stay: the lowest indices in mode B, the highest in mode A
      bins[tid] = 0u;
      __syncthreads();
      for (int j = lane, q = 0; j < cnt; j += 32) {
        if (list[j] == dstar) {
          while (from[q + 1] <= j) q++;
          atomicAdd(&bins[warp * ppw + q], 1u);
        }
      }
      __syncthreads();
      const int have = (tid < W_NW * ppw) ? static_cast<int>(bins[tid]) : 0;
      const int q = (mode == 0) ? neq - kept + 1 : kept;     // rank, from the lowest index, of the member at the edge
      int incl = have;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(FULL, incl, o); if (lane >= o) incl += t; }
      if (lane == 31) sc.i0[warp] = incl;
      if (tid == 0) { sh.bc[0] = -1; sh.bc[2] = -1; }
      __syncthreads();
      const int pre = incl - have + __reduce_add_sync(FULL, (lane < warp && lane < W_NW) ? sc.i0[lane] : 0);
      const int below = min(max(q - pre, 0), have), strictly = min(max(q - 1 - pre, 0), have);
      bins[tid] = static_cast<uint32_t>((mode == 0) ? have - strictly : below);
      if (have > 0 && pre < q && q <= pre + have) { sh.bc[0] = tid; sh.bc[1] = q - pre; }
      __syncthreads();
      if (!ties_in) {
        // the member's index: one piece of the row again
        const int pi = sh.bc[0], rank = sh.bc[1];
        if (pi < 0) return WHY_CUT_BELOW;
        constexpr int NV = (PV + W_NT - 1) / W_NT;
        const int w = pi / ppw, vb = w * span + (pi - w * ppw) * PV, v = vb + tid * NV;
        const int vend = min(min(vb + PV, w * span + span), rv.nvec);
        uint32_t mask = 0u;
        const int i0 = v * VEC - rv.shift;
#pragma unroll
        for (int h = 0; h < NV; h++) {
          if (tid * NV + h < PV && v + h < vend) {
            float x[VEC];
            Elem<T>::unpack(__ldg(rv.vbase + v + h), x);
#pragma unroll
            for (int c = 0; c < VEC; c++) {
              const int i = i0 + h * VEC + c;
              if (i >= 0 && i < rv.V && x[c] >= xB && x[c] < xA && scale_t(x[c], Tm) - m == dstar) mask |= 1u << (h * VEC + c);
            }
          }
        }
        const int n = __popc(mask);
        int inc = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(FULL, inc, o); if (lane >= o) inc += t; }
        if (lane == 31) sc.i1[warp] = inc;
        __syncthreads();
        const int ahead = inc - n + __reduce_add_sync(FULL, (lane < warp && lane < W_NW) ? sc.i1[lane] : 0);
        if (ahead < rank && rank <= ahead + n) {
          for (int z = rank - ahead; z > 1; z--) mask &= mask - 1u;
          sh.bc[2] = i0 + __ffs(mask) - 1;
        }
        __syncthreads();
        if (sh.bc[2] < 0) return WHY_CUT_BELOW;                         // (a list that disagrees with the row)
        cut_key = zone_key(dstar, sh.bc[2], mode);
        cut_incl = 1;
      }
    } else {
      __syncthreads();
    }
    zw = mine ? sh.zw[lane] : 0.0;
    if (!one_class) {
      // candidates above the class, and the class when all of it stays, count with the warps that listed them
      const double add = (lane < nc && (d_l > dstar || (d_l == dstar && ties_in))) ? e_l : 0.0;
      for (int i = 0; i < nc; i++) {
        const double ae = __shfl_sync(FULL, add, i);
        if (__shfl_sync(FULL, from_l, i) == lane) zw += ae;
      }
    }
    if (by_piece && mine) {
      int stay = 0;
      for (int q = 0; q < ppw; q++) stay += static_cast<int>(bins[lane * ppw + q]);
      zw += estar * stay;
    }
  }
  // ---- kept mass, and the warp in whose part of the row u falls: u < prefix / Re (generate.go:231-239) as u Re < prefix
  const double wv = mine ? sh.kw[lane] * cf + zw : 0.0;
  const double wi = warp_scan_incl_d(wv, lane);
  const double Re = __shfl_sync(FULL, wi, W_NW - 1);
  const double u = A.uniforms[row_id];
  const double tgt = u * Re;
  auto kept_mass = [&](float xv, int i) -> double {          // final rule for one logit: its kept mass (0 when cut away)
    if (i < 0 || i >= rv.V) return 0.0;
    const float d = (t_is_one ? xv : __fdiv_rn(xv, Tm)) - m;
    if (cut_on && !(xv >= xA)) {
      if (!(xv >= xB)) return 0.0;
      const unsigned long long key = zone_key(d, i, mode);
      if (!(key < cut_key || (cut_incl && key == cut_key))) return 0.0;
    }
    return exp_safe(d, s_tab);
  };
  const int how = (cut_on ? HOW_CUT | sh.placed : 0) | (one_class ? HOW_ONE_CLASS : 0) | (by_piece ? HOW_BY_PIECE : 0) | (by_piece && !ties_in ? HOW_INDEX : 0) | (exact ? HOW_EXACT : 0);
  if (!(Re > 0.0)) {                                         // mode A removed every token
    wide_write_nothing_kept(A, row_id, m, S, 3, 0, how, flags);
    return 0;
  }
  WideResult res;
  res.m = m; res.S = S; res.Re = Re; res.path = 3; res.why = 0; res.how = how;
  int psel = 0x7fffffff;
  double before = Re;
  const unsigned hit = __ballot_sync(FULL, mine && tgt < wi);
  if (hit) {                                                 // uniform: the same bits in every warp
    const int ws = __ffs(hit) - 1;
    const double base = __shfl_sync(FULL, wi - wv, ws);
    for (int q = warp; q < ppw; q += W_NW) {                 // that warp's pieces, by all warps
      double zp = 0.0;
      if (cut_on) {
        const float* lw = reinterpret_cast<const float*>(dyn + W1_OFF_LIST) + ws * W1_WCAP;
        const double* mw = reinterpret_cast<const double*>(dyn + W1_OFF_MASS) + ws * W1_WCAP;
        const int* fw = reinterpret_cast<const int*>(dyn + W1_OFF_FROM) + ws * (W_MAX_PPW + 1);
        const int j1 = fw[q + 1];
        for (int j = fw[q] + lane; j < j1; j += 32) {
          const float d = lw[j];
          if (d <= 0.0f) {
            const bool in = d > dstar || (d == dstar && ties_in && !by_piece);
            zp += in ? (low ? 0.0 : mw[j]) : (low ? -mw[j] : 0.0);
          }
        }
        zp = warp_sum_d(zp);
        if (by_piece) zp += estar * static_cast<int>(bins[ws * ppw + q]);
      }
      if (lane == 0) sh.pm[q] = part[ws * ppw + q] * cf + zp;
    }
    __syncthreads();
    const double pv = (lane < ppw) ? sh.pm[lane] : 0.0;
    const double pi = base + warp_scan_incl_d(pv, lane);
    const unsigned in = __ballot_sync(FULL, lane < ppw && tgt < pi);
    const int q = in ? __ffs(in) - 1 : ppw - 1;              // (rounding: the warp's last piece, from which the walk goes on)
    psel = ws * ppw + q;
    before = __shfl_sync(FULL, pi - pv, q);
  }
  wide_draw<T>(A, row_id, rv, span, ppw, psel, before, u, res, flags, sh, kept_mass);
  return 0;
}
