// Ground state: integral blocks, DIIS and the CCSD amplitude equations
// (ugacc ccwfn.cc:12-120, :188-626).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "cc.h"

namespace ucc {

void tc_forget(Ctx& c, const double* p, size_t n);  // tc_gemm.cu

// ---------------------------------------------------------------------------------------
// Integral blocks
// ---------------------------------------------------------------------------------------
Tensor narrow(const Tensor& t, int axis, int64_t start, int64_t len) {
  Tensor r = t;
  r.p = t.p + start * t.s[axis];
  r.d[axis] = len;
  return r;
}

static void store_fock(Ctx& c, const double* fock) {
  const int no = c.no, nv = c.nv, n = no + nv;
  c.fock.assign(fock, fock + (size_t)n * n);
  c.eps.resize(n);
  for (int p = 0; p < n; p++) c.eps[p] = fock[(size_t)p * n + p];
  auto put = [&](const char* name, int r0, int nr, int c0, int nc) {
    std::vector<double> h((size_t)nr * nc);
    for (int i = 0; i < nr; i++)
      for (int j = 0; j < nc; j++) h[(size_t)i * nc + j] = fock[(size_t)(r0 + i) * n + c0 + j];
    Tensor t = c.alloc(name, {nr, nc}, false);
    UCC_CUDA(cudaMemcpyAsync(t.p, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice, c.stream));
    UCC_CUDA(cudaStreamSynchronize(c.stream));
  };
  put("foo", 0, no, 0, no);
  put("fov", 0, no, no, nv);
  put("fvo", no, nv, 0, no);
  put("fvv", no, nv, no, nv);
  Tensor e = c.alloc("eps", {n}, false);
  UCC_CUDA(cudaMemcpyAsync(e.p, c.eps.data(), n * sizeof(double), cudaMemcpyHostToDevice, c.stream));
  UCC_CUDA(cudaStreamSynchronize(c.stream));
}

static const char* kStored[] = {"oooo", "ooov", "oovv", "ovov", "ovvv", "vvvv"};

static void build_L_blocks(Ctx& c) {
  const int no = c.no, nv = c.nv;
  auto two_minus = [&](const char* name, const Tensor& X, const Tensor& Xswap) {
    std::vector<int64_t> dims(X.d, X.d + X.rank);
    Tensor out = c.alloc(name, dims, false);
    permute_add(c, Xswap, -1.0, 0.0, out);
    permute_add(c, X, 2.0, 1.0, out);
  };
  Tensor Voovv = c.get("Voovv"), Vooov = c.get("Vooov"), Vovvv = c.get("Vovvv"), Vovov = c.get("Vovov");
  two_minus("Loovv", Voovv, view(Voovv, "ijab->ijba"));
  two_minus("Looov", Vooov, view(Vooov, "mnie->nmie"));
  two_minus("Lovvv", Vovvv, view(Vovvv, "mafe->maef"));
  // L[n,a,f,i] = 2 <ni|fa> - <na|if>
  two_minus("Lovvo", view(Voovv, "nifa->nafi"), view(Vovov, "naif->nafi"));
  (void)no;
  (void)nv;
}

static void choose_pair_rows(Ctx& c) {
  size_t free_b = 0, total_b = 0;
  UCC_CUDA(cudaMemGetInfo(&free_b, &total_b));
  c.pair_rows = ccsd_bytes(c.no, c.nv) <= kPairRowsShare * (double)total_b;
}

void load_from_ints(Ctx& c, int no, int nv, const double* fock, const double* ints) {
  c.no = no;
  c.nv = nv;
  c.naux = 0;
  store_fock(c, fock);
  const int64_t n = no + nv;
  for (const char* blk : kStored) {
    int64_t lo[4], len[4];
    for (int k = 0; k < 4; k++) {
      lo[k] = blk[k] == 'o' ? 0 : no;
      len[k] = blk[k] == 'o' ? no : nv;
    }
    std::vector<double> h((size_t)len[0] * len[1] * len[2] * len[3]);
    size_t w = 0;
    for (int64_t p = 0; p < len[0]; p++)
      for (int64_t q = 0; q < len[1]; q++)
        for (int64_t r = 0; r < len[2]; r++) {
          const double* src = ints + (((lo[0] + p) * n + lo[1] + q) * n + lo[2] + r) * n + lo[3];
          std::memcpy(&h[w], src, sizeof(double) * len[3]);
          w += len[3];
        }
    Tensor t = c.alloc(std::string("V") + blk, {len[0], len[1], len[2], len[3]}, false);
    UCC_CUDA(cudaMemcpyAsync(t.p, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice, c.stream));
    UCC_CUDA(cudaStreamSynchronize(c.stream));
  }
  build_L_blocks(c);
  choose_pair_rows(c);
  UCC_CUDA(cudaStreamSynchronize(c.stream));
}

void load_from_df(Ctx& c, int no, int nv, int naux, const double* fock, const double* Bh) {
  c.no = no;
  c.nv = nv;
  c.naux = naux;
  store_fock(c, fock);
  const int64_t n = no + nv;
  Tensor B = c.alloc("Bdf", {naux, n, n}, false);
  UCC_CUDA(cudaMemcpyAsync(B.p, Bh, sizeof(double) * naux * n * n, cudaMemcpyHostToDevice, c.stream));
  const bool saved = c.force_fp64;
  c.force_fp64 = true;  // the Hamiltonian itself is always built in FP64
  for (const char* blk : kStored) {
    int64_t lo[4], len[4];
    for (int k = 0; k < 4; k++) {
      lo[k] = blk[k] == 'o' ? 0 : no;
      len[k] = blk[k] == 'o' ? no : nv;
    }
    Tensor X = c.alloc(std::string("V") + blk, {len[0], len[1], len[2], len[3]}, false);
    // <pq|rs> = (pr|qs) = sum_Q B[Q,p,r] B[Q,q,s], chunked over p to bound the scratch
    const int64_t per_p = len[1] * len[2] * len[3];
    const int64_t chunk = std::max<int64_t>(1, std::min<int64_t>(len[0], (int64_t)(256LL << 20) / per_p));
    Tensor Bqs = narrow(narrow(B, 1, lo[1], len[1]), 2, lo[3], len[3]);
    for (int64_t p0 = 0; p0 < len[0]; p0 += chunk) {
      const int64_t np = std::min(chunk, len[0] - p0);
      Tensor Bpr = narrow(narrow(B, 1, lo[0] + p0, np), 2, lo[2], len[2]);
      Tensor Xc = narrow(X, 0, p0, np);
      contract(c, "Qpr,Qqs->pqrs", 1.0, Bpr, Bqs, 0.0, Xc);
    }
  }
  c.force_fp64 = saved;
  c.drop("Bdf");
  build_L_blocks(c);
  choose_pair_rows(c);
  UCC_CUDA(cudaStreamSynchronize(c.stream));
}

Tensor V(Ctx& c, const std::string& b) {
  for (const char* s : kStored)
    if (b == s) return c.get("V" + b);
  if (b == "oovo") return view(c.get("Vooov"), "nmje->mnej");
  if (b == "ovvo") return view(c.get("Voovv"), "mjeb->mbej");
  if (b == "ovoo") return view(c.get("Vooov"), "mjib->mbij");
  if (b == "vovv") return view(c.get("Vovvv"), "mafe->amef");
  if (b == "vvvo") return view(c.get("Vovvv"), "iabe->abei");
  if (b == "vovo") return view(c.get("Vovov"), "maie->amei");
  if (b == "voov") return view(c.get("Voovv"), "mieb->bmie");
  throw Error(UCC_BAD_ARGS, "no integral block " + b);
}

Tensor L(Ctx& c, const std::string& b) {
  if (b == "oovv" || b == "ooov" || b == "ovvv" || b == "ovvo") return c.get("L" + b);
  if (b == "oovo") return view(c.get("Looov"), "mnie->nmei");
  if (b == "vovv") return view(c.get("Lovvv"), "mafe->amef");
  throw Error(UCC_BAD_ARGS, "no L block " + b);
}

Tensor Fk(Ctx& c, const std::string& b) { return c.get("f" + b); }

// ---------------------------------------------------------------------------------------
// DIIS
// ---------------------------------------------------------------------------------------
Diis::Diis(Ctx& c, int64_t n, int nmax)
    : c_(c), n_(n), nmax_(nmax), err_((size_t)n * nmax, c.stream), vec_((size_t)n * nmax, c.stream),
      B_((size_t)nmax * nmax, 0.0) {}

void Diis::overlaps(double* out) {
  VecList e;
  const int cnt = std::min(count_ + 1, nmax_);
  for (int p = 0; p < cnt; p++) e.p[p] = err_.p + (size_t)p * n_;
  multidot_async(c_, cnt, e, err(), n_, out);
}

void Diis::accept(const HostBlock& h, int first) {
  const int s = slot(), cnt = std::min(count_ + 1, nmax_);
  for (int p = 0; p < cnt; p++) B_[(size_t)s * nmax_ + p] = B_[(size_t)p * nmax_ + s] = h[first + p];
  count_ = cnt;
  nadded_++;
}

std::vector<double> diis_coefficients(const std::vector<double>& Bin, int n) {
  const int m = n + 1;
  std::vector<double> B((size_t)m * m, 0.0), c(m, 0.0);
  double mx = 0.0;
  for (int p = 0; p < n; p++)
    for (int q = 0; q < n; q++) {
      B[p * m + q] = Bin[(size_t)p * n + q];
      mx = std::max(mx, std::fabs(B[p * m + q]));
    }
  if (mx > 0.0)
    for (int p = 0; p < n; p++)
      for (int q = 0; q < n; q++) B[p * m + q] /= mx;
  for (int p = 0; p < n; p++) B[p * m + n] = B[n * m + p] = -1.0;
  B[n * m + n] = 0.0;
  c[n] = -1.0;
  for (int col = 0; col < m; col++) {
    int piv = col;
    for (int r = col + 1; r < m; r++)
      if (std::fabs(B[r * m + col]) > std::fabs(B[piv * m + col])) piv = r;
    if (piv != col) {
      for (int k = 0; k < m; k++) std::swap(B[col * m + k], B[piv * m + k]);
      std::swap(c[col], c[piv]);
    }
    const double d = B[col * m + col];
    UCC_REQUIRE(d != 0.0, UCC_NAN_DETECTED, "DIIS: singular B matrix");
    for (int r = col + 1; r < m; r++) {
      const double f = B[r * m + col] / d;
      if (f == 0.0) continue;
      for (int k = col; k < m; k++) B[r * m + k] -= f * B[col * m + k];
      c[r] -= f * c[col];
    }
  }
  for (int r = m - 1; r >= 0; r--) {
    double s = c[r];
    for (int k = r + 1; k < m; k++) s -= B[r * m + k] * c[k];
    c[r] = s / B[r * m + r];
  }
  c.resize(n);
  return c;
}

void Diis::reset() {
  count_ = 0;
  nadded_ = 0;
  std::fill(B_.begin(), B_.end(), 0.0);
}

void Diis::extrapolate(double* out) {
  const int n = count_;
  std::vector<double> Bn((size_t)n * n);
  for (int p = 0; p < n; p++)
    for (int q = 0; q < n; q++) Bn[(size_t)p * n + q] = B_[(size_t)p * nmax_ + q];
  const std::vector<double> coef = diis_coefficients(Bn, n);
  VecList v;
  for (int p = 0; p < n; p++) v.p[p] = vec_.p + (size_t)p * n_, v.coef[p] = coef[p];
  lincomb(c_, n, v, n_, out);
}

// ---------------------------------------------------------------------------------------
// CCSD (ccwfn.cc:188-626)
// ---------------------------------------------------------------------------------------
double flops_ccsd_iter(double no, double nv) {
  return 2.0 * (no * no * nv * nv * nv * nv + 2.0 * no * no * no * no * nv * nv + 10.0 * no * no * no * nv * nv * nv +
                8.0 * no * no * nv * nv * nv);
}

// Two blocks that are there together and filled, or not at all: their presence says that they are built.
template <typename F>
static void build_blocks(Ctx& c, const char* p, const std::vector<int64_t>& pdims, const char* m,
                         const std::vector<int64_t>& mdims, F&& fill) {
  if (c.has(p)) return;
  try {
    Tensor P = c.alloc(p, pdims, false), M = c.alloc(m, mdims, false);
    fill(P.p, M.p);
  } catch (...) {
    c.drop(p);
    c.drop(m);
    throw;
  }
}

void pair_operator(Ctx& c) {
  const int64_t no = c.no, nv = c.nv, vp = nv * (nv + 1) / 2, vm = nv * (nv - 1) / 2, mb = c.pair_rows ? no * nv : 0;
  build_blocks(c, "Vpp", {vp + mb, vp}, "Vmm", {vm + mb, vm}, [&](double* P, double* M) {
    pack_vvvv(c, c.nv, 0, c.get("Vvvvv").p, P, M);
    if (mb) pack_ovvv(c, c.no, c.nv, c.get("Vovvv").p, P + vp * vp, M + vm * vm);
  });
}

double ccsd_bytes(int64_t no, int64_t nv) {
  const double o = (double)no, v = (double)nv;
  // <ab|ef> and half of it packed; <ma|ef>, its L form, a gathered copy and the packed rows; vectors of the
  // length of t2: 16 of DIIS, 6 blocks of integrals, amplitudes, residual and tau, a sweep's scratch
  return 8.0 * (1.5 * v * v * v * v + 4.0 * o * v * v * v + 36.0 * o * o * v * v);
}

bool release_pair_operator(Ctx& c, bool rows) {
  if (rows ? !c.pair_rows : !c.has("Vpp")) return false;
  c.pair_rows = false;
  UCC_CUDA(cudaStreamSynchronize(c.stream));
  for (const char* k : {"Vpp", "Vmm"})
    if (c.has(k)) {
      const DeviceBuffer& b = *c.store.at(k);
      tc_forget(c, b.p, b.n);
      c.drop(k);
    }
  UCC_CUDA(cudaStreamSynchronize(c.stream));
  trim_pool(c.device);
  return true;
}

// R2 += alpha sum_ef W_abef amp_ijef on packed pairs (pairs.cu), W from an HBAR block: S = Tp Vp^T
// over (i<=j, a<=b, e<=f) and A = Tm Vm^T over strict pairs, a quarter of the multiply-adds of
// the plain contraction; amp must be invariant under (i,j,e,f) -> (j,i,f,e).  The packed
// operator (names vp_name / vm_name, constant blocks) is built from block `src` once; mode 1
// stores it as [e<=f][a<=b].
void packed_ladder(Ctx& c, double alpha, const Tensor& amp, const char* src, int mode, const char* vp_name,
                   const char* vm_name, double* R2) {
  const int no = c.no, nv = c.nv;
  const int64_t op = (int64_t)no * (no + 1) / 2, om = (int64_t)no * (no - 1) / 2;
  const int64_t vp = (int64_t)nv * (nv + 1) / 2, vm = (int64_t)nv * (nv - 1) / 2;
  build_blocks(c, vp_name, {vp, vp}, vm_name, {vm, vm},
               [&](double* P, double* M) { pack_vvvv(c, nv, mode, c.get(src).p, P, M); });
  UCC_REQUIRE(amp.dense(), UCC_BAD_ARGS, "packed ladder: dense amplitudes");
  Temp Tp(c, {op, vp}), Tm(c, {om, vm}), S(c, {op, vp}), A(c, {om, vm});
  pack_tau(c, no, nv, amp.p, Tp->p, Tm->p);
  const char* spec = mode == 1 ? "pe,eq->pq" : "pe,qe->pq";
  contract(c, spec, 1.0, Tp, c.get(vp_name), 0.0, S);
  contract(c, spec, 1.0, Tm, c.get(vm_name), 0.0, A);
  unpack_ladder(c, no, nv, alpha, S->p, A->p, R2);
}

namespace {

void copy_into(Ctx& c, const Tensor& src, Tensor dst) { permute_add(c, src, 1.0, 0.0, dst); }

// build_F, ccwfn.cc:311-356
void build_F(Ctx& c, const Tensor& t1, const Tensor& ttau) {
  Tensor Fvv = c.get("Fvv"), Foo = c.get("Foo"), Fov = c.get("Fov");
  copy_into(c, Fk(c, "vv"), Fvv);
  contract(c, "me,ma->ae", -0.5, Fk(c, "ov"), t1, 1.0, Fvv);
  contract(c, "mf,mafe->ae", 1.0, t1, L(c, "ovvv"), 1.0, Fvv);
  contract(c, "mnaf,mnef->ae", -1.0, ttau, L(c, "oovv"), 1.0, Fvv);
  copy_into(c, Fk(c, "oo"), Foo);
  contract(c, "ie,me->mi", 0.5, t1, Fk(c, "ov"), 1.0, Foo);
  contract(c, "ne,mnie->mi", 1.0, t1, L(c, "ooov"), 1.0, Foo);
  contract(c, "inef,mnef->mi", 1.0, ttau, L(c, "oovv"), 1.0, Foo);
  copy_into(c, Fk(c, "ov"), Fov);
  contract(c, "nf,mnef->me", 1.0, t1, L(c, "oovv"), 1.0, Fov);
}

// Products of tau with the packed operator, one GEMM per symmetry: the particle ladder's rows
// (a <= b) and, with c.pair_rows, the (m, b) rows of Zmbij = sum_ef <mb|ef> tau_ijef below them.  A
// batch whose members' packed operators would not fit in memory goes without (S and A stay null).
struct PairProducts {
  std::unique_ptr<Temp> S, A;
  bool rows = false;  // Zmbij is there
  PairProducts(Ctx& c, const Tensor& tau) {
    if (recorder() && !recorder()->packed) return;
    const int64_t no = c.no, nv = c.nv, op = no * (no + 1) / 2, om = no * (no - 1) / 2;
    const int64_t vp = nv * (nv + 1) / 2, vm = nv * (nv - 1) / 2;
    if (!recorder()) pair_operator(c);
    rows = c.get("Vpp").d[0] > vp;
    S = std::make_unique<Temp>(c, std::vector<int64_t>{op, c.get("Vpp").d[0]});
    A = std::make_unique<Temp>(c, std::vector<int64_t>{om, c.get("Vmm").d[0]});
    Temp Tp(c, {op, vp}), Tm(c, {om, vm});
    pack_tau(c, c.no, c.nv, tau.p, Tp->p, Tm->p);
    product(c, Tp, c.get("Vpp"), S->t);
    product(c, Tm, c.get("Vmm"), A->t);
  }
  const double* s() const { return S ? S->t.p : nullptr; }
  const double* a() const { return A ? A->t.p : nullptr; }
  int64_t lds() const { return S ? S->t.d[1] : 0; }
  int64_t lda() const { return A ? A->t.d[1] : 0; }

 private:
  // out = T Op^T; a batch records it whatever the member's size, so that all members record
  // the same operations (no = 1: no strict pairs of occupied indices, nv = 1: K = 0)
  static void product(Ctx& c, const Tensor& T, const Tensor& Op, const Tensor& out) {
    if (recorder()) {
      GemmEpilogue epi;
      epi.s_mhi = out.d[1];
      dgemm_strided(c, T.d[0], Op.d[0], T.d[1], 1.0, T.p, T.d[1], 1, Op.p, 1, T.d[1], 0.0, out.p, epi, 1, 0, 0, 0,
                    nullptr);
    } else if (out.size() && !T.d[1]) {
      fill(c, out.size(), 0.0, out.p);
    } else {
      contract(c, "pe,qe->pq", 1.0, T, Op, 0.0, out);
    }
  }
};

// build_W, ccwfn.cc:358-430, with the two ring intermediates
//   Wovov[m,b,j,e]  (:390-404)  and  B = 2 Wovvo + Wovov(..je->..ej):
// in B the amplitude products of Wovvo (:406-424) and Wovov collapse to one,
//   B[m,b,e,j] = L_mbej + t1_jf L_mbef - t1_nb L_mnej + L_mnef P_jnfb,  P = t2(jnbf) - X,
// so two products over (n, f) do the work of three (tests/test_ring_algebra.py).
void build_W(Ctx& c, const Tensor& t1, const Tensor& tau, const Tensor& X, const Tensor& P) {
  Tensor Woooo = c.get("Woooo"), Wovov = c.get("Wovov"), Bovvo = c.get("Bovvo");
  copy_into(c, V(c, "oooo"), Woooo);
  contract(c, "je,mnie->mnij", 1.0, t1, V(c, "ooov"), 1.0, Woooo);
  contract(c, "ie,mnej->mnij", 1.0, t1, V(c, "oovo"), 1.0, Woooo);
  contract(c, "ijef,mnef->mnij", 1.0, tau, V(c, "oovv"), 1.0, Woooo);
  permute_add(c, V(c, "ovov"), -1.0, 0.0, Wovov);
  contract(c, "jf,mbfe->mbje", -1.0, t1, V(c, "ovvv"), 1.0, Wovov);
  contract(c, "nb,mnje->mbje", 1.0, t1, V(c, "ooov"), 1.0, Wovov);
  contract(c, "mnfe,jnfb->mbje", 1.0, V(c, "oovv"), X, 1.0, Wovov);
  copy_into(c, L(c, "ovvo"), Bovvo);
  contract(c, "jf,mbef->mbej", 1.0, t1, L(c, "ovvv"), 1.0, Bovvo);
  contract(c, "nb,mnej->mbej", -1.0, t1, L(c, "oovo"), 1.0, Bovvo);
  contract(c, "mnef,jnfb->mbej", 1.0, L(c, "oovv"), P, 1.0, Bovvo);
}

// build_t1, ccwfn.cc:432-469 (unscaled residual); S = t2 - t2(ba)/2
void build_t1(Ctx& c, const Tensor& t1, const Tensor& t2, const Tensor& S, Tensor R1) {
  transpose_add(c, "ai->ia", 1.0, Fk(c, "vo"), 0.0, R1);
  contract(c, "ie,ae->ia", 1.0, t1, c.get("Fvv"), 1.0, R1);
  contract(c, "ma,mi->ia", -1.0, t1, c.get("Foo"), 1.0, R1);
  contract(c, "imae,me->ia", 2.0, S, c.get("Fov"), 1.0, R1);
  contract(c, "nf,nafi->ia", 1.0, t1, L(c, "ovvo"), 1.0, R1);
  contract(c, "mief,maef->ia", 2.0, S, V(c, "ovvv"), 1.0, R1);
  contract(c, "mnae,nmei->ia", -1.0, t2, L(c, "oovo"), 1.0, R1);
}

// build_t2, ccwfn.cc:471-539 (unscaled residual).
//
// The residual is symmetric under the simultaneous swap (i<->j, a<->b): the reference
// computes each term and its swapped partner explicitly.  Here one member of each pair (half
// of the self-symmetric hole ladder) goes into a half residual Rh, the exchange ring
// t2_imea Wovov_mbje into H, whose half and whose (i,j,b,a) transpose are the last two of the
// reference's ring terms, and assemble_r2 adds <ij|ab>, the particle ladder, Q and Q(ji,ba)
// with Q = Rh + H/2 + H(ijba) in one pass.
void build_t2(Ctx& c, const Tensor& t1, const Tensor& t2, const Tensor& tau, const Tensor& S,
              const PairProducts& pairs, Tensor R2) {
  const int no = c.no, nv = c.nv;
  Tensor Fvv = c.get("Fvv"), Foo = c.get("Foo"), Fov = c.get("Fov");
  Tensor Woooo = c.get("Woooo"), Wovov = c.get("Wovov"), Bovvo = c.get("Bovvo");
  Temp Rh(c, {no, no, nv, nv}), H(c, {no, no, nv, nv});
  {
    Temp F1(c, {nv, nv}), F2(c, {no, no});  // Fvv - t1 Fov / 2, Foo + t1 Fov / 2
    copy_into(c, Fvv, F1);
    contract(c, "mb,me->be", -0.5, t1, Fov, 1.0, F1);
    copy_into(c, Foo, F2);
    contract(c, "je,me->mj", 0.5, t1, Fov, 1.0, F2);
    contract(c, "ijae,be->ijab", 1.0, t2, F1, 0.0, Rh);
    contract(c, "imab,mj->ijab", -1.0, t2, F2, 1.0, Rh);
  }
  contract(c, "mnab,mnij->ijab", 0.5, tau, Woooo, 1.0, Rh);
  contract(c, "ie,abej->ijab", 1.0, t1, V(c, "vvvo"), 1.0, Rh);
  contract(c, "imae,mbej->ijab", 1.0, S, Bovvo, 1.0, Rh);
  contract(c, "imea,mbje->ijab", 1.0, t2, Wovov, 0.0, H);
  {
    // Za[m,b,i,j] = <mb|ij> + Zmbij + t1[i,e] <mb|ej> + t1[j,e] <mb|ie>  ->  - t1[m,a] Za[m,b,i,j]
    Temp Za(c, {no, nv, no, no});
    if (pairs.rows)
      unpack_z(c, no, nv, pairs.s(), pairs.a(), Za->p);
    else
      contract(c, "mbef,ijef->mbij", 1.0, V(c, "ovvv"), tau, 0.0, Za);
    permute_add(c, V(c, "ovoo"), 1.0, 1.0, Za);
    contract(c, "ie,mbej->mbij", 1.0, t1, V(c, "ovvo"), 1.0, Za);
    contract(c, "je,mbie->mbij", 1.0, t1, V(c, "ovov"), 1.0, Za);
    contract(c, "ma,mbij->ijab", -1.0, t1, Za, 1.0, Rh);
  }
  if (!pairs.s()) contract(c, "ijef,abef->ijab", 0.5, tau, V(c, "vvvv"), 1.0, Rh);
  assemble_r2(c, no, nv, V(c, "oovv").p, pairs.s(), pairs.lds(), pairs.a(), pairs.lda(), Rh->p, H->p, R2.p);
}

// the unscaled residual R(t_old) into r, given tau/ttau of t_old (ccwfn.cc:311-539); ev
// collects event pairs around the packed products
void residual(Ctx& c, const double* t_old, double* r, std::vector<cudaEvent_t>* ev) {
  const int no = c.no, nv = c.nv;
  Tensor t1 = amp1(c, const_cast<double*>(t_old)), t2 = amp2(c, const_cast<double*>(t_old)), tau = c.get("tau");
  build_F(c, t1, c.get("ttau"));
  cudaEvent_t a = nullptr, b = nullptr;
  if (ev) {
    pair_operator(c);  // once per Hamiltonian: not in the products' time
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    cudaEventRecord(a, c.stream);
  }
  PairProducts pairs(c, tau);
  if (ev) {
    cudaEventRecord(b, c.stream);
    ev->push_back(a);
    ev->push_back(b);
  }
  Temp S(c, {no, no, nv, nv});
  {
    Temp X(c, {no, no, nv, nv}), P(c, {no, no, nv, nv});
    ring_amplitudes(c, no, nv, t1.p, t2.p, X->p, P->p, S->p);
    build_W(c, t1, tau, X, P);
  }
  build_t1(c, t1, t2, S, amp1(c, r));
  build_t2(c, t1, t2, tau, S, pairs, amp2(c, r));
}

// ccwfn.cc:270-273 assigns instead of accumulating: only the last (i,a) pair counts
struct Energy {
  DotList d;
  double fov;
  int two, last;
  Energy(Ctx& c, const Tensor& t1, const Tensor& tau)
      : d(c), fov(c.fock[(size_t)(c.no - 1) * (c.no + c.nv) + (c.no + c.nv - 1)]) {
    two = dot_all(c, tau, L(c, "oovv"), d);
    last = d.add(1, t1.p + (int64_t)c.no * c.nv - 1, nullptr);
  }
  double value() const { return 2.0 * fov * d[last] + d[two]; }  // after a wait for the stream
};

}  // namespace

// CCSD work arrays of one context (amplitudes packed as [t1 | t2])
void ccsd_alloc(Ctx& c) {
  const int no = c.no, nv = c.nv;
  const int64_t np = npacked(c);
  c.alloc("T", {np}, false);
  c.alloc("Told", {np}, true);
  c.alloc("R", {np}, false);
  c.alloc("tau", {no, no, nv, nv}, false);
  c.alloc("ttau", {no, no, nv, nv}, false);
  c.alloc("Fvv", {nv, nv}, false);
  c.alloc("Foo", {no, no}, false);
  c.alloc("Fov", {no, nv}, false);
  c.alloc("Woooo", {no, no, no, no}, false);
  c.alloc("Wovov", {no, nv, no, nv}, false);
  c.alloc("Bovvo", {no, nv, nv, no}, false);
}

void ccsd_residual(Ctx& c, const double* t_old, double* r) { residual(c, t_old, r, nullptr); }

double ccsd_energy(Ctx& c, const double* t) {
  Energy e(c, amp1(c, const_cast<double*>(t)), c.get("tau"));
  e.d.fetch();
  return e.value();
}

// residual norm near which BF16 hi+lo split products with FP32 accumulation stop
// resolving the update (measured ~1.5e-6 at no=16/nv=160)
constexpr double kMixedFloor = 2e-6;
// delta sweeps resolve residuals down to ~3e-5 of their anchor's residual (measured at
// no=32/nv=320: an anchor at 4.3e-5 left the delta residuals 1.3e-9 off), so an anchor
// above kReanchor * r_convergence is re-taken once the deltas reach that level
constexpr double kReanchor = 1e4;

MixedSweeps::MixedSweeps(Ctx& c)
    : c_(c),
      mixed_(c.opt.precision == UCC_MIXED),
      refine_(c.opt.precision == UCC_MIXED && c.opt.refine_sweeps > 0),
      split_phase_(c.opt.precision == UCC_MIXED) {
  c_.anchors.clear();
}

MixedSweeps::~MixedSweeps() { c_.anchors.clear(); }

// Truncating each operand to S base-2^6 digits leaves a relative error near 2^-6S in every
// product term; the digits cover the target level's bits plus a margin of kDigitMarginBits
// for the sum over K and the spread of the operands' magnitudes (an anchor error shows as a
// delta residual that stalls above the target, which re-anchors with all digits).
constexpr int kDigitMarginBits = 14;

int MixedSweeps::record_digits() const {
  if (!(record_target_ > 0.0)) return 9;
  const int d = (int)std::ceil((std::log2(1.0 / record_target_) + kDigitMarginBits) / 6.0);
  return std::min(9, std::max(4, d));
}

MixedSweeps::Kind MixedSweeps::begin() {
  kind_ = !mixed_ ? kFp64 : split_phase_ ? kSplit : record_next_ ? kRecord : kDelta;
  if (kind_ == kRecord) {
    c_.anchors.begin(1);
    digits_ = record_digits();
    c_.anchors.digits = digits_;
  }
  if (kind_ == kDelta) c_.anchors.begin(2);
  return kind_;
}

void MixedSweeps::end() {
  c_.anchors.mode = 0;
  c_.anchors.digits = 9;
}

bool MixedSweeps::after(double rms, bool* restart_diis) {
  *restart_diis = false;
  sweeps_++;
  const double rc = c_.opt.r_convergence;
  bool done = false;
  if (kind_ == kFp64) {
    done = rms < rc;
  } else if (kind_ == kSplit) {
    split++;
    if (!refine_ && rms < rc) done = true;
    // hand over near the split-product noise floor, or when the residual stops falling
    // within three decades of it: two sweeps in a row that do not halve it (one slow sweep
    // is common early on: from a learned guess at no=32/nv=320 the norm went 1.0e-2 ->
    // 5.3e-3, and handing over there left 10 delta sweeps to do instead of 7)
    const double level = std::max(rc, std::max(c_.opt.mixed_switch, kMixedFloor));
    split_slow_ = (sweeps_ > 2 && rms < 1e3 * level && rms > 0.5 * rms_prev_) ? split_slow_ + 1 : 0;
    if (!done && refine_ && (rms < level || split_slow_ >= 2)) {
      split_phase_ = false;
      record_next_ = true;
      // the deltas after this anchor run down to the re-anchoring level, or to r_convergence
      record_target_ = rms > kReanchor * rc ? kReanchor * rc : rc;
      *restart_diis = true;  // the split-sweep history extrapolates a different map
    }
  } else if (kind_ == kRecord) {
    record++;
    record_next_ = false;
    stalls_ = 0;
    anchor_rms_ = rms;
    // only a residual from products with all digits ends the solve
    done = rms < rc && record >= c_.opt.refine_sweeps && digits_ == 9;
    if (!done && rms < rc && digits_ < 9) {
      record_next_ = true;
      record_target_ = 0.0;
    }
    // the FP64 residual is well above what the last delta sweep reported: those sweeps'
    // anchor was too far away and their vectors would mislead the extrapolation
    if (!done && last_ == kDelta && rms > 2.0 * rms_prev_) *restart_diis = true;
  } else {
    delta++;
    if (rms < rc) {
      record_next_ = true;  // confirm with an FP64 residual
      record_target_ = 0.0;
    } else if (anchor_rms_ > kReanchor * rc && rms < kReanchor * rc) {
      record_next_ = true;  // the anchor is too far for the deltas to resolve rc: re-anchor here
      record_target_ = rc;
    } else if (rms > 0.7 * rms_prev_) {
      if (++stalls_ >= 2) {  // corrections no longer resolved: re-anchor
        record_next_ = true;
        record_target_ = 0.0;
      }
    } else {
      stalls_ = 0;
    }
  }
  rms_prev_ = rms;
  last_ = kind_;
  return done;
}

CCSDResult run_ccsd(Ctx& c) {
  UCC_REQUIRE(c.loaded, UCC_BAD_STATE, "no Hamiltonian loaded");
  const int no = c.no, nv = c.nv;
  const int64_t np = npacked(c);
  ccsd_alloc(c);
  Tensor T = c.get("T"), Told = c.get("Told");
  Tensor eps = c.get("eps");
  const double* d_do = eps.p;
  const double* d_dv = eps.p + no;
  HostBlock sums(c);  // of a sweep: sum of squares, then the DIIS overlaps

  // MP2 guess t1 = f_ia / D1, t2 = <ij|ab> / D2 (ccwfn.cc:75-87), unless amplitudes were given
  if (!c.has("T_guess")) {
    Temp R0(c, {np}, true);
    copy_into(c, Fk(c, "ov"), amp1(c, R0->p));
    copy_into(c, V(c, "oovv"), amp2(c, R0->p));
    jacobi_update(c, no, nv, d_do, d_dv, 0.0, R0->p, R0->p + (int64_t)no * nv, Told.p, Told.p + (int64_t)no * nv, T.p,
                  T.p + (int64_t)no * nv, sums.p);
  } else {  // a supplied guess (restart file, learned guess) applies to this solve only
    UCC_CUDA(cudaMemcpyAsync(T.p, c.get("T_guess").p, sizeof(double) * np, cudaMemcpyDeviceToDevice, c.stream));
    UCC_CUDA(cudaStreamSynchronize(c.stream));
    if (c.pair_rows)
      c.taken = "T_guess";  // kept for a second attempt (release_pair_operator)
    else
      c.drop("T_guess");
  }
  auto tau_of = [&](double* buf) {
    build_tau(c, no, nv, buf, buf + (int64_t)no * nv, 1.0, c.get("tau").p, 0.5, c.get("ttau").p);
  };
  tau_of(c.get("T").p);
  CCSDResult res;
  auto en = std::make_unique<Energy>(c, amp1(c, c.get("T").p), c.get("tau"));
  en->d.fetch();
  res.e_mp2 = en->value();
  en.reset();
  if (c.opt.print) {
    std::printf("\n\tThe Coupled-Cluster Iteration:\n");
    std::printf("\t---------------------------------------------------\n");
    std::printf("\t Iter   Correlation Energy   T1 Norm      RMS   \n");
    std::printf("\t---------------------------------------------------\n");
    std::printf("\t  %3d  %20.15f\n", 0, res.e_mp2);
  }
  Diis diis(c, np, 8);
  std::vector<cudaEvent_t> ev;
  // a solve that stops in its first sweep reports the energy of its starting amplitudes, as any
  // other reports that of the amplitudes its last sweep started from
  double rms = INFINITY, eccsd = res.e_mp2;
  MixedSweeps sw(c);  // mixed precision: split, record and delta sweeps (cc.h)
  const bool mixed = sw.mixed();
  bool converged = false;
  int iter = 0;
  auto t_prev = std::chrono::steady_clock::now();  // printed sweep times (the loop synchronises each sweep)
  for (iter = 1; iter <= c.opt.maxiter; iter++) {
    c.store["T"].swap(c.store["Told"]);  // amp_save, ccwfn.cc:300-309
    double* to = c.get("Told").p;
    double* tn = c.get("T").p;
    double* r = c.get("R").p;
    const MixedSweeps::Kind kind = sw.begin();
    {
      Fp64Scope scope(c, kind != MixedSweeps::kSplit);
      residual(c, to, r, &ev);
    }
    sw.end();
    double noise = -1.0, drift = -1.0;
    if (c.opt.print >= 2 && mixed) {
      // diagnostics: distance of this residual from the FP64 one at the same amplitudes,
      // and of the amplitudes from the last anchor
      if (kind == MixedSweeps::kRecord) {
        c.alloc("T_anchor", {np}, false);
        UCC_CUDA(cudaMemcpyAsync(c.get("T_anchor").p, to, sizeof(double) * np, cudaMemcpyDeviceToDevice, c.stream));
      } else {
        Temp Rx(c, {np});
        {
          Fp64Scope f(c);
          ccsd_residual(c, to, Rx->p);
        }
        axpby(c, np, -1.0, r, 1.0, Rx->p);
        noise = std::sqrt(dot(c, np, Rx->p, Rx->p));
        if (kind == MixedSweeps::kDelta) {
          axpby(c, np, 1.0, to, 0.0, Rx->p);
          axpby(c, np, -1.0, c.get("T_anchor").p, 1.0, Rx->p);
          drift = std::sqrt(dot(c, np, Rx->p, Rx->p));
        }
      }
    }
    jacobi_update(c, no, nv, d_do, d_dv, 0.0, r, r + (int64_t)no * nv, to, to + (int64_t)no * nv, tn,
                  tn + (int64_t)no * nv, sums.p, c.opt.diis ? diis.err() : nullptr, c.opt.diis ? diis.vec() : nullptr);
    if (c.opt.diis) diis.overlaps(sums.p + 1);
    UCC_CUDA(cudaStreamSynchronize(c.stream));  // the only wait of a sweep
    if (en) eccsd = en->value();
    rms = std::sqrt(sums[0]);
    tc_check(c);
    UCC_REQUIRE(std::isfinite(rms), UCC_NAN_DETECTED, "CCSD residual is not finite");
    bool restart = false;
    if (sw.after(rms, &restart)) {
      converged = true;
      break;
    }
    if (restart) diis.reset();
    if (c.opt.diis && !restart) {
      diis.accept(sums, 1);
      if (diis.size() > 2) diis.extrapolate(tn);
    }
    tau_of(tn);
    en = std::make_unique<Energy>(c, amp1(c, tn), c.get("tau"));
    if (c.opt.print) {
      en->d.fetch();
      eccsd = en->value();
      double t1n = std::sqrt(dot(c, (int64_t)no * nv, tn, tn) / (2 * no));
      static const char* tag[] = {"", " split", " record", " delta"};
      const auto t_now = std::chrono::steady_clock::now();
      const double ms = std::chrono::duration<double, std::milli>(t_now - t_prev).count();
      t_prev = t_now;
      std::printf("\t  %3d  %20.15f  %8.6f  %8.6e%s", iter, eccsd, t1n, rms, tag[kind]);
      if (mixed) std::printf("  %8.1f ms", ms);
      if (noise >= 0.0) std::printf("  |R-R64| %.3e", noise);
      if (drift >= 0.0) std::printf("  |T-T0| %.3e", drift);
      std::printf("\n");
    }
  }
  if (c.has("T_anchor")) c.drop("T_anchor");
  c.stats.mixed_iterations = sw.split;
  c.stats.anchored_iterations = sw.delta;
  const int fp64_iters = mixed ? sw.record : std::min(iter, c.opt.maxiter);
  tau_of(c.get("T").p);
  UCC_CUDA(cudaStreamSynchronize(c.stream));
  if (en) eccsd = en->value();
  for (size_t k = 0; k + 1 < ev.size(); k += 2) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ev[k], ev[k + 1]);
    c.stats.ladder_ms += ms;
    c.stats.ladder_launches += 1;
    const double o = no, v = nv;
    // the ladder and, with the (m, b) rows, Zmbij as the equations have them
    c.stats.ladder_flops += 2.0 * o * o * v * v * v * v + (c.pair_rows ? 2.0 * o * o * o * v * v * v : 0.0);
    c.stats.ladder_bytes += 8.0 * (v * v * v * v + 3.0 * o * o * v * v + (c.pair_rows ? o * v * v * v + o * o * o * v : 0.0));
    cudaEventDestroy(ev[k]);
    cudaEventDestroy(ev[k + 1]);
  }
  res.iterations = std::min(iter, c.opt.maxiter);
  res.e_ccsd = eccsd;
  res.converged = converged;
  c.stats.fp64_iterations = fp64_iters;
  c.have_ccsd = res.converged;
  c.have_tgrad = false;  // new amplitudes: earlier (T) gradient pieces no longer apply
  return res;
}

}  // namespace ucc
