// basis.cu -- contracted shells and primitive-pair tables from the
// reference's flat basis arrays (src/myQC/basis.f90:23-226 layout), plus the
// accurate Boys table used in MQ_MODE_TIGHT.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <type_traits>

#include "internal.h"

namespace mq {

static double gto_norm(int l, double a, double pi) {
  // primitive normalisation, the formula of gtoD (src/integrals/auxilary.f90:704-726)
  if (l == 0) return std::pow(2.0 * a / pi, 3.0 / 4.0);
  return std::pow(128.0 * std::pow(a, 5.0) / std::pow(pi, 3.0), 1.0 / 4.0);
}

int build_shells(mq_ctx *c, int nnuc, const int *Z, const double *xyz, const double *bas, const double *set,
                 const int *basinfo, const int *setinfo) {
  if (nnuc <= 0 || !Z || !xyz || !bas || !set || !basinfo || !setinfo) return set_err(c, MQ_EINVAL, "null system array");
  const int ops = basinfo[0], norb = basinfo[1];
  const int nset = setinfo[0], setl = setinfo[1];
  if (norb <= 0 || nset <= 0 || setl != 3 + ops) return set_err(c, MQ_EINVAL, "inconsistent basinfo/setinfo");
  c->nnuc = nnuc;
  c->Z.assign(Z, Z + nnuc);
  c->xyz.resize(3 * (size_t)nnuc);
  for (int a = 0; a < nnuc; ++a)
    for (int k = 0; k < 3; ++k) c->xyz[3 * a + k] = xyz[a + (size_t)nnuc * k];  // xyz(0:nnuc-1,0:2)
  const double pi = c->mode == MQ_MODE_REFERENCE ? PI_REF : PI_TRUE;

  // per AO: the sets that carry it and its coefficient in each
  std::vector<std::vector<std::pair<int, double>>> ao_sets(norb);
  std::vector<int> set_lmax(nset), set_ctr(nset);
  for (int s = 0; s < nset; ++s) {
    const int *si = setinfo + 1 + s * setl;  // si[1]=#AO, si[2]=lmax, si[3]=centre, si[4..]=AOs
    set_lmax[s] = si[2];
    set_ctr[s] = si[3];
    for (int k = 0; k < si[1]; ++k) {
      int o = si[4 + k];
      if (o < 0 || o >= norb) return set_err(c, MQ_EINVAL, "setinfo AO index out of range");
      ao_sets[o].push_back({s, bas[s * ops + k]});
    }
  }
  // group AOs that share atom and primitive sets into shells
  std::map<std::pair<int, std::vector<int>>, std::vector<int>> groups;
  std::vector<std::pair<int, std::vector<int>>> order;
  for (int o = 0; o < norb; ++o) {
    const int *bi = basinfo + 2 + 5 * o;  // [n, l, ori, nprim, centre]
    if (bi[1] > 1) return set_err(c, MQ_EINVAL, "only s and p functions are supported");
    std::vector<int> key;
    for (auto &pr : ao_sets[o]) key.push_back(pr.first);
    std::sort(key.begin(), key.end());
    if (key.empty() || (int)key.size() > KMAX) return set_err(c, MQ_EINVAL, "AO with 0 or too many primitives");
    auto k = std::make_pair(bi[4], key);
    if (!groups.count(k)) order.push_back(k);
    groups[k].push_back(o);
  }
  c->shells.clear();
  for (auto &k : order) {
    std::vector<int> &aos = groups[k];
    std::vector<int> s_aos, p_aos[3];
    for (int o : aos) {
      const int *bi = basinfo + 2 + 5 * o;
      if (bi[1] == 0) s_aos.push_back(o);
      else if (bi[2] >= 0 && bi[2] <= 2) p_aos[bi[2]].push_back(o);
      else return set_err(c, MQ_EINVAL, "bad p orientation");
    }
    size_t np = p_aos[0].size();
    if (p_aos[1].size() != np || p_aos[2].size() != np || np > 1)
      return set_err(c, MQ_EINVAL, "p functions must come as one x,y,z triple per primitive set group");
    size_t nsh = std::max(s_aos.size(), np);
    for (size_t t = 0; t < nsh; ++t) {
      HostShell sh{};
      sh.atom = k.first;
      sh.has_s = t < s_aos.size();
      sh.has_p = t < np;
      sh.type = sh.has_p ? 1 : 0;
      sh.nprim = (int)k.second.size();
      sh.qlmax = 0;
      int so = sh.has_s ? s_aos[t] : -1, px = sh.has_p ? p_aos[0][t] : -1;
      for (int i = 0; i < sh.nprim; ++i) {
        int s = k.second[i];
        sh.alpha[i] = set[s];
        sh.qlmax = std::max(sh.qlmax, set_lmax[s]);
        auto coef_of = [&](int o) {
          double v = 0.0;
          if (o >= 0)
            for (auto &pr : ao_sets[o])
              if (pr.first == s) v = pr.second;
          return v;
        };
        double csv = coef_of(so), cpv = coef_of(px);
        sh.cs[i] = sh.has_s ? csv * gto_norm(0, set[s], pi) : 0.0;
        sh.cp[i] = sh.has_p ? cpv * gto_norm(1, set[s], pi) : 0.0;
      }
      // AO indices: s, px, py, pz must be consecutive (the reference orders a
      // section's functions that way, basis.f90:182-192)
      if (sh.has_p && sh.has_s && (p_aos[0][t] != so + 1 || p_aos[1][t] != so + 2 || p_aos[2][t] != so + 3))
        return set_err(c, MQ_EINVAL, "sp shell AOs are not consecutive");
      if (sh.has_p && (p_aos[1][t] != px + 1 || p_aos[2][t] != px + 2))
        return set_err(c, MQ_EINVAL, "p AOs are not consecutive");
      if (!sh.has_s) return set_err(c, MQ_EINVAL, "p functions without an s function on the same primitive sets");
      sh.ao0 = so;
      c->shells.push_back(sh);
    }
  }
  c->nshell = (int)c->shells.size();
  c->nao = norb;
  return MQ_OK;
}

void free_pairs(mq_ctx *c) {
  c->pt = PairTable{};
  c->schwarz_valid = 0;
}

// Shell pairs of one molecule, in class order (ss), (sp,s), (sp,sp), with
// their surviving primitive pairs.  The host finds what survives and its order;
// everything else of a pair is formed on the device (pair_fill_kernel).
void pairs_host(const std::vector<HostShell> &shells, const std::vector<double> &xyz, HostPairs &h) {
  h = HostPairs{};
  const int ns = (int)shells.size();
  h.shells.resize(ns);
  for (int s = 0; s < ns; ++s) {
    const HostShell &sh = shells[s];
    PairShell &d = h.shells[s];
    d = PairShell{};
    for (int k = 0; k < 3; ++k) d.x[k] = xyz[3 * sh.atom + k];
    for (int i = 0; i < sh.nprim; ++i) d.alpha[i] = sh.alpha[i], d.cs[i] = sh.cs[i], d.cp[i] = sh.cp[i];
    d.ao0 = sh.ao0;
  }
  struct Cand {
    int A, B, n, first;
  };
  std::vector<Cand> pl[3];
  std::vector<double> K;
  std::vector<int> ij;
  const size_t np = (size_t)ns * (ns + 1) / 2;
  K.reserve(9 * np);
  ij.reserve(9 * np);
  for (int a = 0; a < ns; ++a)
    for (int b = 0; b <= a; ++b) {
      int iA = a, iB = b;
      if (shells[b].type > shells[a].type) std::swap(iA, iB);
      const HostShell &A = shells[iA], &B = shells[iB];
      const double *xa = &xyz[3 * A.atom], *xb = &xyz[3 * B.atom];
      double AB2 = 0;
      for (int k = 0; k < 3; ++k) AB2 += (xa[k] - xb[k]) * (xa[k] - xb[k]);
      // the surviving primitive pairs, K descending (ties keep the (i, j)
      // order): the pairs of a ket passing the screen against one bra primitive
      // are then a prefix of the ket's list, and the integral kernels visit
      // exactly the surviving primitive quartets
      double Kp[KMAX * KMAX];
      int ip[KMAX * KMAX], n = 0;
      for (int i = 0; i < A.nprim; ++i)
        for (int j = 0; j < B.nprim; ++j) {
          const double a1 = A.alpha[i], b1 = B.alpha[j];
          const double Kab = std::exp(-a1 * b1 * AB2 / (a1 + b1));
          // a primitive pair whose EIJ is below 1e-14 fails the reference's
          // screen EIJ*EGH < 1e-14 (int2e.f90:257; int1e.f90:238) for any
          // partner, since EGH <= 1
          if (!(Kab >= 1.0e-14)) continue;
          int t = n++;
          for (; t > 0 && Kp[t - 1] < Kab; --t) Kp[t] = Kp[t - 1], ip[t] = ip[t - 1];
          Kp[t] = Kab;
          ip[t] = i | j << 8;
        }
      pl[A.type + B.type].push_back({iA, iB, n, (int)K.size()});
      K.insert(K.end(), Kp, Kp + n);
      ij.insert(ij.end(), ip, ip + n);
    }
  h.shA.reserve(np);
  h.shB.reserve(np);
  h.off.reserve(np + 1);
  h.K.reserve(K.size());
  h.ij.reserve(K.size());
  for (int cl = 0; cl < 3; ++cl) {
    h.class_off[cl] = (int)h.shA.size();
    // within a class, pairs with more primitive pairs first: neighbouring quartets
    // of an integral launch (one warp) then loop over similar primitive counts
    std::stable_sort(pl[cl].begin(), pl[cl].end(), [](const Cand &x, const Cand &y) { return x.n > y.n; });
    for (const Cand &q : pl[cl]) {
      h.shA.push_back(q.A);
      h.shB.push_back(q.B);
      h.off.push_back((int)h.K.size());
      h.K.insert(h.K.end(), K.begin() + q.first, K.begin() + q.first + q.n);
      h.ij.insert(h.ij.end(), ij.begin() + q.first, ij.begin() + q.first + q.n);
    }
  }
  h.class_off[3] = (int)h.shA.size();
  h.off.push_back((int)h.K.size());
}

// The table's other fields from the shells, one warp per pair; ij: the primitives of each pair.
__global__ void pair_fill_kernel(PairTable t, const PairShell *__restrict__ shells, const int *__restrict__ shell0,
                                 const int *__restrict__ ij) {
  const int P = blockIdx.x, m = t.mol[P];
  const PairShell &A = shells[shell0[m] + t.shA[P]], &B = shells[shell0[m] + t.shB[P]];
  if (threadIdx.x == 0) {
    t.aoA[P] = A.ao0;
    t.aoB[P] = B.ao0;
    t.schwarz[P] = 1.0e300;
  }
  if (threadIdx.x < 3) {
    t.geom[6 * (size_t)P + threadIdx.x] = A.x[threadIdx.x];
    t.geom[6 * (size_t)P + 3 + threadIdx.x] = B.x[threadIdx.x] - A.x[threadIdx.x];
  }
  for (int q = t.pp_off[P] + threadIdx.x; q < t.pp_off[P + 1]; q += blockDim.x) {
    const int i = ij[q] & 255, j = ij[q] >> 8;
    const double a = A.alpha[i], b = B.alpha[j], pp = a + b, K = t.K[q];
    double X[3], PA[3], PB[3], c4[4];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      X[k] = (a * A.x[k] + b * B.x[k]) / pp;
      PA[k] = X[k] - A.x[k];
      PB[k] = X[k] - B.x[k];
    }
    const double i2p = 1.0 / (2.0 * pp);
    c4[0] = K * A.cs[i] * B.cs[j];
    c4[1] = K * A.cs[i] * B.cp[j];
    c4[2] = K * A.cp[i] * B.cs[j];
    c4[3] = K * A.cp[i] * B.cp[j];
    t.p[q] = pp;
    t.inv2p[q] = i2p;
    t.beta[q] = b;
    t.Px[q] = X[0], t.Py[q] = X[1], t.Pz[q] = X[2];
    t.PAx[q] = PA[0], t.PAy[q] = PA[1], t.PAz[q] = PA[2];
    t.PBx[q] = PB[0], t.PBy[q] = PB[1], t.PBz[q] = PB[2];
#pragma unroll
    for (int k = 0; k < 4; ++k) t.c4[4 * (size_t)q + k] = c4[k];
    float4 *f = t.pf + 4 * (size_t)q;
    f[0] = make_float4((float)pp, (float)i2p, (float)K, (float)X[0]);
    f[1] = make_float4((float)X[1], (float)X[2], (float)PA[0], (float)PA[1]);
    f[2] = make_float4((float)PA[2], (float)PB[0], (float)PB[1], (float)PB[2]);
    f[3] = make_float4((float)c4[0], (float)c4[1], (float)c4[2], (float)c4[3]);
  }
}

// ---- The exponent sums p of a table take few distinct values (shells of one
// element share their exponents), and alpha = pq/(p+q) and the prefactor
// 2 pi^5/2 / (p q sqrt(p+q)) of a primitive quartet depend on its two sums
// alone: the distinct sums are numbered with a hash table, and both quantities
// are tabulated once for all pairs of them.
constexpr int PQ_SLOTS = 4096, PQ_PROBES = 64;
struct PqHash {
  unsigned long long key[PQ_SLOTS];  // bit patterns of p (0: free; p > 0)
  int id[PQ_SLOTS];
  double p[PQ_MAX];
  int overflow;
};

__global__ void pq_insert_kernel(int npp, const double *__restrict__ p, PqHash *__restrict__ h, int *__restrict__ slot) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= npp) return;
  const unsigned long long k = (unsigned long long)__double_as_longlong(p[i]);
  unsigned s = (unsigned)((k * 0x9E3779B97F4A7C15ull) >> 52);
  int found = -1;
  for (int t = 0; t < PQ_PROBES && found < 0; ++t, s = (s + 1) % PQ_SLOTS) {
    unsigned long long o = *(volatile unsigned long long *)&h->key[s];
    if (o == 0) o = atomicCAS(&h->key[s], 0ull, k);
    if (o == 0 || o == k) found = (int)s;
  }
  if (found < 0) h->overflow = 1;
  slot[i] = found;
}

// the slots in use numbered in slot order (one CTA); more than PQ_MAX, or a sum without a slot: none
__global__ void __launch_bounds__(1024) pq_number_kernel(PqHash *__restrict__ h, int *__restrict__ pq_n) {
  __shared__ int cnt[1024];
  constexpr int PER = PQ_SLOTS / 1024;
  int c = 0;
  for (int k = 0; k < PER; ++k) c += h->key[threadIdx.x * PER + k] != 0;
  cnt[threadIdx.x] = c;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    const int v = threadIdx.x >= o ? cnt[threadIdx.x - o] : 0;
    __syncthreads();
    cnt[threadIdx.x] += v;
    __syncthreads();
  }
  int id = cnt[threadIdx.x] - c;
  for (int k = 0; k < PER; ++k) {
    const int s = threadIdx.x * PER + k;
    if (h->key[s] == 0) continue;
    h->id[s] = id;
    if (id < PQ_MAX) h->p[id] = __longlong_as_double((long long)h->key[s]);
    ++id;
  }
  if (threadIdx.x == 1023) *pq_n = h->overflow || cnt[1023] > PQ_MAX ? 0 : cnt[1023];
}

__global__ void pq_table_kernel(const PqHash *__restrict__ h, const int *__restrict__ pq_n, double pref0,
                                double2 *__restrict__ pq) {
  const int n = *pq_n;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n * n; i += gridDim.x * blockDim.x) {
    const double p = h->p[i / n], q = h->p[i % n], s = p + q;
    pq[i] = make_double2(p * q / s, pref0 / (p * q * sqrt(s)));
  }
}

// the record of each primitive pair (layout in eri_low.cuh)
__global__ void pp_record_kernel(PairTable t, const PqHash *__restrict__ h, const int *__restrict__ slot) {
  const int P = blockIdx.x;
  for (int i = t.pp_off[P] + threadIdx.x; i < t.pp_off[P + 1]; i += blockDim.x) {
    const double *c = t.c4 + 4 * (size_t)i;
    const double be = t.beta[i] / t.p[i], H = -1.0 / t.p[i];
    double *r = t.rec + (size_t)PP_REC * i;
    r[0] = t.Px[i];
    r[1] = t.Py[i];
    r[2] = t.Pz[i];
    r[3] = be;
    r[4] = t.K[i];
    r[5] = 1.0e-14 / t.K[i];
    r[6] = c[0];
    r[7] = c[2] * be;
    r[8] = c[2] * H;
    r[9] = c[1] * (be - 1.0);
    r[10] = c[1] * H;
    r[11] = c[3] * be * (be - 1.0);
    r[12] = c[3] * H;
    r[13] = H;
    t.pid[i] = *t.pq_n > 0 ? h->id[slot[i]] : 0;
  }
}

static int pair_records(mq_ctx *c, PairTable &t, int mode) {
  if (t.npp == 0) return MQ_OK;
  char *w = (char *)buf(c, "pair_hash", sizeof(PqHash) + sizeof(int) * (size_t)t.npp);
  if (!w) return MQ_ENOMEM;
  PqHash *h = (PqHash *)w;
  int *slot = (int *)(w + sizeof(PqHash));
  const double pref0 = mode == MQ_MODE_REFERENCE ? 2.0 * 17.493419544621675 : 2.0 * 17.493418327624862;  // 2 pi^2.5
  MQ_CUDA(c, cudaMemsetAsync(h, 0, sizeof(PqHash), c->stream));
  pq_insert_kernel<<<(t.npp + 255) / 256, 256, 0, c->stream>>>(t.npp, t.p, h, slot);
  pq_number_kernel<<<1, 1024, 0, c->stream>>>(h, t.pq_n);
  pq_table_kernel<<<64, 256, 0, c->stream>>>(h, t.pq_n, pref0, t.pq);
  pp_record_kernel<<<t.npairs, 32, 0, c->stream>>>(t, h, slot);
  c->stats.launches += 4;
  MQ_CUDA(c, cudaGetLastError());
  return MQ_OK;
}

// The table of M molecules, class first, then molecule, in one device block
// (256-byte aligned pieces; the context's buffer `name`, once the work queued on the
// stream, which may read the previous table, has finished).  Only what pairs_host
// found is staged, through one pinned host buffer and one copy.
int upload_pairs(mq_ctx *c, const HostPairs *const *mols, int M, const char *name, PairTable &t, int mode) {
  t = PairTable{};
  size_t npairs = 0, npp = 0, nsh = 0;
  for (int m = 0; m < M; ++m) npairs += mols[m]->shA.size(), npp += mols[m]->K.size(), nsh += mols[m]->shells.size();
  if (npairs > 2147483646ull || npp > 2147483646ull) return set_err(c, MQ_EINVAL, "pair table too large");
  t.npairs = (int)npairs;
  t.npp = (int)npp;
  size_t total = 0;
  std::vector<std::pair<void **, size_t>> items;
  auto room = [&](auto *&dst, size_t count) {
    items.push_back({(void **)&dst, total});
    total += (std::max<size_t>(count, 1) * sizeof(*dst) + 255) / 256 * 256;
  };
  PairShell *shells = nullptr;
  int *shell0 = nullptr, *ij = nullptr;
  room(shells, nsh);
  room(shell0, M);
  room(t.shA, npairs);
  room(t.shB, npairs);
  room(t.pp_off, npairs + 1);
  room(t.mol, npairs);
  room(t.K, npp);
  room(ij, npp);
  const size_t copied = total;  // behind it: what the device forms itself
  room(t.aoA, npairs);
  room(t.aoB, npairs);
  room(t.schwarz, npairs);
  room(t.geom, 6 * npairs);
  for (double **v : {&t.p, &t.inv2p, &t.beta, &t.Px, &t.Py, &t.Pz, &t.PAx, &t.PAy, &t.PAz, &t.PBx, &t.PBy, &t.PBz})
    room(*v, npp);
  room(t.c4, 4 * npp);
  room(t.pf, 4 * npp);
  room(t.rec, PP_REC * npp);
  room(t.pid, npp);
  room(t.pq, (size_t)PQ_MAX * PQ_MAX);
  room(t.pq_n, 1);
  MQ_CUDA(c, cudaStreamSynchronize(c->stream));
  char *dev = (char *)buf(c, name, total);
  if (!dev) return MQ_ENOMEM;
  if (c->pin_bytes < copied) {
    if (c->pin) cudaFreeHost(c->pin);
    c->pin = nullptr;
    c->pin_bytes = 0;
    MQ_CUDA(c, cudaHostAlloc(&c->pin, copied, cudaHostAllocDefault));
    c->pin_bytes = copied;
  }
  for (auto &it : items) *it.first = (char *)c->pin + it.second;  // (the staged pieces first, as host pointers)
  size_t P = 0, q = 0, s = 0;
  for (int m = 0; m < M; ++m) {
    shell0[m] = (int)s;
    std::copy(mols[m]->shells.begin(), mols[m]->shells.end(), shells + s);
    s += mols[m]->shells.size();
  }
  for (int cl = 0; cl < 3; ++cl) {
    t.class_off[cl] = (int)P;
    for (int m = 0; m < M; ++m) {
      const HostPairs &h = *mols[m];
      const int P0 = h.class_off[cl], P1 = h.class_off[cl + 1], q0 = h.off[P0], q1 = h.off[P1];
      std::copy(h.shA.begin() + P0, h.shA.begin() + P1, t.shA + P);
      std::copy(h.shB.begin() + P0, h.shB.begin() + P1, t.shB + P);
      std::fill(t.mol + P, t.mol + P + (P1 - P0), m);
      for (int k = P0; k < P1; ++k) t.pp_off[P + (k - P0)] = (int)q + h.off[k] - q0;
      std::copy(h.K.begin() + q0, h.K.begin() + q1, t.K + q);
      std::copy(h.ij.begin() + q0, h.ij.begin() + q1, ij + q);
      P += P1 - P0;
      q += q1 - q0;
    }
  }
  t.class_off[3] = (int)P;
  t.pp_off[P] = (int)q;
  for (auto &it : items) *it.first = dev + it.second;
  MQ_CUDA(c, cudaMemcpyAsync(dev, c->pin, copied, cudaMemcpyHostToDevice, c->stream));
  if (npairs > 0) {
    pair_fill_kernel<<<(unsigned)npairs, 32, 0, c->stream>>>(t, shells, shell0, ij);
    c->stats.launches += 1;
    MQ_CUDA(c, cudaGetLastError());
  }
  MQ_CUDA(c, cudaStreamSynchronize(c->stream));  // the staging buffer is reused by the next upload
  return pair_records(c, t, mode);
}

int build_pairs(mq_ctx *c) {
  free_pairs(c);
  HostPairs h;
  pairs_host(c->shells, c->xyz, h);
  const HostPairs *hp = &h;
  MQ_TRY(upload_pairs(c, &hp, 1, "pair_table", c->pt, c->mode));
  c->pair_class_count = {h.class_off[1] - h.class_off[0], h.class_off[2] - h.class_off[1],
                         h.class_off[3] - h.class_off[2]};
  c->hp_shA = h.shA;
  c->hp_shB = h.shB;
  c->hp_aoA.resize(h.shA.size());
  c->hp_aoB.resize(h.shA.size());
  for (size_t P = 0; P < h.shA.size(); ++P) {
    c->hp_aoA[P] = c->shells[h.shA[P]].ao0;
    c->hp_aoB[P] = c->shells[h.shB[P]].ao0;
  }
  for (int k = 0; k < 4; ++k) c->hp_class_off[k] = h.class_off[k];
  c->qs.valid = 0;
  c->qs.tables_valid = 0;
  return MQ_OK;
}

// F_m(T) for T = 0.0, 0.1, ..., 36.0 and m = 0..12 by the power series
//   F_m(T) = e^-T sum_k (2T)^k / ((2m+1)(2m+3)...(2m+2k+1))
// at m = 12 in long double, then downward recursion F_m = (2T F_{m+1} + e^-T)/(2m+1).
// The table is a constant: computed once per process (the long-double series
// is slow where long double is a software type, as on aarch64).
static void tight_boys_compute(std::vector<double> &tab);
static void fine_boys_compute(std::vector<double> &tab);
void tight_boys_table(std::vector<double> &tab) {
  static std::once_flag once;
  static std::vector<double> cached;
  std::call_once(once, [] { tight_boys_compute(cached); });
  tab = cached;
}

// The tight table as the kernels read it: F_m(Tk) [TIGHT_NT][TIGHT_NM], the grid
// values Tk, then for m = 0..BOYS_SCALED_M-1 the Taylor coefficients of F_m
// about Tk, F_{m+k}(Tk) / k! for k = 0..8 ([m][TIGHT_NT][9]).
void tight_boys_device_table(std::vector<double> &tab) {
  std::vector<double> f;
  tight_boys_table(f);
  tab = f;
  for (int k = 0; k < TIGHT_NT; ++k) tab.push_back(k / 10.0);
  for (int m = 0; m < BOYS_SCALED_M; ++m)
    for (int t = 0; t < TIGHT_NT; ++t) {
      double fact = 1.0;
      for (int k = 0; k < 9; ++k) {
        if (k > 0) fact *= k;
        tab.push_back(f[(size_t)t * TIGHT_NM + m + k] / fact);
      }
    }
  static std::once_flag once;
  static std::vector<double> fine;
  std::call_once(once, [] { fine_boys_compute(fine); });
  while (tab.size() < BOYS_FINE_OFF) tab.push_back(0.0);
  tab.insert(tab.end(), fine.begin(), fine.end());
}

// Values F_0 .. F_{nm-1} at T, the series at the top order and downward recursion.
static void boys_series(long double T, int nm, long double *F) {
  const int m = nm - 1;
  long double term = 1.0L / (2 * m + 1), sum = term;
  for (int k = 1; k < 2000; ++k) {
    term *= 2.0L * T / (2 * m + 2 * k + 1);
    sum += term;
    if (term < 1e-22L * sum) break;
  }
  const long double e = expl(-T);
  F[m] = e * sum;
  for (int j = m - 1; j >= 0; --j) F[j] = (2.0L * T * F[j + 1] + e) / (2.0L * j + 1.0L);
}

// [m < 4][577 rows, T step 1/16][8]: F_m(T) as a polynomial of degree 6 in
// d = Tk - T, |d| <= 1/32, and Tk.  The Taylor polynomial of degree 8 with its
// two highest terms economised over the interval: x^8 and x^7 (x = 32 d)
// replaced through the Chebyshev polynomials T8 = 128 x^8 - 256 x^6 + 160 x^4
// - 32 x^2 + 1 and T7 = 64 x^7 - 112 x^5 + 56 x^3 - 7 x, which leaves at most
// F_{m+7} / (7! 64 32^7) = 9e-17 F_{m+7}.
static void fine_boys_compute(std::vector<double> &tab) {
  constexpr int NM = BOYS_FINE_M + 8;
  tab.assign((size_t)BOYS_FINE_M * BOYS_FINE_NT * 8, 0.0);
  for (int t = 0; t < BOYS_FINE_NT; ++t) {
    long double F[NM];
    boys_series(t / 16.0L, NM, F);
    for (int m = 0; m < BOYS_FINE_M; ++m) {
      long double a[9], fact = 1.0L, h = 1.0L;  // coefficients of x^k
      for (int k = 0; k < 9; ++k) {
        if (k) fact *= k, h /= 32.0L;
        a[k] = F[m + k] / fact * h;
      }
      a[6] += 2.0L * a[8], a[4] -= 1.25L * a[8], a[2] += 0.25L * a[8], a[0] -= a[8] / 128.0L;
      a[5] += 1.75L * a[7], a[3] -= 0.875L * a[7], a[1] += 7.0L / 64.0L * a[7];
      double *row = tab.data() + ((size_t)m * BOYS_FINE_NT + t) * 8;
      long double s = 1.0L;
      for (int k = 0; k < 7; ++k, s *= 32.0L) row[k] = (double)(a[k] * s);
      row[7] = t / 16.0;
    }
  }
}

static void tight_boys_compute(std::vector<double> &tab) {
  tab.assign((size_t)TIGHT_NT * TIGHT_NM, 0.0);
  for (int it = 0; it < TIGHT_NT; ++it) {
    long double F[TIGHT_NM];
    boys_series(it / 10.0L, TIGHT_NM, F);
    for (int j = 0; j < TIGHT_NM; ++j) tab[(size_t)it * TIGHT_NM + j] = (double)F[j];
  }
}

}  // namespace mq
