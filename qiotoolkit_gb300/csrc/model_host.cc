// model_host.cc -- model construction and upload, schedules, device setup.
#include <algorithm>
#include <array>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <map>
#include <mutex>
#include <set>
#include <unordered_map>

#include "host.h"

namespace qio
{
void fail(int status, const std::string& msg) { throw Error(status, msg); }

void cuda_check(cudaError_t e, const char* what)
{
  if (e == cudaSuccess) return;
  if (e == cudaErrorMemoryAllocation)
    fail(2, std::string(what) + ": out of device memory");
  if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver)
    fail(5, std::string(what) + ": " + cudaGetErrorString(e));
  fail(3, std::string(what) + ": " + cudaGetErrorString(e));
}

// Device bytes held in buffers.  QIO_DEVICE_MEMORY_LIMIT (bytes, read at
// each allocation) caps them, for callers that share a GPU: an allocation
// past the cap fails as out of device memory (status 2), as it would on a
// full device.
static std::atomic<long long> g_held{0};

static long long device_memory_limit()
{
  const char* e = std::getenv("QIO_DEVICE_MEMORY_LIMIT");
  return e ? std::atoll(e) : 0;
}

DevBuf::DevBuf(size_t n) : bytes(n)
{
  if (!n) return;
  const long long cap = device_memory_limit();
  if (cap > 0 && g_held.load() + (long long)n > cap)
    fail(2, "cudaMalloc: out of device memory (over QIO_DEVICE_MEMORY_LIMIT)");
  cuda_check(cudaMalloc(&ptr, n), "cudaMalloc");
  g_held += (long long)n;
}
DevBuf::~DevBuf()
{
  if (ptr)
  {
    cudaFree(ptr);
    g_held -= (long long)bytes;
  }
}
DevBuf& DevBuf::operator=(DevBuf&& o) noexcept
{
  if (this != &o)
  {
    if (ptr)
    {
      cudaFree(ptr);
      g_held -= (long long)bytes;
    }
    ptr = o.ptr;
    bytes = o.bytes;
    o.ptr = nullptr;
    o.bytes = 0;
  }
  return *this;
}

void h2d(void* dst, const void* src, size_t bytes, const char* what)
{
  if (!bytes) return;
  cuda_check(cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice), what);
  cuda_check(cudaStreamSynchronize(cudaStreamLegacy), what);
}

cudaError_t allow_shared(const void* kernel, int bytes)
{
  if (bytes <= 32 * 1024) return cudaSuccess;  // (with the kernels' static bytes below the default limit)
  static std::mutex mu;
  static std::set<std::pair<int, const void*>> raised;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> g(mu);
  if (raised.count({dev, kernel})) return cudaSuccess;
  cudaFuncAttributes at;
  if ((e = cudaFuncGetAttributes(&at, kernel)) != cudaSuccess) return e;
  int most = 0;
  if ((e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)at.sharedSizeBytes);
  if (e == cudaSuccess) raised.insert({dev, kernel});
  return e;
}

static std::mutex g_dev_mu;
static std::map<int, int*> g_err;

int* device_error_flag()
{
  int dev = 0;
  cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
  std::lock_guard<std::mutex> g(g_dev_mu);
  auto it = g_err.find(dev);
  return it == g_err.end() ? nullptr : it->second;
}

void check_device_error(cudaStream_t s)
{
  int* e = device_error_flag();
  if (!e) return;
  int h = 0;
  cuda_check(cudaMemcpyAsync(&h, e, 4, cudaMemcpyDeviceToHost, s), "D2H error flag");
  cuda_check(cudaStreamSynchronize(s), "sync");
  if (h)
  {
    cuda_check(cudaMemsetAsync(e, 0, 4, s), "memset");
    fail(4, "a device-side wait for a bulk copy gave up (bounded wait); results are invalid");
  }
}

void ensure_device()
{
  static std::mutex& mu = g_dev_mu;
  static std::set<int> ready;
  int count = 0;
  cudaError_t e = cudaGetDeviceCount(&count);
  if (e != cudaSuccess || count == 0)
    fail(5, "no CUDA device available: the GB300 library has no CPU fallback");
  int dev = 0;
  cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
  std::lock_guard<std::mutex> g(mu);
  if (ready.count(dev)) return;
  upload_tables(dev);
  cuda_check(cudaGetLastError(), "upload_tables");
  int* flag = nullptr;
  cuda_check(cudaMalloc(&flag, 4), "cudaMalloc");
  cuda_check(cudaMemset(flag, 0, 4), "cudaMemset");
  // the tables and the flag are there before any stream's kernel reads them
  cuda_check(cudaStreamSynchronize(cudaStreamLegacy), "sync");
  g_err[dev] = flag;
  ready.insert(dev);
}

// ---------------------------------------------------------------------------
// Graph models: normalize_edges (graph/graph.h:74-177).  Names are numbered
// in order of first appearance; a repeated name in a term throws for Ising
// ("Duplicated ids detected in term!") and is merged for PUBO
// (model/pubo.h:82); members are sorted; terms without members add to the
// constant cost; each variable lists its terms in ascending term id.
// ---------------------------------------------------------------------------
static void build_graph(HostModel& m, int64_t n_terms, const int64_t* off,
                        const int32_t* ids, const double* coef)
{
  if (n_terms <= 0)
    fail(1, "parameter `terms`: size must be greater than 0, found 0");
  const bool merge = (m.kind == K_PUBO || m.kind == K_PUBO_PLAIN);
  std::unordered_map<int32_t, int> name_to_id;
  std::vector<std::vector<int>> members;
  std::vector<std::vector<int>> node_edges;
  m.min_loc = INT32_MAX;
  m.min_coupling = std::numeric_limits<double>::max();
  for (int64_t t = 0; t < n_terms; t++)
  {
    if (off[t + 1] < off[t]) fail(1, "term offsets must be non-decreasing");
    std::vector<int> mem;
    for (int64_t k = off[t]; k < off[t + 1]; k++)
    {
      auto it = name_to_id.find(ids[k]);
      int id;
      if (it == name_to_id.end())
      {
        id = (int)m.names.size();
        name_to_id.emplace(ids[k], id);
        m.names.push_back(ids[k]);
        node_edges.emplace_back();
      }
      else
        id = it->second;
      if (std::find(mem.begin(), mem.end(), id) == mem.end())
      {
        mem.push_back(id);
        node_edges[id].push_back((int)members.size());
      }
      else if (!merge)
        fail(1, "Duplicated ids detected in term!");
    }
    std::sort(mem.begin(), mem.end());
    int loc = (int)mem.size();
    m.max_loc = std::max(m.max_loc, loc);
    m.min_loc = std::min(m.min_loc, loc);
    m.total_loc += loc;
    if (!mem.empty())
    {
      m.accum_dep += (int64_t)loc * (loc - 1);
      m.min_coupling = std::min(m.min_coupling, std::fabs(coef[t]));
      m.max_coupling = std::max(m.max_coupling, std::fabs(coef[t]));
      members.push_back(std::move(mem));
      m.tcost.push_back(coef[t]);
    }
    else
      m.const_cost += coef[t];
  }
  if (m.min_loc == INT32_MAX) m.min_loc = 0;
  m.N = (int64_t)m.names.size();
  m.M = (int64_t)members.size();
  if (m.N > INT32_MAX / 2 || m.M > INT32_MAX / 2) fail(1, "model too large");
  m.row.assign(m.N + 1, 0);
  for (int64_t v = 0; v < m.N; v++) m.row[v + 1] = m.row[v] + (int)node_edges[v].size();
  m.K = m.row[m.N];
  m.inc.resize(m.K);
  m.coef.resize(m.K);
  for (int64_t v = 0; v < m.N; v++)
    for (size_t j = 0; j < node_edges[v].size(); j++)
    {
      int t = node_edges[v][j];
      m.inc[m.row[v] + j] = (uint32_t)t;
      m.coef[m.row[v] + j] = m.tcost[t];
    }
  m.trow.assign(m.M + 1, 0);
  for (int64_t t = 0; t < m.M; t++) m.trow[t + 1] = m.trow[t] + (int)members[t].size();
  m.tvar.resize(m.trow[m.M]);
  for (int64_t t = 0; t < m.M; t++)
    for (size_t j = 0; j < members[t].size(); j++)
      m.tvar[m.trow[t] + j] = (uint32_t)members[t][j];
}

// ---------------------------------------------------------------------------
// MaxSat::configure(clauses) (model/max_sat.h:295-397): clauses containing a
// variable and its negation are always true and dropped; variables used
// only there are free (rendered as 1); the remaining variables are numbered
// by ascending name; clause c (1-based in the reference, c-1 here) lists
// each variable once, negated literals marked.
// ---------------------------------------------------------------------------
static void build_maxsat(HostModel& m, int64_t n_terms, const int64_t* off,
                         const int32_t* ids, const double* coef)
{
  if (n_terms <= 0) fail(1, "parameter `terms` must not be empty");
  std::vector<char> always(n_terms, 0);
  std::set<int32_t> used, maybe_free;
  for (int64_t c = 0; c < n_terms; c++)
  {
    std::set<int32_t> seen;
    for (int64_t k = off[c]; k < off[c + 1]; k++)
    {
      int32_t v = ids[k];
      if (v == 0 || v == INT32_MIN)
        fail(1, "MaxSat variables cannot have the name " + std::to_string(v) +
                    " since it cannot be negated to indicate 'not " +
                    std::to_string(v) + "'.");
      if (seen.count(-v)) always[c] = 1;
      seen.insert(v);
    }
    for (int32_t v : seen) (always[c] ? maybe_free : used).insert(std::abs(v));
  }
  for (int32_t v : maybe_free)
    if (!used.count(v)) m.free_vars.push_back(v);
  m.names.assign(used.begin(), used.end());
  m.N = (int64_t)m.names.size();
  std::map<int32_t, int> name_to_id;
  for (size_t i = 0; i < m.names.size(); i++) name_to_id[m.names[i]] = (int)i;
  std::vector<std::vector<uint32_t>> affected(m.N);
  std::vector<std::vector<uint32_t>> members;
  m.min_loc = INT32_MAX;
  for (int64_t c = 0; c < n_terms; c++)
  {
    if (always[c]) continue;
    int t = (int)members.size();
    m.tcost.push_back(coef[c]);
    m.max_coupling = std::max(m.max_coupling, std::fabs(coef[c]));
    std::vector<uint32_t> mem;
    std::set<int> seen;
    for (int64_t k = off[c]; k < off[c + 1]; k++)
    {
      int32_t name = ids[k];
      int id = name_to_id[std::abs(name)];
      if (seen.count(id)) continue;
      seen.insert(id);
      uint32_t neg = name < 0 ? kNegBit : 0u;
      affected[id].push_back((uint32_t)t | neg);
      mem.push_back((uint32_t)id | neg);
    }
    m.max_loc = std::max(m.max_loc, (int)mem.size());
    m.min_loc = std::min(m.min_loc, (int)mem.size());
    members.push_back(std::move(mem));
  }
  if (m.min_loc == INT32_MAX) m.min_loc = 0;
  m.M = (int64_t)members.size();
  if (m.M == 0)
  {
    // the model is "empty": every clause is always true
    m.N = 0;
    m.names.clear();
  }
  m.row.assign(m.N + 1, 0);
  for (int64_t v = 0; v < m.N; v++) m.row[v + 1] = m.row[v] + (int)affected[v].size();
  m.K = m.row[m.N];
  m.inc.resize(m.K);
  m.coef.resize(m.K);
  for (int64_t v = 0; v < m.N; v++)
    for (size_t j = 0; j < affected[v].size(); j++)
    {
      uint32_t e = affected[v][j];
      m.inc[m.row[v] + j] = e;
      m.coef[m.row[v] + j] = m.tcost[e & ~kNegBit];
    }
  m.trow.assign(m.M + 1, 0);
  for (int64_t t = 0; t < m.M; t++) m.trow[t + 1] = m.trow[t] + (int)members[t].size();
  m.tvar.resize(m.trow[m.M]);
  for (int64_t t = 0; t < m.M; t++)
    for (size_t j = 0; j < members[t].size(); j++) m.tvar[m.trow[t] + j] = members[t][j];
}

// Window-conflict masks: bit d-1 of nbr[v] is set when variable v-d (d in
// 1..32) shares a term with v.
static void build_nbr(HostModel& m)
{
  m.nbr.assign(m.N, 0u);
  std::vector<int> mem;
  for (int64_t t = 0; t < m.M; t++)
  {
    mem.clear();
    for (int k = m.trow[t]; k < m.trow[t + 1]; k++) mem.push_back((int)(m.tvar[k] & ~kNegBit));
    std::sort(mem.begin(), mem.end());
    for (size_t j = 0; j < mem.size(); j++)
      for (size_t i = j; i-- > 0;)
      {
        int d = mem[j] - mem[i];
        if (d > 32) break;
        if (d >= 1) m.nbr[mem[j]] |= 1u << (d - 1);
      }
  }
}

// Later co-members for the per-block field updates: for incidence k of v
// (term t), each member u of t with 0 < u - v <= 31 and a row of at most 32
// incidences, encoded as (u - v, position of t in u's row).  When u flips
// nothing is posted (it has been decided already); when v flips, these are
// the undecided variables of the same 32-variable block whose cost
// difference changes.
static void build_levels(HostModel& m);

static void build_near(HostModel& m)
{
  m.near.assign(m.K, 0ULL);
  for (int64_t v = 0; v < m.N; v++)
    for (int q = m.row[v]; q < m.row[v + 1]; q++)
    {
      uint32_t t = m.inc[q] & ~kNegBit;
      unsigned long long w = 0;
      int cnt = 0;
      bool over = false;
      for (int j = m.trow[t]; j < m.trow[t + 1]; j++)
      {
        int64_t u = (int64_t)(m.tvar[j] & ~kNegBit);
        int64_t d = u - v;
        if (d < 1 || d > 31) continue;
        if (m.row[u + 1] - m.row[u] > 32) continue;
        int kp = -1;
        for (int x = m.row[u]; x < m.row[u + 1]; x++)
          if ((m.inc[x] & ~kNegBit) == t) { kp = x - m.row[u]; break; }
        if (kp < 0) continue;
        if (cnt == 6) { over = true; break; }
        w |= ((unsigned long long)d | ((unsigned long long)kp << 5)) << (10 * cnt);
        cnt++;
      }
      m.near[q] = over ? (7ULL << 61) : (w | ((unsigned long long)cnt << 61));
    }
}

// Tables of the block-decided sweep (fields.cu).  A variable's field H_v is its
// flip's cost difference, up to its own spin's sign, in fixed point q =
// round(c * 2^S):
//   Ising: H_v = sum over v's terms of q, negated where the product of the other
//     members' spins is; the cost difference of flipping v is -2 (1 - 2 s_v) H_v;
//   counter models: H_v = sum over the terms none of whose other literals is
//     true of +q (v's literal plain) or -q (negated); the cost difference is
//     H_v when s_v is true and -H_v otherwise.
// S is the largest scale with 2^S * max_v sum_row |c| <= 2^30 (2^22 when a
// weight also carries its term's row position in its low 8 bits), so
// a field never overflows and differs from the reference's FP64 sum by less
// than deg + 1 units.  Integer models use S = 0: the field is then exact.
//
// A term is kept as its other members' literals: literal 2u + 1 is u negated, 2N
// none (false).  Terms of more than four members are wide: the sweep keeps a
// byte for each (true literals, or the parity).
// Eligible: Ising with the term cache or counter models, fewer than 32766
// variables and 2^18 terms, rows of at most 255 incidences.
static void build_fields(HostModel& m)
{
  m.fc_desc.clear();
  m.fc_tab.clear();
  m.fc_oth.clear();
  m.fc_wide.clear();
  m.fc_words = 0;
  if (!(m.flavor == F_PARITY || m.flavor == F_COUNTER) || m.N == 0 || m.N >= 32766) return;
  if (!m.pair_only && m.M >= (1 << 18)) return;  // (a term's byte would not fit shared memory)
  double amax = 0;
  for (int64_t v = 0; v < m.N; v++)
  {
    if (m.row[v + 1] - m.row[v] > 255) return;
    double s = 0;
    for (int q = m.row[v]; q < m.row[v + 1]; q++) s += std::fabs(m.coef[q]);
    amax = std::max(amax, s);
  }
  m.fc_pack = !m.int_mode && !m.pair_only;
  if (m.int_mode) m.fc_S = 0;
  else
  {
    const int top = m.fc_pack ? 22 : 30;
    int e = 0;
    if (amax > 0) std::frexp(amax, &e);  // amax < 2^e
    m.fc_S = amax > 0 ? top - e : 0;
    if (m.fc_S < -900 || m.fc_S > 900) return;  // 2^-S must stay a normal double
  }
  // (sums of these wrap as the device's do; what they end in does not)
  auto fixed = [&](int q) -> uint32_t {
    long long f = m.int_mode ? (long long)m.coef_i[q] : std::llrint(std::ldexp(m.coef[q], m.fc_S));
    return (uint32_t)(int)(m.fc_pack ? f * 256 : f);
  };
  const bool pair = m.pair_only, ising = m.flavor == F_PARITY;
  const int nb = (int)((m.N + 31) / 32);
  const int KI = 4;  // fields.cu: entries per lane of a block's chunk
  const int ew = pair ? 2 : 4;                          // 32-bit words of an entry
  const size_t ent_at = 8 + (pair ? 64 : 128);          // 32-bit words before a chunk's entries
  const size_t rec_at = ent_at + (size_t)KI * 32 * ew;  // ... and its records
  const uint32_t none = (uint32_t)(2 * m.N);
  std::vector<int> wide_of;  // term -> wide term, or -1
  if (!pair)
  {
    wide_of.assign((size_t)m.M, -1);
    for (int64_t t = 0; t < m.M; t++)
      if (m.trow[t + 1] - m.trow[t] > 4)
      {
        wide_of[t] = (int)m.fc_wide.size();
        m.fc_wide.push_back((int)t);
      }
    m.fc_oth.assign((size_t)m.K * 2, 0);
  }
  m.fc_desc.assign((size_t)nb * 4, 0);
  struct Rec { uint32_t lit[3]; uint32_t val; };
  struct Entry { uint32_t w[4]; };
  std::vector<Rec> rec[32][3];  // by number of others
  std::vector<Entry> in[32], wide[32];
  m.fc_tab.reserve((size_t)m.K * 3 + (size_t)nb * rec_at);
  for (int b = 0; b < nb; b++)
  {
    const int v0 = b * 32, v1 = (int)std::min<int64_t>(m.N, v0 + 32);
    for (int l = 0; l < 32; l++)
    {
      for (auto& r : rec[l]) r.clear();
      in[l].clear();
      wide[l].clear();
    }
    uint32_t base[32] = {}, degree[32] = {}, negs[32] = {}, alone[32] = {};
    int rows[4] = {}, kin = 0;
    for (int l = 0; l < 32; l++)
    {
      const int v = v0 + l;
      const int deg = v < v1 ? m.row[v + 1] - m.row[v] : 0;
      degree[l] = (uint32_t)deg;
      for (int k = 0; k < deg; k++)
      {
        const int q = m.row[v] + k;
        const uint32_t f = fixed(q);
        if (pair)
        {
          const int u = m.other[q];
          base[l] += f;
          if (u < 0) continue;
          rec[l][0].push_back({{(uint32_t)u, 0, 0}, 2u * f});
          if (u >= v0 && u < v) in[l].push_back({{1u << (u - v0), 2u * f, 0, 0}});
          continue;
        }
        const uint32_t t = m.inc[q] & ~kNegBit, vneg = m.inc[q] >> 31;
        const uint32_t val = ising ? f : (vneg ? 0u - f : f);
        const uint32_t at = m.fc_pack ? (uint32_t)(k & 31) : 0u;  // the row position beside a weight
        if (k < 32) negs[l] |= vneg << k;
        // the other members: before this one in the block, and the rest
        uint32_t mates = 0, neg = 0, lit[3] = {none, none, none};
        int n = 0;
        uint32_t rest[2] = {none, none};
        int nrest = 0;
        for (int j = m.trow[t]; j < m.trow[t + 1]; j++)
        {
          const uint32_t u = m.tvar[j] & ~kNegBit, un = ising ? 0u : m.tvar[j] >> 31;
          if ((int)u == v) continue;
          if (wide_of[t] < 0) lit[n++] = 2 * u + un;
          if ((int)u >= v0 && (int)u < v)
          {
            mates |= 1u << (u - v0);
            neg |= un << (u - v0);
          }
          else if (nrest < 2) rest[nrest++] = 2 * u + un;  // (more only without mates, or wide)
        }
        uint32_t* o = &m.fc_oth[(size_t)q * 2];
        for (int i = 0; i < 3; i++) lit[i] = i < n ? lit[i] : none;
        o[0] = (n > 0 ? lit[0] : 0xFFFFu) | (n > 1 ? lit[1] : 0xFFFFu) << 16;
        o[1] = (n > 2 ? lit[2] : 0xFFFFu) | vneg << 16 | (wide_of[t] >= 0 ? 1u << 17 : 0u);
        if (wide_of[t] >= 0)
        {
          const uint32_t w = (uint32_t)wide_of[t];
          wide[l].push_back({{w | vneg << 31, (mates ? 0u : ising ? 2u * f : val) | at, mates ? 1u : 0u, 0}});
          if (mates) in[l].push_back({{mates, neg | vneg << l, 0xFFFC0000u | w, val | at}});
        }
        else if (mates)
        {
          in[l].push_back({{mates, neg, rest[0] | rest[1] << 16, val | at}});
        }
        else if (n > 0) rec[l][n - 1].push_back({{lit[0], lit[1], lit[2]}, (ising ? 2u * f : val) | at});
        else if (!ising) alone[l] |= 1u << (k & 31);
        if (!mates) base[l] += val;
      }
      kin = std::max(kin, (int)in[l].size());
      rows[3] = std::max(rows[3], (int)wide[l].size());
    }
    // Rows of records of one, two and three literals (a shorter one may fill a
    // longer one's row)
    for (int l = 0; l < 32; l++) rows[2] = std::max(rows[2], (int)rec[l][2].size());
    rows[2] = (rows[2] + 1) & ~1;
    auto left = [&](int l, int c) {  // records that the longer rows leave
      int n = 0;
      for (int i = 2; i >= c; i--) n += (int)rec[l][i].size() - (i > c ? rows[i] : 0);
      return n;
    };
    for (int l = 0; l < 32; l++) rows[1] = std::max(rows[1], left(l, 1));
    rows[1] = (rows[1] + 1) & ~1;
    for (int l = 0; l < 32; l++) rows[0] = std::max(rows[0], left(l, 0));
    rows[0] = (rows[0] + 3) & ~3;
    const bool matrix = pair && kin > KI;
    const size_t words = rec_at / 2 + 32 * (size_t)(rows[0] + rows[1] + rows[2] + rows[3]) + 16 * (size_t)rows[2] +
                         (matrix ? 512 : 64 * (size_t)std::max(0, kin - KI));
    const size_t at = m.fc_tab.size();
    m.fc_tab.resize(at + ((2 * words + 3) & ~(size_t)3), 0u);
    uint32_t* tab = &m.fc_tab[at];
    m.fc_desc[(size_t)b * 4] = (int)(at / 2);
    m.fc_desc[(size_t)b * 4 + 1] = (int)((words + 1) & ~(size_t)1);
    m.fc_words = std::max(m.fc_words, m.fc_desc[(size_t)b * 4 + 1]);
    tab[0] = (uint32_t)(rows[0] / 4) | (uint32_t)(rows[1] / 2) << 7 | (uint32_t)(rows[2] / 2) << 15 |
             (uint32_t)std::min(kin, KI) << 23;
    tab[1] = (uint32_t)rows[3] | (uint32_t)(matrix ? 1 : std::max(0, kin - KI)) << 8;
    uint32_t* s0 = tab + rec_at;
    uint32_t* s1 = s0 + 64 * rows[0];
    uint32_t* s2 = s1 + 64 * rows[1];
    uint32_t* s2c = s2 + 64 * rows[2];
    uint32_t* s3 = s2c + 32 * rows[2];
    uint32_t* more = s3 + 64 * rows[3];
    for (int l = 0; l < 32; l++)
    {
      uint32_t* own = tab + 8 + (pair ? 2 : 4) * l;
      own[0] = base[l];
      own[1] = degree[l];
      if (!pair)
      {
        own[2] = negs[l];
        own[3] = alone[l];
      }
      // (padding records have no weight, and an op that leaves the mask alone)
      // (longest first)
      int c = 2;
      size_t x = 0;
      const uint32_t pad = pair ? 0u : ising ? none : none + 1;
      auto take = [&]() -> Rec {
        while (c >= 0 && x == rec[l][c].size()) c--, x = 0;
        return c >= 0 ? rec[l][c][x++] : Rec{{pad, none, none}, 0u};
      };
      for (int k = 0; k < rows[2]; k++)
      {
        const Rec r = take();
        s2[(k * 32 + l) * 2] = r.lit[0] | r.lit[1] << 16;
        s2[(k * 32 + l) * 2 + 1] = r.val;
        s2c[k * 32 + l] = r.lit[2];
      }
      for (int k = 0; k < rows[1]; k++)
      {
        const Rec r = take();
        s1[(k * 32 + l) * 2] = r.lit[0] | r.lit[1] << 16;
        s1[(k * 32 + l) * 2 + 1] = r.val;
      }
      for (int k = 0; k < rows[0]; k++)
      {
        const Rec r = take();
        s0[(k * 32 + l) * 2] = r.lit[0];
        s0[(k * 32 + l) * 2 + 1] = r.val;
      }
      for (int k = 0; k < rows[3]; k++)
      {
        const bool have = (size_t)k < wide[l].size();
        s3[(k * 32 + l) * 2] = have ? wide[l][k].w[0] | wide[l][k].w[2] << 29 : 1u << 30;
        s3[(k * 32 + l) * 2 + 1] = have ? wide[l][k].w[1] : 0u;
      }
      if (matrix)
      {
        // one entry with the members' lanes and no value
        for (const Entry& e : in[l])
        {
          tab[ent_at + l * ew] |= e.w[0];
          more[32 * __builtin_ctz(e.w[0]) + l] += e.w[1];
        }
        continue;
      }
      for (size_t k = 0; k < in[l].size(); k++)
        memcpy(k < (size_t)KI ? tab + ent_at + (k * 32 + l) * ew : more + ((k - KI) * 32 + l) * ew, in[l][k].w, ew * 4);
    }
  }
}

// Integer mode: every coefficient is an integer of magnitude <= 2^20 and the
// per-variable sums stay below 2^30, so int32/int64 arithmetic gives the same
// values as the reference's FP64 sums (all partial sums are exact).
static void detect_int_mode(HostModel& m)
{
  bool ok = m.M > 0;
  for (double c : m.tcost)
    if (!(std::floor(c) == c && std::fabs(c) <= 1048576.0)) { ok = false; break; }
  if (ok)
    for (int64_t v = 0; v < m.N && ok; v++)
    {
      double s = 0;
      for (int q = m.row[v]; q < m.row[v + 1]; q++) s += std::fabs(m.coef[q]);
      if (2 * s >= 1073741824.0) ok = false;
    }
  m.int_mode = ok;
  m.fscreen = true;
  m.scan32 = false;
  if (!ok)
  {
    m.coef_f.resize(m.K);
    for (int64_t q = 0; q < m.K; q++)
    {
      const double a = std::fabs(m.coef[q]);
      if (!(a == 0.0 || (a >= 1e-30 && a <= 1e30))) m.fscreen = false;
      m.coef_f[q] = (float)m.coef[q];
    }
  }
  else
  {
    double mx = 0;
    for (int64_t v = 0; v < m.N; v++)
    {
      double s = 0;
      for (int q = m.row[v]; q < m.row[v + 1]; q++) s += std::fabs(m.coef[q]);
      mx = std::max(mx, 2 * s);
    }
    m.scan32 = 32.0 * mx < 2147483647.0;
  }
  if (ok)
  {
    m.coef_i.resize(m.K);
    for (int64_t q = 0; q < m.K; q++) m.coef_i[q] = (int)m.coef[q];
    m.tcost_i.resize(m.M);
    for (int64_t t = 0; t < m.M; t++) m.tcost_i[t] = (int)m.tcost[t];
  }
}

std::unique_ptr<HostModel> build_model(int kind, int64_t n_terms,
                                       const int64_t* off, const int32_t* ids,
                                       const double* coef)
{
  if (kind < 0 || kind > 4) fail(1, "unknown model kind " + std::to_string(kind));
  if (n_terms < 0 || (n_terms > 0 && (!off || !coef)))
    fail(1, "model arrays must not be null");
  std::unique_ptr<HostModel> m(new HostModel());
  m->kind = kind;
  if (kind == K_MAXSAT) build_maxsat(*m, n_terms, off, ids, coef);
  else build_graph(*m, n_terms, off, ids, coef);
  switch (kind)
  {
    case K_ISING: m->flavor = F_PARITY; break;
    case K_ISING_PLAIN: m->flavor = F_PLAIN_ISING; break;
    case K_PUBO: m->flavor = F_COUNTER; break;
    case K_PUBO_PLAIN: m->flavor = F_PLAIN_PUBO; break;
    default: m->flavor = F_COUNTER; break;
  }
  // byte counters hold up to 255 members; wider PUBO terms use the
  // counter-free evaluation (same results, model::Pubo semantics)
  if (m->flavor == F_COUNTER && m->max_loc > 255)
  {
    if (kind == K_MAXSAT) fail(1, "MaxSat clauses with more than 255 variables are not supported");
    m->flavor = F_PLAIN_PUBO;
  }
  // GraphProperties::rescale (graph/graph_properties.h:24-40)
  // (MaxSat keeps markov::Model's default factor 1, markov/model.h:193)
  m->scale_factor = (kind == K_MAXSAT || m->max_coupling <= 1 || m->max_coupling == 0)
                        ? 1.0
                        : 1.0 / m->max_coupling;
  build_nbr(*m);
  detect_int_mode(*m);
  if (m->flavor == F_PARITY || m->flavor == F_COUNTER) build_near(*m);
  if (m->flavor == F_PARITY)
  {
    // term parity from the member spins: with one or two members per term
    // the cached term bit is the other member's spin (or a constant)
    bool pair = m->M > 0;
    for (int64_t t = 0; t < m->M && pair; t++) pair = m->trow[t + 1] - m->trow[t] <= 2;
    m->pair_only = pair;
    if (pair)
    {
      m->other.assign(m->K, -1);
      for (int64_t v = 0; v < m->N; v++)
        for (int q = m->row[v]; q < m->row[v + 1]; q++)
        {
          uint32_t t = m->inc[q] & ~kNegBit;
          for (int j = m->trow[t]; j < m->trow[t + 1]; j++)
          {
            int u = (int)(m->tvar[j] & ~kNegBit);
            if (u != v) m->other[q] = u;
          }
        }
      const int pad = (int)(((m->N + 31) / 32) * 32);  // the padding spin
      if (m->int_mode)
      {
        m->rec_i.resize(2 * m->K);
        bool small = pad < (1 << 24);
        for (int64_t q = 0; q < m->K; q++)
        {
          m->rec_i[2 * q] = m->other[q] >= 0 ? m->other[q] : pad;
          m->rec_i[2 * q + 1] = m->coef_i[q];
          small = small && m->coef_i[q] >= -128 && m->coef_i[q] <= 127;
        }
        if (small)
        {
          m->rec_p.resize(m->K);
          for (int64_t q = 0; q < m->K; q++)
            m->rec_p[q] = ((unsigned)m->rec_i[2 * q] << 8) | ((unsigned)m->coef_i[q] & 0xFFu);
        }
        build_levels(*m);
      }
      else
      {
        m->rec_f.resize(2 * m->K);
        for (int64_t q = 0; q < m->K; q++)
        {
          long long u = m->other[q] >= 0 ? m->other[q] : pad;
          double ub;
          memcpy(&ub, &u, 8);
          m->rec_f[2 * q] = ub;
          m->rec_f[2 * q + 1] = m->coef[q];
        }
      }
    }
  }
  build_fields(*m);
  return m;
}

// Level schedule of an ordered sweep (levels.cu): level(v) = 1 + the largest
// level among v's neighbours u < v, 0 without one, so neighbours never share
// a level and each variable comes after its lower neighbours and before its
// higher ones.  Entries list the variables level by level (index order
// within a level); with 8-bit coefficients and at most 15 incidences per
// variable an entry carries the variable's records too (4, 8 or 16 words),
// else it is the variable alone.  The kernel sums a lane's differences in
// 32-bit integers: models whose differences could overflow them stay on the
// other kernels.
static void build_levels(HostModel& m)
{
  m.lv_ok = m.lv_d8 = false;
  m.n_levels = m.lv_recs = m.lv_width = 0;
  m.lv_off.clear();
  m.lv_ent.clear();
  m.lv_pos.clear();
  if (m.N <= 0) return;
  std::vector<int> L((size_t)m.N, 0);
  int maxl = 0, maxdeg = 0;
  long long bound = 0, widest = 0;  // sum and largest of the variables' |largest difference|
  for (int64_t v = 0; v < m.N; v++)
  {
    int l = 0;
    for (int q = m.row[v]; q < m.row[v + 1]; q++)
    {
      const int u = m.other[q];
      if (u >= 0 && u < v) l = std::max(l, L[u] + 1);
      bound += 2LL * std::llabs((long long)m.coef_i[q]);
    }
    long long dv = 0;
    for (int q = m.row[v]; q < m.row[v + 1]; q++) dv += 2LL * std::llabs((long long)m.coef_i[q]);
    widest = std::max(widest, dv);
    L[v] = l;
    maxl = std::max(maxl, l);
    maxdeg = std::max(maxdeg, m.row[v + 1] - m.row[v]);
  }
  if (bound >= (1LL << 31)) return;
  const int nl = maxl + 1;
  std::vector<int> off((size_t)nl + 1, 0);
  for (int64_t v = 0; v < m.N; v++) off[L[v] + 1]++;
  int width = 0;
  for (int t = 0; t < nl; t++)
  {
    width = std::max(width, off[t + 1]);
    off[t + 1] += off[t];
  }
  // record slots of an entry: the fewest of 3, 4, 6, 7, 15 that hold the
  // largest row (8-bit coefficients only), else 0 (the variable alone)
  int recs = 0;
  if (!m.rec_p.empty())
    for (int c : {3, 4, 6, 7, 15})
      if (maxdeg <= c)
      {
        recs = c;
        break;
      }
  const int ew = recs ? lv_entry_words(recs) : 1;
  const int pad = (int)(((m.N + 31) / 32) * 32);
  std::vector<int> fill(off.begin(), off.end() - 1);
  std::vector<uint32_t> ent((size_t)m.N * ew, recs ? lv_record(pad, 0) : 0u);
  std::vector<int> pos((size_t)((m.N + 31) / 32) * 32, 0);
  for (int64_t v = 0; v < m.N; v++)
  {
    pos[v] = fill[L[v]];
    uint32_t* e = &ent[(size_t)fill[L[v]]++ * ew];
    e[0] = (uint32_t)v;
    if (recs)
      for (int q = m.row[v], j = 1; q < m.row[v + 1]; q++, j++)
        e[j] = lv_record(m.other[q] >= 0 ? m.other[q] : pad, m.coef_i[q]);
  }
  m.lv_off.swap(off);
  m.lv_ent.swap(ent);
  m.lv_pos.swap(pos);
  m.n_levels = nl;
  m.lv_recs = recs;
  m.lv_width = width;
  m.lv_d8 = widest <= 127;
  m.lv_ok = true;
}

// 256 bytes of tail padding: bulk copies of incidence ranges round their end up
// to 16 bytes
static size_t boundary(size_t n) { return (n + 255) & ~(size_t)255; }
size_t HostModel::device_copy_bytes() const
{
  size_t n = 0;
  device_arrays([&](const auto& v) { n = boundary(n) + v.size() * sizeof(v[0]); });
  return boundary(n) + 256;
}

void HostModel::upload() const
{
  ensure_device();
  std::vector<char> blob(device_copy_bytes());
  std::array<size_t, 22> at;
  size_t n = 0, k = 0;
  device_arrays([&](const auto& v) {
    at[k++] = n = boundary(n);
    if (!v.empty()) memcpy(blob.data() + n, v.data(), v.size() * sizeof(v[0]));
    n += v.size() * sizeof(v[0]);
  });
  const auto [o_row, o_inc, o_coef, o_ci, o_nbr, o_trow, o_tvar, o_tc, o_tci, o_cf, o_near, o_oth, o_ri, o_rf, o_rp,
              o_lo, o_le, o_lp, o_ft, o_fd, o_fo, o_fw] = at;
  // The block-decided sweep's tables, the last arrays, stay away where the device
  // has no room for them (hubs in every block make them most of a model); the
  // windowed sweep runs the model then.
  bool tables = !fc_desc.empty();
  try
  {
    dmem = DevBuf(blob.size());
  }
  catch (const Error& e)
  {
    if (e.status != 2 || !tables) throw;
    cudaGetLastError();  // (the refused allocation)
    tables = false;
    blob.resize(boundary(o_ft) + 256);
    dmem = DevBuf(blob.size());
  }
  h2d(dmem.ptr, blob.data(), blob.size(), "model upload");
  char* b = (char*)dmem.ptr;
  dev.flavor = flavor;
  dev.n_vars = (int)N;
  dev.n_terms = (int)M;
  dev.n_inc = (int)K;
  dev.sweep_size = (int)N;
  dev.int_mode = int_mode ? 1 : 0;
  dev.row = (const int*)(b + o_row);
  dev.inc = (const uint32_t*)(b + o_inc);
  dev.coef = (const double*)(b + o_coef);
  dev.coef_i = int_mode ? (const int*)(b + o_ci) : nullptr;
  dev.nbr = (const uint32_t*)(b + o_nbr);
  dev.trow = (const int*)(b + o_trow);
  dev.tvar = (const uint32_t*)(b + o_tvar);
  dev.tcost = (const double*)(b + o_tc);
  dev.tcost_i = int_mode ? (const int*)(b + o_tci) : nullptr;
  dev.coef_f = int_mode ? nullptr : (const float*)(b + o_cf);
  dev.near = near.empty() ? nullptr : (const unsigned long long*)(b + o_near);
  dev.fscreen = fscreen ? 1 : 0;
  dev.scan32 = scan32 ? 1 : 0;
  dev.pair_only = pair_only ? 1 : 0;
  int md = 0;
  for (int64_t v = 0; v < N; v++) md = std::max(md, row[v + 1] - row[v]);
  dev.max_deg = md;
  int mb = 0;
  for (int64_t b = 0; b < N; b += 32) mb = std::max(mb, row[std::min<int64_t>(b + 32, N)] - row[b]);
  dev.max_block_inc = mb;
  dev.other = other.empty() ? nullptr : (const int*)(b + o_oth);
  dev.rec_i = rec_i.empty() ? nullptr : (const int2*)(b + o_ri);
  dev.rec_f = rec_f.empty() ? nullptr : (const double2*)(b + o_rf);
  dev.rec_p = rec_p.empty() ? nullptr : (const unsigned int*)(b + o_rp);
  dev.lv_ok = lv_ok ? 1 : 0;
  dev.lv_off = lv_ok ? (const int*)(b + o_lo) : nullptr;
  dev.lv_ent = lv_ok ? (const uint32_t*)(b + o_le) : nullptr;
  dev.lv_pos = lv_ok ? (const int*)(b + o_lp) : nullptr;
  dev.n_levels = lv_ok ? n_levels : 0;
  dev.lv_recs = lv_ok ? lv_recs : 0;
  dev.lv_d8 = lv_d8 ? 1 : 0;
  dev.fc_desc = tables ? (const int4*)(b + o_fd) : nullptr;
  dev.fc_tab = tables ? (const uint2*)(b + o_ft) : nullptr;
  dev.fc_words = fc_words;
  dev.fc_oth = tables ? (const uint2*)(b + o_fo) : nullptr;
  dev.fc_wterm = tables ? (const int*)(b + o_fw) : nullptr;
  dev.fc_wide = (int)fc_wide.size();
  dev.fc_inv = std::ldexp(1.0, -fc_S);
  int ordinal = -1;
  cuda_check(cudaGetDevice(&ordinal), "cudaGetDevice");
  upload_device = ordinal;
  uploaded = true;
}

DevModel HostModel::device_view(bool full_maxsat_sweep) const
{
  DevModel d = device();
  // MaxSat does not override get_sweep_size() (markov/model.h:169): one
  // attempt (variable 0) per sweep unless the full sweep is requested.
  if (kind == K_MAXSAT && !full_maxsat_sweep) d.sweep_size = N > 0 ? 1 : 0;
  return d;
}

static std::vector<int32_t> flatten_ids(const json::Value& terms, std::vector<int64_t>& off,
                                        std::vector<double>& coef)
{
  std::vector<int32_t> ids;
  off.assign(1, 0);
  for (const auto& t : terms.arr)
  {
    const json::Value* c = t.find("c");
    const json::Value* i = t.find("ids");
    if (!c || !c->is_number()) fail(1, "parameter `c` is required");
    if (!i || !i->is_array()) fail(1, "parameter `ids` is required");
    coef.push_back(c->num);
    for (const auto& x : i->arr)
    {
      if (!x.is_number() || !x.is_int) fail(1, "ids must be integers");
      ids.push_back((int32_t)x.i);
    }
    off.push_back((int64_t)ids.size());
  }
  return ids;
}

std::unique_ptr<HostModel> build_model_json(const json::Value& doc, int kind)
{
  const json::Value* cf = doc.find("cost_function");
  if (!cf || !cf->is_object()) fail(1, "Input field `cost_function` is required.");
  const json::Value* type = cf->find("type");
  if (kind < 0)
  {
    if (!type || !type->is_string()) fail(1, "parameter `type` is required");
    if (type->str == "ising") kind = K_ISING;
    else if (type->str == "pubo") kind = K_PUBO;
    else if (type->str == "maxsat") kind = K_MAXSAT;
    else fail(1, "Unknown model type: " + type->str);
  }
  const json::Value* ver = cf->find("version");
  if (ver && ver->is_string() && kind != K_MAXSAT && ver->str != "1.0" && ver->str != "1.1")
    fail(1, "Expecting `version` equals 1.0 or 1.1, but found: " + ver->str);
  const json::Value* terms = cf->find("terms");
  if (!terms || !terms->is_array()) fail(1, "parameter `terms` is required");
  std::vector<int64_t> off;
  std::vector<double> coef;
  std::vector<int32_t> ids = flatten_ids(*terms, off, coef);
  return build_model(kind, (int64_t)coef.size(), off.data(), ids.data(), coef.data());
}

// ---------------------------------------------------------------------------
// Schedules.  Linear a + p(b-a) (schedule/linear.cc:15-18), geometric
// a(b/a)^p (schedule/geometric.cc:9-12), lists of constant points
// (Segments of constants, schedule/segments.cc:15-43,45-110), input mapping
// and clamping (schedule/schedule.cc:17-25), discretisation (38-89).
// ---------------------------------------------------------------------------
double Schedule::progress_value(double p) const
{
  switch (type)
  {
    case 0: return initial + p * (final_ - initial);
    case 1: return initial * pow(final_ / initial, p);
    case 2: return initial;
    default:
    {
      double position = get_start() + p * (get_stop() - get_start());
      if (position < 0) return values.front();
      for (size_t i = 0; i < values.size(); i++)
      {
        double stop = (double)i;
        if (position > stop) continue;
        double start = (double)i;
        if (i > 0 && position < start)
        {
          double last_stop = (double)(i - 1);
          double q = (position - last_stop) / (start - last_stop);
          return (1 - q) * values[i - 1] + q * values[i];
        }
        return values[i];
      }
      return values.back();
    }
  }
}
double Schedule::get_start() const { return has_start ? start_ : 0; }
double Schedule::get_stop() const
{
  if (has_stop) return stop_;
  if (type == 3) return (double)values.size() - 1;
  return 1;
}
int Schedule::get_count() const
{
  if (has_count) return count_;
  if (type == 3) return (int)values.size();
  return (int)round(std::abs(get_stop() - get_start()));
}
double Schedule::get_value(double input) const
{
  double start = get_start(), stop = get_stop();
  if (start == stop) return progress_value(0);
  double progress = (input - start) / (stop - start);
  return progress_value(std::min(1., std::max(0., progress)));
}
std::vector<double> Schedule::discretized() const
{
  int count = get_count();
  if (count < 2) fail(1, "Can not get_discretized_values(count) for less than 2 values");
  std::vector<double> d;
  for (int i = 0; i < count; i++) d.push_back(progress_value(double(i) / (count - 1)));
  return d;
}
std::string Schedule::render() const
{
  if (type == 0 || type == 1)
    return std::string("{\"type\":\"") + (type == 0 ? "linear" : "geometric") +
           "\",\"initial\":" + json::number(initial) + ",\"final\":" + json::number(final_) + "}";
  if (type == 2) return json::number(initial);
  std::string s = "{\"type\":\"segments\",\"segments\":[";
  for (size_t i = 0; i < values.size(); i++)
    s += (i ? "," : "") + std::string("{\"value\":") + json::number(values[i]) + "}";
  return s + "]}";
}

Schedule parse_schedule(const json::Value& v, const std::string& name)
{
  Schedule s;
  if (v.is_number())
  {
    s.type = 2;
    s.initial = v.num;
    return s;
  }
  if (v.is_array())
  {
    if (v.arr.empty())
      fail(1, "parameter `" + name + "`: unable to initialize schedule:\n  Linear: parameter `type` is required\n  Geometric: parameter `type` is required\n  Segments: `segments` must be specified as a non-empty array.\n  Constant: expected double, found array");
    s.type = 3;
    for (const auto& x : v.arr)
    {
      if (!x.is_number()) fail(1, "parameter `" + name + "`: list values must be numbers");
      s.values.push_back(x.num);
    }
    return s;
  }
  if (!v.is_object()) fail(1, "parameter `" + name + "`: unable to initialize schedule");
  const json::Value* type = v.find("type");
  std::string t = (type && type->is_string()) ? type->str : "";
  auto num = [&](const char* k, double& out, bool required) {
    const json::Value* x = v.find(k);
    if (!x) { if (required) fail(1, "parameter `" + std::string(k) + "` is required"); return false; }
    if (!x->is_number()) fail(1, "parameter `" + std::string(k) + "`: expected number");
    out = x->num;
    return true;
  };
  if (t == "linear" || t == "geometric")
  {
    s.type = t == "linear" ? 0 : 1;
    num("initial", s.initial, true);
    num("final", s.final_, true);
    if (s.type == 1 && s.initial <= 0) fail(1, "initial must be positive for geometric");
    if (s.type == 1 && s.final_ <= 0) fail(1, "final must be positive for geometric");
  }
  else if (t == "constant")
  {
    s.type = 2;
    num("value", s.initial, true);
  }
  else if (t == "segments")
  {
    s.type = 3;
    const json::Value* segs = v.find("segments");
    if (!segs || !segs->is_array() || segs->arr.empty())
      fail(1, "`segments` must be specified as a non-empty array.");
    for (const auto& x : segs->arr)
    {
      if (x.is_number()) s.values.push_back(x.num);
      else if (x.is_object() && x.find("value") && x["value"].is_number())
        s.values.push_back(x["value"].num);
      else fail(1, "only constant segments are supported");
    }
  }
  else
    fail(1, "parameter `" + name + "`: unable to initialize schedule:\n  Linear: parameter `type` is required");
  double d;
  if (num("start", d, false)) { s.has_start = true; s.start_ = d; }
  if (num("stop", d, false)) { s.has_stop = true; s.stop_ = d; }
  if (num("count", d, false)) { s.has_count = true; s.count_ = (int)d; }
  return s;
}
}  // namespace qio

// ---------------------------------------------------------------------------
// Bounds on a single flip's cost difference, used by the parameter-free
// solvers to place their temperature ranges.
// ---------------------------------------------------------------------------
namespace qio
{
static const double kMinDeltaDefault = 0.1;  // MIN_DELTA_DEFAULT, model/graph_model.h:16

// utils::least_diff_method, utils/utils.cc:43-53: replace the two largest
// values by their difference until one value is left
static double least_diff_one(std::multiset<double> s)
{
  while (s.size() > 1)
  {
    auto a = std::prev(s.end());
    const double x = *a;
    s.erase(a);
    auto b = std::prev(s.end());
    const double y = *b;
    s.erase(b);
    s.insert(x - y);
  }
  return *s.begin();
}

// the two-set form, utils/utils.cc:55-100: the largest of each set cancel;
// the smallest non-zero remainder is kept
static double least_diff_two(std::multiset<double> a, std::multiset<double> b)
{
  double mn = std::numeric_limits<double>::max();
  if (a.empty() && !b.empty()) return *b.begin();
  if (!a.empty() && b.empty()) return *a.begin();
  while (!a.empty() && !b.empty())
  {
    auto ia = std::prev(a.end());
    const double ca = *ia;
    a.erase(ia);
    auto ib = std::prev(b.end());
    const double cb = *ib;
    b.erase(ib);
    double delta = ca - cb;
    if (delta > 0)
      a.insert(delta);
    else if (delta < 0)
    {
      delta = -delta;
      b.insert(delta);
    }
    else if (a.size() < b.size())
      a.insert(ca);
    else
      b.insert(cb);
    if (mn > delta && delta != 0) mn = delta;
  }
  return mn;
}

// Ising: twice the largest sum of |c| over a variable's terms
// (model/ising.h:176-179, graph/graph.h:453-485); PUBO: that sum itself
// (model/graph_model.h:194-197)
double estimate_max_cost_diff(const HostModel& m)
{
  if (m.kind == K_MAXSAT) fail(1, "cost difference estimates are not available for maxsat models");
  double mx = 0;
  for (int64_t v = 0; v < m.N; v++)
  {
    double s = 0;
    for (int q = m.row[v]; q < m.row[v + 1]; q++) s += std::abs(m.coef[q]);
    mx = s > mx ? s : mx;
  }
  return (m.kind == K_ISING || m.kind == K_ISING_PLAIN) ? mx * 2 : mx;
}

// Ising (model/ising.h:181-224): per variable the single-set least
// difference of its |c|, zeros skipped, the smallest doubled; PUBO
// (model/pubo.h:127-184): the two-set least difference of its positive and
// negated negative c.  No non-zero value: MIN_DELTA_DEFAULT (doubled for
// Ising).
double estimate_min_cost_diff(const HostModel& m)
{
  if (m.kind == K_MAXSAT) fail(1, "cost difference estimates are not available for maxsat models");
  const bool ising = m.kind == K_ISING || m.kind == K_ISING_PLAIN;
  double mn = std::numeric_limits<double>::max();
  for (int64_t v = 0; v < m.N; v++)
  {
    double local;
    if (ising)
    {
      std::multiset<double> s;
      for (int q = m.row[v]; q < m.row[v + 1]; q++) s.insert(std::abs(m.coef[q]));
      if (s.empty()) continue;
      local = least_diff_one(s);
    }
    else
    {
      std::multiset<double> pos, neg;
      for (int q = m.row[v]; q < m.row[v + 1]; q++)
      {
        const double c = m.coef[q];
        if (c > 0) pos.insert(c);
        else if (c < 0) neg.insert(-c);
      }
      local = least_diff_two(pos, neg);
    }
    if (local == 0) continue;
    mn = local < mn ? local : mn;
  }
  if (mn == std::numeric_limits<double>::max()) mn = kMinDeltaDefault;
  return ising ? mn * 2 : mn;
}
}  // namespace qio
