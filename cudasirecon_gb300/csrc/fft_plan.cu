// FFT plans: radix sequences and double-precision twiddle tables, cached per
// (device, length).  The tables are allocated once per length and live until
// process exit.
#include <sys/stat.h>
#include <unistd.h>

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <fstream>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <tuple>
#include <utility>
#include <vector>

#include "kernels.h"
#include "reg_fft.cuh"
#include "tf_fft.cuh"
#include "z_fft.cuh"

namespace simrecon {

namespace {
std::mutex g_mu;
std::map<std::pair<int, int>, FFTPlan> g_plans;

bool factor(int n, std::vector<int>& radix)
{
  radix.clear();
  if (n < 1) return false;
  int m = n;
  int p2 = 0;
  while (m % 2 == 0) {
    m /= 2;
    ++p2;
  }
  // powers of two in as few stages as possible: radix 32 / 16 / 8 / 4 / 2
  // (e.g. 1024 = 32*32, 512 = 32*16, 256 = 16*16, 128 = 16*8, 64 = 8*8)
  static const int plan2[14][3] = {{0, 0, 0},  {2, 0, 0},   {4, 0, 0},   {8, 0, 0},   {16, 0, 0},
                                   {32, 0, 0}, {8, 8, 0},   {16, 8, 0},  {16, 16, 0}, {32, 16, 0},
                                   {32, 32, 0}, {16, 16, 8}, {16, 16, 16}, {32, 16, 16}};
  if (p2 > 13) return false;
  for (int i = 0; i < 3; ++i)
    if (plan2[p2][i]) radix.push_back(plan2[p2][i]);
  for (int r : {3, 5, 7})
    while (m % r == 0) {
      m /= r;
      radix.push_back(r);
    }
  if (m != 1) return false;
  if ((int)radix.size() > kMaxStages) return false;
  return true;
}
}  // namespace

namespace {
thread_local KernelTimer* t_timer = nullptr;
}
void set_kernel_timer(KernelTimer* t) { t_timer = t; }
KernelTimer* kernel_timer() { return t_timer; }

// The radix sequence of get_fft_plan, written into a caller array without
// any allocation (used by the allocation-free FFT entry point).
bool fft_radix_plan(int n, int* radix, int* nstages)
{
  if (n < 1) return false;
  int m = n, p2 = 0, ns = 0;
  while (m % 2 == 0) {
    m /= 2;
    ++p2;
  }
  static const int plan2[14][3] = {{0, 0, 0},  {2, 0, 0},   {4, 0, 0},   {8, 0, 0},   {16, 0, 0},
                                   {32, 0, 0}, {8, 8, 0},   {16, 8, 0},  {16, 16, 0}, {32, 16, 0},
                                   {32, 32, 0}, {16, 16, 8}, {16, 16, 16}, {32, 16, 16}};
  if (p2 > 13) return false;
  for (int i = 0; i < 3; ++i)
    if (plan2[p2][i]) radix[ns++] = plan2[p2][i];
  for (int r : {3, 5, 7})
    while (m % r == 0) {
      if (ns >= kMaxStages) return false;
      m /= r;
      radix[ns++] = r;
    }
  if (m != 1) return false;
  *nstages = ns;
  return true;
}

// ------------------------------------------------------------- site choices
// Which FFT path a call site uses for a length the register path supports:
//  1. a choice forced on the calling thread (the tuner's trial runs),
//  2. the SIMRECON_FFT_REGISTER_SITES hex mask (a manual override),
//  3. the tuned table: choices measured by SRX_tuneFFT on this GPU model and
//     kept in a plan-cache file (SIMRECON_FFT_PLAN_CACHE, else
//     $XDG_CACHE_HOME or ~/.cache /cudasirecon_gb300/fft_plans.tsv), one line
//     per choice: GPU name, site, length, path, and both measured times,
//  4. the built-in default.
namespace {
const char* const kSiteNames[kNumFftSites] = {"ingest_x", "ingest_y", "separate_z", "overlap_x", "overlap_y",
                                              "crosscorr_rows", "crosscorr_cols", "assemble_y", "assemble_x",
                                              "assemble_z", "makeotf", "selftest"};
const char* const kPathNames[] = {"stockham", "register", "two-factor", "compiled"};
thread_local int t_force_site = -1, t_force_path = 0;
thread_local std::set<std::pair<int, int>>* t_seen = nullptr;

struct Tuned {
  bool loaded = false;
  // (gpu name, site, n) -> path, its time and the best other path's
  std::map<std::tuple<std::string, int, int>, std::pair<int, std::pair<double, double>>> table;
};
std::mutex g_tuned_mu;
Tuned g_tuned;
std::map<int, std::string> g_dev_names;

std::string cache_path()
{
  if (const char* e = std::getenv("SIMRECON_FFT_PLAN_CACHE")) return e;
  std::string base;
  if (const char* x = std::getenv("XDG_CACHE_HOME")) base = x;
  else if (const char* h = std::getenv("HOME")) base = std::string(h) + "/.cache";
  else base = "/tmp";
  return base + "/cudasirecon_gb300/fft_plans.tsv";
}

std::string device_name()
{
  int dev = 0;
  cudaGetDevice(&dev);
  auto it = g_dev_names.find(dev);
  if (it != g_dev_names.end()) return it->second;
  cudaDeviceProp prop{};
  std::string name = cudaGetDeviceProperties(&prop, dev) == cudaSuccess ? prop.name : "unknown";
  for (char& c : name)
    if (c == '\t' || c == '\n') c = ' ';
  g_dev_names[dev] = name;
  return name;
}

int site_index(const std::string& name)
{
  for (int i = 0; i < kNumFftSites; ++i)
    if (name == kSiteNames[i]) return i;
  return -1;
}

// caller holds g_tuned_mu
void load_tuned()
{
  if (g_tuned.loaded) return;
  g_tuned.loaded = true;
  std::ifstream f(cache_path());
  std::string line;
  while (std::getline(f, line)) {
    std::vector<std::string> col;
    size_t a = 0;
    for (size_t b; (b = line.find('\t', a)) != std::string::npos; a = b + 1) col.push_back(line.substr(a, b - a));
    col.push_back(line.substr(a));
    if (col.size() < 6) continue;
    const int site = site_index(col[1]);
    const int n = std::atoi(col[2].c_str());
    int path = -1;
    for (int q = 0; q < kNumFftPaths; ++q)
      if (col[3] == kPathNames[q]) path = q;
    if (site < 0 || n <= 0 || path < 0) continue;
    g_tuned.table[{col[0], site, n}] = {path, {std::atof(col[4].c_str()), std::atof(col[5].c_str())}};
  }
}

// caller holds g_tuned_mu; the whole table is rewritten through a temporary
// file and a rename, so a concurrent reader sees the old or the new file
bool save_tuned(std::string* err)
{
  const std::string path = cache_path();
  const size_t slash = path.find_last_of('/');
  if (slash != std::string::npos) {
    std::string dir = path.substr(0, slash), cur;
    for (size_t i = 0; i <= dir.size(); ++i)
      if (i == dir.size() || dir[i] == '/') {
        cur = dir.substr(0, i);
        if (!cur.empty()) mkdir(cur.c_str(), 0755);
      }
  }
  const std::string tmp = path + ".tmp" + std::to_string((long)getpid());
  {
    std::ofstream f(tmp, std::ios::trunc);
    if (!f) {
      *err = "cannot write the FFT plan cache " + tmp;
      return false;
    }
    for (auto& [k, v] : g_tuned.table)
      f << std::get<0>(k) << '\t' << kSiteNames[std::get<1>(k)] << '\t' << std::get<2>(k) << '\t'
        << kPathNames[v.first] << '\t' << v.second.first << '\t' << v.second.second << '\n';
  }
  if (std::rename(tmp.c_str(), path.c_str()) != 0) {
    *err = "cannot replace the FFT plan cache " + path;
    return false;
  }
  return true;
}

bool builtin_choice(FftSite site, int n)
{
  // Built-in choice, from timing both paths in every kernel on GB300 at
  // 256^2 x 32 and 512^2 x 48: the register path wins for all lengths up to
  // 256 and, at any length, in the ingest rows and the short z lines; the
  // 512- and 1024-point transforms of the overlap, correlation and assembly
  // kernels are faster with the Stockham stages (the register path's 130-255
  // registers per thread leave one CTA per SM there).
  switch (site) {
    case kSiteIngestX:
    case kSiteSeparateZ:
    case kSiteAsmZ:
    case kSiteSelfTest:
      return true;
    default:
      return n <= 256;
  }
}
}  // namespace

namespace {
// what was chosen for (site, n) by a force, the environment or the plan
// cache; -1: nothing, the built-in choice holds
int chosen_path(int site, int n)
{
  if (t_force_site == site) return t_force_path;
  static const int forced = [] {
    const char* e = std::getenv("SIMRECON_FFT_REGISTER_SITES");
    return e ? (int)(std::strtoul(e, nullptr, 16) | (1u << kSiteSelfTest)) : -1;
  }();
  if (forced >= 0) return (forced >> site) & 1;
  if (site != kSiteSelfTest && reg_fft_lanes(n)) {
    std::lock_guard<std::mutex> lk(g_tuned_mu);
    load_tuned();
    auto it = g_tuned.table.find({device_name(), site, n});
    if (it != g_tuned.table.end()) return it->second.first;
  }
  return -1;
}
}  // namespace

bool fft_plan_open(FftSite site, int n)
{
  if (!reg_fft_lanes(n)) return true;
  if (t_seen) t_seen->insert({(int)site, n});
  const int c = chosen_path(site, n);
  return c < 0 || c == kPathTwoFactor;
}

bool reg_fft_site_enabled(FftSite site, int n)
{
  if (t_seen) t_seen->insert({(int)site, n});
  const int c = chosen_path(site, n);
  return c >= 0 ? c == kPathRegister : builtin_choice(site, n);
}

namespace {
// a kernel compiled for the length, taken whatever the plan says
bool compiled_at(int site, int n)
{
  const bool pow2 = n == 256 || n == 512 || n == 1024;
  switch (site) {
    case kSiteIngestX: return pow2;       // k_ingest_xw
    case kSiteIngestY: return n == 1024;  // k_fft_cols_4s
    case kSiteOvlY: return n == 512;      // k_ovl_y4
    case kSiteAsmY:                       // k_asm_y4f, k_asm_y4
    case kSiteAsmX: return pow2;          // k_asm_xw
    case kSiteAsmZ: return z_length_ok(n) || n == 80 || n == 96 || n == 128;  // k_asm_zr, k_asm_z2; k_asm_z4
    case kSiteSeparateZ:                  // k_separate_zn; k_separate4
      return (z_length_ok(n) && !reg_fft_lanes(n)) || n == 32 || n == 48 || n == 64 || n == 80 || n == 96 || n == 128;
    default: return false;
  }
}
// a two-factor kernel; *fixed: taken whatever the plan says, in the place of
// the compiled kernels that these lengths had
bool two_factor_at(int site, int n, bool* fixed)
{
  int r1, r2;
  *fixed = false;
  switch (site) {
    case kSiteIngestX: return n % 2 == 0 && tf_factor(n, &r1, &r2);
    case kSiteIngestY: *fixed = n == 256 || n == 512; break;
    case kSiteOvlX: *fixed = n == 256 || n == 512 || n == 1024; break;
    case kSiteOvlY: *fixed = n == 256; break;
    case kSiteCorrRows:
    case kSiteCorrCols:
    case kSiteMakeOtf: break;
    case kSiteAsmY:
    case kSiteAsmX: return n % 4 == 0 && tf_factor(n / 2, &r1, &r2);
    default: return false;
  }
  return tf_factor(n, &r1, &r2);
}
}  // namespace

bool fft_two_factor_choice(FftSite site, int n)
{
  bool fixed;
  return !compiled_at(site, n) && two_factor_at(site, n, &fixed) && !fixed;
}

int fft_path(FftSite site, int n)
{
  bool fixed;
  if (compiled_at(site, n)) return kPathCompiled;
  if (two_factor_at(site, n, &fixed) && (fixed || fft_plan_open(site, n))) return kPathTwoFactor;
  return reg_fft_lanes(n) && reg_fft_site_enabled(site, n) ? kPathRegister : kPathStockham;
}

// where fft_path's answer comes from: the plan's source only where a plan has a
// say
const char* fft_path_source(int site, int n)
{
  bool fixed;
  if (compiled_at(site, n) || !reg_fft_lanes(n) || (two_factor_at(site, n, &fixed) && fixed)) return "built-in";
  const char* src = "";
  fft_plan_choice(site, n, &src);
  return src;
}

void fft_site_force(int site, int path) { t_force_site = site, t_force_path = path; }
void fft_site_unforce() { t_force_site = -1; }
void fft_sites_track(std::set<std::pair<int, int>>* seen) { t_seen = seen; }
const char* fft_path_name(int path) { return path >= 0 && path <= kPathCompiled ? kPathNames[path] : "?"; }
const char* fft_site_name(int site) { return site >= 0 && site < kNumFftSites ? kSiteNames[site] : "?"; }

bool fft_plan_record(int site, int n, int path, double ms, double ms_other, std::string* err)
{
  std::lock_guard<std::mutex> lk(g_tuned_mu);
  load_tuned();
  g_tuned.table[{device_name(), site, n}] = {path, {ms, ms_other}};
  return save_tuned(err);
}

// The plan's choice: 1 register path, 0 Stockham stages, 2 (forced or recorded)
// two-factor kernel; *source: "forced", "environment", "tuned", "built-in" (which
// of the first two, where the site has no other kernel for n) or
// "stockham-only" (no register path for n)
int fft_plan_choice(int site, int n, const char** source)
{
  const char* src = "built-in";
  int r;
  if (site < 0 || site >= kNumFftSites) return -1;
  if (!reg_fft_lanes(n)) {
    src = "stockham-only";
    r = 0;
  } else if (t_force_site == site) {
    src = "forced";
    r = t_force_path;
  } else if (std::getenv("SIMRECON_FFT_REGISTER_SITES")) {
    src = "environment";
    r = reg_fft_site_enabled((FftSite)site, n);
  } else {
    std::lock_guard<std::mutex> lk(g_tuned_mu);
    load_tuned();
    auto it = g_tuned.table.find({device_name(), site, n});
    if (it != g_tuned.table.end()) {
      src = "tuned";
      r = it->second.first;
    } else {
      r = builtin_choice((FftSite)site, n);
    }
  }
  if (source) *source = src;
  return r;
}

std::string fft_plan_cache_path() { return cache_path(); }

void allow_dynamic_smem(const void* func, size_t bytes)
{
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> cur;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  size_t& have = cur[{dev, func}];
  if (bytes > have) {
    if (cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess)
      have = bytes;
  }
}

cudaError_t default_stream_wait() { return cudaStreamSynchronize(cudaStreamLegacy); }

bool fft_length_ok(int n)
{
  std::vector<int> r;
  return factor(n, r);
}

bool get_fft_plan(int n, FFTPlan* plan)
{
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(g_mu);
  auto it = g_plans.find({dev, n});
  if (it != g_plans.end()) {
    *plan = it->second;
    return true;
  }
  std::vector<int> radix;
  if (!factor(n, radix)) return false;
  FFTPlan p{};
  p.n = n;
  p.nstages = (int)radix.size();
  for (int i = 0; i < p.nstages; ++i) p.radix[i] = radix[i];
  std::vector<float2> tw(2 * (size_t)n);
  for (int k = 0; k < n; ++k) {
    double a = -2.0 * M_PI * (double)k / (double)n;
    tw[k] = make_float2((float)cos(a), (float)sin(a));
  }
  const int P = reg_fft_lanes(n);
  if (P) {
    const int E = n / P;
    for (int k1 = 1; k1 < E; ++k1)
      for (int q = 0; q < P; ++q) tw[n + (size_t)(k1 - 1) * P + q] = tw[((size_t)q * k1) % n];
  }
  float2* d = nullptr;
  if (cudaMalloc(&d, sizeof(float2) * 2 * n) != cudaSuccess) return false;
  if (cudaMemcpy(d, tw.data(), sizeof(float2) * 2 * n, cudaMemcpyHostToDevice) != cudaSuccess ||
      default_stream_wait() != cudaSuccess) {
    cudaFree(d);
    return false;
  }
  p.tw = d;
  p.twr = P ? d + n : nullptr;
  g_plans[{dev, n}] = p;
  *plan = p;
  return true;
}

namespace {
std::map<std::pair<int, int>, TfPlan> g_tf_plans;
}  // namespace

bool tf_factor(int n, int* r1, int* r2)
{
  for (int a : kTfSizes)
    if (n % a == 0 && n / a <= a)
      for (int b : kTfSizes)
        if (b == n / a) {
          *r1 = a;
          *r2 = b;
          return true;
        }
  return false;
}

bool get_tf_plan(int n, TfPlan* plan)
{
  TfPlan p{};
  p.n = n;
  if (!tf_factor(n, &p.r1, &p.r2)) return false;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(g_mu);
  auto it = g_tf_plans.find({dev, n});
  if (it != g_tf_plans.end()) {
    *plan = it->second;
    return true;
  }
  std::vector<float2> tw(2 * (size_t)n);
  for (int k1 = 0; k1 < p.r1; ++k1)
    for (int j = 0; j < p.r2; ++j)
      for (int h = 0; h < 2; ++h) {
        const double a = -M_PI * (double)(2 * j * k1 + h * j) / (double)n;
        tw[(size_t)h * n + (size_t)k1 * p.r2 + j] = make_float2((float)cos(a), (float)sin(a));
      }
  float2* d = nullptr;
  if (cudaMalloc(&d, sizeof(float2) * tw.size()) != cudaSuccess) return false;
  if (cudaMemcpy(d, tw.data(), sizeof(float2) * tw.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
      default_stream_wait() != cudaSuccess) {
    cudaFree(d);
    return false;
  }
  p.tw = d;
  p.twh = d + n;
  g_tf_plans[{dev, n}] = p;
  *plan = p;
  return true;
}

}  // namespace simrecon
