// Checks of the on-chip driver's host side (kernels_resident.cu), linked with the
// library's objects and fake_cudart.cpp.  Each returns the number of faults found.
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <unordered_map>
#include <vector>

#include "resident.cuh"

using namespace nrpyell;

extern "C" {
extern void (*g_fake_cooperative)(const void*, dim3, dim3, void**, size_t);
extern void (*g_fake_forget)(const void*, size_t);
}

namespace {

constexpr int kExchangeSlots = 8;
enum Role { kNone, kValue, kTag64, kTagged32 };
std::unordered_map<size_t, int> g_role;  // what each 8-byte word last held since it was cleared
int g_faults = 0;
bool g_single = false;  // precision of the running driver

void forget(const void* p, size_t n) {
  for (size_t w = (size_t)p / 8; w < ((size_t)p + n + 7) / 8; w++) g_role.erase(w);
}

// A word that a launch reads as a tag must hold a tag or nothing.
void use(const void* p, size_t i, int role) {
  int& r = g_role[(size_t)p / 8 + i];
  if (role != kValue && r != kNone && r != role) {
    if (g_faults++ == 0) fprintf(stderr, "word %zu of %p: role %d, before %d\n", i, p, role, r);
  }
  r = role;
}

template <typename T>
void exchange_words(void** args) {
  const ResJob<T>* jobs = *(const ResJob<T>**)args[0];
  const int njobs = *(int*)args[1];
  for (int j = 0; j < njobs; j++) {
    const ResJob<T>& J = jobs[j];
    const size_t n = (size_t)kExchangeSlots * J.xu_slot;
    for (size_t i = 0; i < n; i++) {
      if (sizeof(T) == 4) {
        use(J.xu, i, kTagged32);
      } else {
        use(J.xu, 2 * i, kValue);
        use(J.xu, 2 * i + 1, kTag64);
      }
    }
    for (size_t i = 0; i < (size_t)2 * J.n0t * J.n1t; i++) {
      use(J.part, 2 * i, kValue);
      use(J.part, 2 * i + 1, kTag64);
    }
  }
}
void on_launch(const void*, dim3, dim3, void** args, size_t) {
  if (g_single)
    exchange_words<float>(args);
  else
    exchange_words<double>(args);
}

struct FakeGrid {
  RfmTables rt;
  BcTables bt;
  L2Tables lt;
  std::vector<int> state;
  std::vector<double> history;
  ResGrid g;
  FakeGrid(int n0, int n1, int n2, double log10_tol, int max_steps, double volume) : state(8), history(max_steps + 2) {
    memset((void*)&rt, 0, sizeof(rt));
    memset((void*)&bt, 0, sizeof(bt));
    memset((void*)&lt, 0, sizeof(lt));
    lt.volume = volume;
    memset((void*)&g, 0, sizeof(g));
    g.d.Nxx0 = n0;
    g.d.Nxx1 = n1;
    g.d.Nxx2 = n2;
    g.d.N0 = n0 + 2 * NGHOSTS;
    g.d.N1 = n1 + 2 * NGHOSTS;
    g.d.N2 = n2 + 2 * NGHOSTS;
    g.d.Ntot = (long long)g.d.N0 * g.d.N1 * g.d.N2;
    g.rt = &rt;
    g.bt = &bt;
    g.lt = &lt;
    g.rp.dt = 1e-3;
    g.rp.log10_tol = log10_tol;
    g.rp.max_steps = max_steps;
    g.state = state.data();
    g.history = history.data();
  }
};

template <typename T>
void relax(const std::vector<FakeGrid*>& grids) {
  std::vector<ResGrid> gs;
  for (FakeGrid* f : grids) gs.push_back(f->g);
  std::vector<RelaxResult> r;
  g_single = sizeof(T) == 4;
  if (!relax_resident<T>(gs, &r)) g_faults++;
}

// A launch as the jobs' block 0 leaves it, for jobs that end at g_stop[j]: what
// any other block makes of the state must not depend on when it reads it.
std::vector<int> g_stop;
int g_next_first = 0;
void on_stepping_launch(const void*, dim3, dim3, void** args, size_t) {
  const ResJob<double>* jobs = *(const ResJob<double>**)args[0];
  const int njobs = *(int*)args[1], steps = *(int*)args[3], first = *(int*)args[4];
  if (first != g_next_first) g_faults++;
  g_next_first = first + steps;
  for (int j = 0; j < njobs; j++) {
    int* st = jobs[j].state;
    const bool over = stopped_before(st[1], first);
    if (over != (g_stop[j] < first)) g_faults++;
    for (int n = first; !over && n < first + steps; n++) {
      if (n == g_stop[j])
        st[1] = stop_mark(n);
      else
        st[0] = n + 1;
      if (stopped_before(st[1], first)) g_faults++;
      if (n == g_stop[j]) break;
    }
  }
}

// The stop test of a launch's job against the plain rule (finalize_l2).
std::vector<double> g_sums;
void on_launch_compare_stop(const void*, dim3, dim3, void** args, size_t) {
  const ResJob<double>& J = **(const ResJob<double>**)args[0];
  for (double s : g_sums) {
    const double l2 = log10(1e-16 + sqrt(s / J.volume));
    if (residual_met(J, s) != (J.check_every > 0 ? l2 < J.log10_tol : l2 <= J.log10_tol)) {
      g_faults++;
      fprintf(stderr, "sum %g, volume %g, tolerance %g\n", s, J.volume, J.log10_tol);
    }
  }
}

}  // namespace

extern "C" {

int check_stop_rule(double log10_tol, double volume, int check_every, const double* sums, int n) {
  g_faults = 0;
  g_sums.assign(sums, sums + n);
  FakeGrid a(24, 17, 8, log10_tol, 0, volume);
  a.g.rp.check_every = check_every;
  g_fake_cooperative = on_launch_compare_stop;
  relax<double>({&a});
  g_fake_cooperative = nullptr;
  release_resident();
  return g_faults;
}

// Team sizes that a batch of n grids (Nxx, three ints each) gets, 0: batched launches.
void route_of(int fp64, const int* nxx, int n, int* team) {
  std::vector<Dims> d;
  for (int i = 0; i < n; i++) d.push_back(FakeGrid(nxx[3 * i], nxx[3 * i + 1], nxx[3 * i + 2], -10.0, 0, 1.0).g.d);
  const std::vector<int> t = fp64 ? chip_route<double>(d) : chip_route<float>(d);
  std::copy(t.begin(), t.end(), team);
}

int check_alternates(int fp64, double points) {
  return fp64 ? march_alternates<double>(points, false) : march_alternates<float>(points, true);
}

// Jobs that end at the given steps of several launches.
int check_start_state(const int* stop, int n) {
  g_faults = 0;
  g_next_first = 0;
  g_stop.assign(stop, stop + n);
  std::vector<FakeGrid*> grids;
  std::vector<ResGrid> gs;
  for (int j = 0; j < n; j++) {
    grids.push_back(new FakeGrid(24, 17, 8, -10.0, 1600, 1.0));
    gs.push_back(grids[j]->g);
  }
  std::vector<RelaxResult> r;
  g_fake_cooperative = on_stepping_launch;
  if (!relax_resident<double>(gs, &r)) g_faults++;
  g_fake_cooperative = nullptr;
  for (int j = 0; j < n; j++) {
    if (r[j].steps != stop[j]) g_faults++;
    delete grids[j];
  }
  release_resident();
  return g_faults;
}

// FP64 and FP32 launches in turn, of several grids and team sizes: no word that
// one of them reads as a tag may hold what another wrote as a value.
int check_exchange_roles(void) {
  g_faults = 0;
  g_role.clear();
  g_fake_cooperative = on_launch;
  g_fake_forget = forget;
  FakeGrid a(24, 17, 8, -10.0, 600, 1.0), a2(24, 17, 8, -10.0, 600, 1.0), b(64, 64, 8, -10.0, 5, 1.0),
      c(33, 40, 12, -10.0, 5, 1.0);
  for (int k = 0; k < 2; k++) {
    relax<double>({&b});
    relax<float>({&a});
    relax<double>({&a});
    relax<float>({&a, &a2});
    relax<float>({&c});
    relax<double>({&a, &a2});
    relax<float>({&b});
    relax<double>({&c});
  }
  g_fake_cooperative = nullptr;
  g_fake_forget = nullptr;
  release_resident();
  return g_faults;
}

}  // extern "C"
