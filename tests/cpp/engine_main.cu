// Drives the engine's classes and launchers from inside, for what the C ABI does
// not show.  Usage: engine_main MODE ARGUMENTS; exit code 3 when the engine throws.
//   purify IN OUT   IN: int n, int nocc, n x n doubles F; OUT: int flags, int
//                   error word, n x n doubles P
//   waits MOLECULE  an iteration whose purification waits run out at once, the same
//                   again with the usual limit, a whole SCF of either kind; prints
//                   flags, iteration, error word and the energies
//   server MOLECULE a served request after a lane's wait error was set
//   guess MOLECULE  flags, iteration and error word after an iteration from the guess
//                   that has every purification step but not the eigensolver
//   hcore MOLECULE  the core-core energy after the integrals and after the core
//                   Hamiltonian was formed from them once more
// MOLECULE: the theory number, then "Z x y z" per line (bohr).
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <fstream>
#include <stdexcept>
#include <string>
#include <vector>

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <deque>
#include <map>
#include <memory>
#include <mutex>
#include <thread>
#define private public
#include "server.h"
#undef private

using namespace nddo;

template <typename T>
static T* device(const std::vector<T>& v) {
  T* p = nullptr;
  cuda_check(cudaMalloc(&p, sizeof(T) * v.size()), "cudaMalloc");
  cuda_check(cudaMemcpy(p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice), "copy");
  return p;
}

static int purify(const char* in, const char* out) {
  FILE* f = std::fopen(in, "rb");
  int n = 0, nocc = 0;
  if (!f || std::fread(&n, 4, 1, f) != 1 || std::fread(&nocc, 4, 1, f) != 1) throw std::runtime_error("input");
  std::vector<double> F((size_t)n * n);
  if (std::fread(F.data(), 8, F.size(), f) != F.size()) throw std::runtime_error("input");
  std::fclose(f);
  DevMol mol;
  std::memset(&mol, 0, sizeof(mol));
  mol.natoms = n;
  mol.nao = n;
  mol.nocc = nocc;
  MolState st;
  std::memset(&st, 0, sizeof(st));
  DevMol* d_mol = device(std::vector<DevMol>{mol});
  MolState* d_st = device(std::vector<MolState>{st});
  int* d_list = device(std::vector<int>{0});
  int* d_err = device(std::vector<int>{0});
  double* d_F = device(F);
  double* d_P = device(std::vector<double>(F.size(), 0.0));
  PurState* d_pur = device(std::vector<PurState>(1));
  if (n <= kPurSmallMaxN) {
    launch_purify_small(d_mol, d_list, 1, n, d_st, d_F, d_P, d_pur, d_err, kPurWaitCycles, nullptr);
  } else {
    std::vector<int4> tiles(purify_tiles(0, n, 64, nullptr));
    purify_tiles(0, n, 64, tiles.data());
    int4* d_tiles = device(tiles);
    PurScratch ws;
    for (double*& m : ws.m) m = device(std::vector<double>((F.size() + 31) / 32 * 32, 0.0));
    launch_purify_big(d_mol, d_list, 1, n, d_tiles, (int)tiles.size(), 64, d_st, d_F, d_P, d_pur, ws, kPurBigSteps, true,
                      d_err, kPurWaitCycles, nullptr);
  }
  cuda_check(cudaGetLastError(), "launch");
  cuda_check(cudaDeviceSynchronize(), "purify");
  int err = 0;
  cuda_check(cudaMemcpy(&st, d_st, sizeof(st), cudaMemcpyDeviceToHost), "copy");
  cuda_check(cudaMemcpy(&err, d_err, sizeof(err), cudaMemcpyDeviceToHost), "copy");
  cuda_check(cudaMemcpy(F.data(), d_P, sizeof(double) * F.size(), cudaMemcpyDeviceToHost), "copy");
  f = std::fopen(out, "wb");
  if (!f) throw std::runtime_error("output");
  std::fwrite(&st.flags, 4, 1, f);
  std::fwrite(&err, 4, 1, f);
  std::fwrite(F.data(), 8, F.size(), f);
  std::fclose(f);
  return 0;
}

static MoleculeInput molecule(const char* file) {
  std::ifstream in(file);
  MoleculeInput m;
  in >> m.theory;
  int z;
  double x, y, w;
  while (in >> z >> x >> y >> w) {
    m.Z.push_back(z);
    m.xyz.insert(m.xyz.end(), {x, y, w});
  }
  return m;
}

static ScfSettings settings() {
  ScfSettings s;
  s.max_iter = 60;
  s.damping_weight = 0.0;
  s.diis_start_error = 0.1;
  s.diis_end_error = 0.0;
  return s;
}

static int waits(const char* file) {
  const ScfSettings s = settings();
  Engine eng(0);
  std::vector<double> P[2];
  for (int limited = 1; limited >= 0; --limited) {
    Batch b(&eng, {molecule(file)}, s.diis_num_error_vect);
    b.integrals();
    b.begin(s, {0}, true);
    const int n = b.nao(0);
    for (int pass = 1 - limited; pass < 2; ++pass) {   // without and with time for the waits
      b.pur_wait_ = pass == 0 ? 0 : kPurWaitCycles;
      b.iterate(s, {0}, 1);
      MolState st;
      int err = 0;
      b.copy_states_async(&st);
      b.copy_wait_error_async(&err);
      cuda_check(cudaMemsetAsync(b.d_wait_err_, 0, sizeof(int), b.stream()), "reset");
      cuda_check(cudaStreamSynchronize(b.stream()), "iteration");
      if (limited) std::printf("pass %d flags %d iter %d error %d\n", pass, st.flags, st.iter, err);
    }
    P[limited].resize((size_t)n * n);
    b.copy_matrix(2, 0, P[limited].data());
  }
  std::printf("same_density %d\n", (int)(P[0] == P[1]));
  for (int limited = 1; limited >= 0; --limited) {
    Batch b(&eng, {molecule(file)}, s.diis_num_error_vect);
    if (limited) b.pur_wait_ = 0;
    b.integrals();
    for (int again = 0; again <= limited; ++again) {
      if (again) b.pur_wait_ = kPurWaitCycles, ++b.layout_version_;   // a graph holds the limit it was captured with
      try {
        b.scf(s, true);
        std::printf("scf_ok 1\n");
      } catch (const std::exception& e) {
        std::printf("scf_error %s\n", e.what());
      }
      std::vector<MolResult> r;
      b.results(&r);
      std::printf("energy %.15e status %d iterations %d\n", r[0].energy, r[0].status, r[0].iterations);
    }
  }
  return 0;
}

static int server(const char* file) {
  Engine eng(0);
  Server srv(&eng, settings(), (size_t)1 << 30, 300);
  for (int k = 0; k < 2; ++k) {
    if (k) {
      const int one = 1;
      for (auto& L : srv.lanes_)
        cuda_check(cudaMemcpy(L->b->d_wait_err_, &one, sizeof(int), cudaMemcpyHostToDevice), "copy");
    }
    srv.submit(molecule(file));
    int got = 0;
    try {
      for (int t = 0; t < 100 && !got; ++t) got = srv.poll(100000);
    } catch (const std::exception& e) {
      std::printf("poll_error %s\n", e.what());
    }
    ServeResult r;
    if (got && srv.take(&r)) std::printf("served status %d energy %.15e\n", r.status, r.energy);
  }
  return 0;
}

static int guess(const char* file) {
  const ScfSettings s = settings();
  Engine eng(0);
  Batch b(&eng, {molecule(file)}, s.diis_num_error_vect);
  b.integrals();
  b.begin(s, {0}, true);
  b.iterate(s, {0}, 1);
  MolState st;
  int err = 0;
  b.copy_states_async(&st);
  b.copy_wait_error_async(&err);
  cuda_check(cudaStreamSynchronize(b.stream()), "iteration");
  std::printf("n %d flags %d iter %d error %d\n", b.nao(0), st.flags, st.iter, err);
  return 0;
}

static int hcore(const char* file) {
  Engine eng(0);
  Batch b(&eng, {molecule(file)}, 5);
  for (int k = 0; k < 2; ++k) {
    if (k == 0) b.integrals();
    else
      launch_hcore_kernel(b.d_atoms, b.d_pairs, b.d_mols, b.d_list, 1, b.natoms(0), b.d_blocks, b.d_ecore_pair, b.d_td,
                          eng.eri(), b.d_epc, b.d_H, b.d_state, b.stream());
    MolState st;
    b.copy_states_async(&st);
    cuda_check(cudaStreamSynchronize(b.stream()), "hcore");
    std::printf("ecore %.17e\n", st.ecore);
  }
  return 0;
}

int main(int argc, char** argv) {
  try {
    const std::string mode = argc > 1 ? argv[1] : "";
    if (mode == "purify" && argc == 4) return purify(argv[2], argv[3]);
    if (mode == "waits" && argc == 3) return waits(argv[2]);
    if (mode == "guess" && argc == 3) return guess(argv[2]);
    if (mode == "hcore" && argc == 3) return hcore(argv[2]);
    if (mode == "server" && argc == 3) return server(argv[2]);
    std::fprintf(stderr, "unknown mode\n");
    return 2;
  } catch (const std::exception& e) {
    std::printf("error %s\n", e.what());
    return 3;
  }
}
