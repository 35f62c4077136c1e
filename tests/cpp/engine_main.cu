// Drives the engine's classes and launchers from inside, for what the C ABI does
// not show.  Usage: engine_main MODE ARGUMENTS; exit code 3 when the engine throws.
//   purify IN OUT   IN: int n, int nocc, n x n doubles F; OUT: int flags, int
//                   error word, n x n doubles P
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <exception>
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
  if (n <= kPurSmallMaxN) {
    launch_purify_small(d_mol, d_list, 1, n, d_st, d_F, d_P, d_err, nullptr);
  } else {
    std::vector<int4> tiles(purify_tiles(0, n, 64, nullptr));
    purify_tiles(0, n, 64, tiles.data());
    int4* d_tiles = device(tiles);
    PurState* d_pur = device(std::vector<PurState>(1));
    PurScratch ws;
    for (double*& m : ws.m) m = device(std::vector<double>((F.size() + 31) / 32 * 32, 0.0));
    launch_purify_big(d_mol, d_list, 1, n, d_tiles, (int)tiles.size(), 64, d_st, d_F, d_P, d_pur, ws, kPurBigSteps, true,
                      d_err, nullptr);
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

int main(int argc, char** argv) {
  try {
    const std::string mode = argc > 1 ? argv[1] : "";
    if (mode == "purify" && argc == 4) return purify(argv[2], argv[3]);
    std::fprintf(stderr, "unknown mode\n");
    return 2;
  } catch (const std::exception& e) {
    std::printf("error %s\n", e.what());
    return 3;
  }
}
