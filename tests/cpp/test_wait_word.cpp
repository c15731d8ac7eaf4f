// Error words of the FP64 contraction's device-side waits: one word's error is reported by its
// own check, once, and a context's only by that context.  The error is written through the
// word's device address, as a wait that gives up would write it.
#include "tb_runtime.hpp"

#include "tamm_b200.h"

#include <cstdio>

static int failures = 0;
#define CHECK(x)                                                  \
  do {                                                            \
    if(!(x)) {                                                    \
      std::printf("FAILED line %d: %s\n", __LINE__, #x);          \
      failures++;                                                 \
    }                                                             \
  } while(0)

static bool raises(tb::WaitWord& w) {
  try {
    w.check();
  } catch(const tb::Error& e) {
    return e.code == TB_ERR_TIMEOUT;
  }
  return false;
}

static void give_up(int* word) {
  const int code = 34;
  CHECK(cudaMemcpy(word, &code, sizeof(int), cudaMemcpyHostToDevice) == cudaSuccess);
}

int main() {
  {
    tb::WaitWord a, b;
    CHECK(a.device() != b.device() && !raises(a) && !raises(b));
    give_up(b.device());
    CHECK(!raises(a));
    CHECK(raises(b));
    CHECK(!raises(b));
    give_up(a.device()); // goes with the word
  }
  {
    tb::WaitWord c, d; // on the lines of a and b
    CHECK(!raises(c) && !raises(d));
  }
  tb_ctx x = nullptr, y = nullptr;
  CHECK(tb_ctx_create(0, 1 << 20, &x) == TB_OK && tb_ctx_create(0, 1 << 20, &y) == TB_OK);
  give_up(y->p->waits->device());
  CHECK(tb_ctx_synchronize(x) == TB_OK);
  CHECK(tb_ctx_synchronize(y) == TB_ERR_TIMEOUT);
  CHECK(tb_ctx_synchronize(y) == TB_OK);
  // a block product reports its own waits, not a context's
  give_up(x->p->waits->device());
  double* m = nullptr;
  CHECK(cudaMalloc(reinterpret_cast<void**>(&m), 3 * sizeof(double)) == cudaSuccess);
  const double  v[3] = {2.0, 3.0, 0.0};
  double        r    = 0.0;
  const int64_t one  = 1;
  const int     i = 1, j = 2, k = 3, la[2] = {i, k}, lb[2] = {k, j}, lc[2] = {i, j};
  const int64_t dims[2] = {one, one};
  CHECK(cudaMemcpy(m, v, sizeof v, cudaMemcpyHostToDevice) == cudaSuccess);
  CHECK(tb_block_multiply(1.0, m, dims, la, 2, m + 1, dims, lb, 2, 1.0, m + 2, dims, lc, 2, 1, TB_MODE_FP64, nullptr) == TB_OK);
  CHECK(cudaMemcpy(&r, m + 2, sizeof r, cudaMemcpyDeviceToHost) == cudaSuccess && r == 6.0);
  cudaFree(m);
  CHECK(tb_ctx_synchronize(x) == TB_ERR_TIMEOUT);
  tb_ctx_destroy(x);
  tb_ctx_destroy(y);
  if(failures == 0) std::printf("ALL PASSED\n");
  return failures == 0 ? 0 : 1;
}
