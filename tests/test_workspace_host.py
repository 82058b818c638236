"""The sweep workspace (fh_pool.h) against a memory cache that the test fakes:
what it remembers of the batches that fitted has to go with a slot that a
failed growth loses, so that the next sweep looks at the free memory again and
comes in smaller batches."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "fh_pool.h"

#include <cstdio>
#include <cstdlib>

static size_t room = 1000, used = 0;
namespace fhb {
cudaError_t cache_alloc(void **p, size_t bytes, cudaStream_t) {
    if (used + bytes > room) return cudaErrorMemoryAllocation;
    used += bytes;
    size_t *q = (size_t *)std::malloc(sizeof(size_t) + bytes);
    *q = bytes;
    *p = q;
    return cudaSuccess;
}
void cache_free(void *p, cudaStream_t) {
    used -= *(size_t *)p;
    std::free(p);
}
}  // namespace fhb

#define CHECK(x)                                  \
    if (!(x)) {                                   \
        std::printf("line %d: %s\n", __LINE__, #x); \
        return 1;                                 \
    }

int main() {
    {
        fhb::DevPool pool;
        void *a = nullptr, *b = nullptr, *again = nullptr;
        CHECK(pool.get(2, 400, &a) == cudaSuccess && pool.get(0, 300, &b) == cudaSuccess);
        pool.batch[1] = 8;
        CHECK(pool.get(2, 100, &again) == cudaSuccess && again == a);  // a smaller batch
        CHECK(pool.get(0, 500, &again) == cudaSuccess);                // growth that fits
        CHECK(pool.batch[1] == 8 && pool.held() == 900);
        CHECK(pool.get(2, 600, &again) != cudaSuccess);  // growth that does not: the slot is gone
        CHECK(pool.held() == 500 && used == 500);
        CHECK(pool.batch[0] == 0 && pool.batch[1] == 0 && pool.batch[2] == 0);
        CHECK(pool.get(2, 450, &again) == cudaSuccess && pool.held() == 950);  // a smaller batch fits
        pool.batch[2] = 3;
        pool.release();
        CHECK(pool.held() == 0 && used == 0 && pool.batch[2] == 0);
        CHECK(pool.get(2, 900, &again) == cudaSuccess);
    }
    CHECK(used == 0);  // the destructor frees
    return 0;
}
"""


def test_a_lost_slot_forgets_the_batches_that_fitted(tmp_path):
    from fasterhenry_b200 import build
    source, program = tmp_path / "pool.cpp", tmp_path / "pool"
    source.write_text(PROGRAM)
    subprocess.run([build.HOST_CXX, "-std=c++17", "-Wall", "-I" + build.CSRC,
                    "-I" + os.path.join(build.CUDA_HOME, "include"), str(source), "-o", str(program)], check=True)
    r = subprocess.run([str(program)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
