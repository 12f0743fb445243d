"""The materializing join's match count, its kernel text run on the CPU: a thread for every CUDA thread of one
CTA, the first one always released ahead of the others by a barrier (an order the hardware may take). Every
tile's count must be that of its own left rows, whatever the order."""
import re
import subprocess
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parent.parent / "vectisdb_b200" / "csrc" / "kernels.cu"

SHIM = r"""
#include <algorithm>
#include <barrier>
#include <chrono>
#include <cstdint>
#include <cstdio>
#include <memory>
#include <thread>
#include <vector>
using std::max;
typedef unsigned long long u64;
typedef uint32_t u32;
#define __global__
#define __launch_bounds__(n)
#define __shared__ static
constexpr int kJoinBlock = 64, kJoinItems = 4, kJoinTile = kJoinBlock * kJoinItems;
struct Dim { uint32_t x; };
static thread_local Dim threadIdx;
static std::barrier<> cta(kJoinBlock);
static std::vector<std::unique_ptr<std::barrier<>>> warps;
static uint64_t lanes[kJoinBlock];
static void __syncthreads() {
	cta.arrive_and_wait();
	if (threadIdx.x != 0) std::this_thread::sleep_for(std::chrono::milliseconds(2));
}
static uint64_t __shfl_xor_sync(unsigned, uint64_t v, int o) {
	std::barrier<> &b = *warps[threadIdx.x / 32];
	lanes[threadIdx.x] = v;
	b.arrive_and_wait();
	const uint64_t r = lanes[threadIdx.x ^ o];
	b.arrive_and_wait();
	return r;
}
template <typename T> static T atomicAdd(T *p, T v) { return __atomic_fetch_add(p, v, __ATOMIC_SEQ_CST); }
template <typename T> static T atomicOr(T *p, T v) { return __atomic_fetch_or(p, v, __ATOMIC_SEQ_CST); }
static void atomicMax(uint32_t *p, uint32_t v) {
	for (uint32_t o = *p; o < v && !__atomic_compare_exchange_n(p, &o, v, false, __ATOMIC_SEQ_CST, __ATOMIC_SEQ_CST);) {}
}
template <typename T> static void st_relaxed(T *p, T v) { *p = v; }
template <typename... A> static u64 tile_scanner(A...) { return 0; }  // the CTA below is not the scanning one
template <typename... A> static void tiles_total(A...) {}
constexpr uint32_t kJoinRunLimit = 4096;
struct JoinRunsView { const uint32_t *info = nullptr; };
struct uint2 { uint32_t x, y; };
static uint2 JoinRunOf(const JoinRunsView &, uint64_t key) { return {0, static_cast<uint32_t>(key)}; }  // key = matches
"""

MAIN = r"""
int main() {
	const uint64_t n = 7 * kJoinTile + 13, ntiles = (n + kJoinTile - 1) / kJoinTile;
	std::vector<uint64_t> keys(n), want(ntiles), chain(2 + (ntiles + 1) / 2 + ntiles);
	for (uint64_t i = 0; i < n; i++) want[i / kJoinTile] += keys[i] = (i / kJoinTile + 1) * (i % 3);
	chain[1] = 1;  // the scanning CTA has taken the first ticket
	for (int w = 0; w < kJoinBlock / 32; w++) warps.push_back(std::make_unique<std::barrier<>>(32));
	std::vector<std::thread> threads;
	for (uint32_t t = 0; t < kJoinBlock; t++) {
		threads.emplace_back([&, t] {
			threadIdx.x = t;
			JoinMatchCountKernel<uint64_t>(keys.data(), n, JoinRunsView(), ntiles, chain.data()@EXTRA@);
		});
	}
	for (auto &t : threads) t.join();
	const uint32_t *counts = reinterpret_cast<uint32_t *>(chain.data() + 2);
	for (uint64_t t = 0; t < ntiles; t++) {
		if (counts[t] != want[t] + 1) return std::printf("tile %d: %u, not %d\n", (int)t, counts[t], (int)want[t] + 1), 1;
	}
	return 0;
}
"""


def test_every_tile_is_counted_by_the_whole_cta(tmp_path):
    text = SOURCE.read_text()
    found = re.search(r"template <typename K>\n__global__ void __launch_bounds__\(kJoinBlock\) JoinMatchCountKernel.*?\n}\n",
                      text, re.S)
    assert found
    extra = found.group(0).split(")", 2)[1].count(",") - 4  # arguments after the chain
    (tmp_path / "cta.cpp").write_text(SHIM + found.group(0) + MAIN.replace("@EXTRA@", ", 0" * max(0, extra)))
    built = subprocess.run(["g++", "-std=c++20", "-O1", "-pthread", "-o", str(tmp_path / "cta"), str(tmp_path / "cta.cpp")],
                           capture_output=True, text=True)
    assert built.returncode == 0, built.stderr
    try:
        ran = subprocess.run([str(tmp_path / "cta")], capture_output=True, text=True, timeout=60)
    except subprocess.TimeoutExpired:
        pytest.fail("threads of one CTA parted: they no longer meet at the same barriers")
    assert ran.returncode == 0, ran.stdout
