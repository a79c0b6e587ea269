"""Host-side logic of the library that needs no GPU: the per-device bookkeeping that guards settings CUDA
keeps per device (kernel attributes, symbol addresses), compiled with g++ from the header the library uses."""
import os
import re
import subprocess
import sys
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "per_device.h"
#include <cstdio>
int main()
{
    mpq::PerDeviceOnce once;
    int bad = 0;
    // nothing is configured at the start, on any device
    for (int d = 0; d < mpq::PerDeviceOnce::MAX_DEVICES; ++d) bad += !once.needs(d);
    // configuring device 0 leaves device 1 unconfigured (the fault a per-process flag has)
    once.mark(0);
    bad += once.needs(0);
    bad += !once.needs(1);
    once.mark(1);
    bad += once.needs(1);
    bad += !once.needs(2);
    // indices outside the table are always (re)configured and never written
    bad += !once.needs(-1);
    bad += !once.needs(mpq::PerDeviceOnce::MAX_DEVICES);
    once.mark(-1);
    once.mark(mpq::PerDeviceOnce::MAX_DEVICES + 5);
    bad += !once.needs(-1);
    bad += !once.needs(mpq::PerDeviceOnce::MAX_DEVICES + 5);
    // two independent instances (two kernels) do not share state
    mpq::PerDeviceOnce other;
    bad += !other.needs(0);
    std::printf("%d\n", bad);
    return bad;
}
"""


def test_per_device_flags_are_per_device():
    with tempfile.TemporaryDirectory() as tmp:
        src, exe = os.path.join(tmp, "t.cpp"), os.path.join(tmp, "t")
        open(src, "w").write(PROGRAM)
        subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "makepad_b200", "csrc"), src, "-o", exe])
        out = subprocess.run([exe], capture_output=True, text=True)
        assert out.returncode == 0 and out.stdout.strip() == "0", out.stdout + out.stderr


NUMBERS = r"""
#include "per_device.h"
#include <cstdio>
#include <thread>
#include <vector>
int main()
{
    int bad = 0, asked = 0, v[3];
    mpq::PerDeviceNumbers<3> table;
    auto fails = [&](int (&n)[3]) { ++asked; n[0] = 7; return false; };
    auto works = [&](int (&n)[3]) { ++asked; n[0] = n[1] = n[2] = 5; return true; };
    table.get(2, v, fails);
    bad += asked != 1 || v[0] || v[1] || v[2];                             // nothing is known, and nothing is kept
    table.get(2, v, works);
    bad += asked != 2 || v[0] != 5 || v[2] != 5;                           // a failed query is made again
    table.get(2, v, fails);
    bad += asked != 2 || v[0] != 5;                                        // a good one is not
    table.get(3, v, works);
    table.get(-1, v, works);
    table.get(mpq::PerDeviceOnce::MAX_DEVICES, v, works);
    bad += asked != 5;
    mpq::PerDeviceNumbers<3> shared;                                       // several threads: one asks, all see whole rows
    asked = 0;
    std::vector<std::thread> threads;
    std::vector<int> wrong(8);
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&, t] {
            int n[3];
            for (int i = 0; i < 1000; ++i) { shared.get(i & 1, n, works); wrong[t] += n[0] != 5 || n[1] != 5 || n[2] != 5; }
        });
    for (auto& t : threads) t.join();
    for (int w : wrong) bad += w;
    bad += asked != 2;
    std::printf("%d\n", bad);
    return bad;
}
"""


def test_numbers_of_a_device_are_asked_for_again_where_the_query_failed():
    _run(NUMBERS, "-pthread")
    text = open(os.path.join(ROOT, "makepad_b200", "csrc", "mpq.cu")).read()
    body = text[text.index("static void q4_rect_clusters("):]
    assert "PerDeviceNumbers<" in body[:body.index("\n}")]


def test_no_per_process_flag_guards_a_per_device_setting():
    """Every cudaFuncSetAttribute in the library sits behind PerDeviceOnce, none behind a plain static bool."""
    csrc = os.path.join(ROOT, "makepad_b200", "csrc")
    for f in os.listdir(csrc):
        if f.endswith((".cu", ".cuh")):
            text = open(os.path.join(csrc, f)).read()
            assert "static bool configured" not in text, f


SCRATCH = r"""
#include "scratch.h"
#include <cstdio>
#include <cstdlib>
#include <map>
static std::map<void*, size_t> live;            // the fake device's blocks
static size_t most = 0;                         // the largest request that it grants
static cudaError_t last = cudaSuccess;
extern "C" cudaError_t cudaMalloc(void** p, size_t n)
{
    if (n > most) return last = cudaErrorMemoryAllocation;
    live[*p = malloc(1)] = n;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void* p)
{
    if (p) { live.erase(p); free(p); }
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
int main()
{
    int bad = 0;
    mpq::Scratch s;
    most = 1000000;
    bad += s.reserve(100) != cudaSuccess || s.bytes() != 100;
    void* first = s.as<void>();
    bad += s.reserve(60) != cudaSuccess || s.as<void>() != first;           // enough: nothing changes
    bad += s.reserve(150) != cudaSuccess || s.bytes() != 200;               // replaced by one of twice the size
    bad += !live.count(first) || !live.count(s.as<void>());                 // and the replaced block still exists
    // many small steps: the blocks that were replaced are together smaller than the one in use
    for (size_t n = 200; n < 20000; n += 7) bad += s.reserve(n) != cudaSuccess || s.bytes() < n;
    size_t all = 0;
    for (auto& b : live) all += b.second;
    bad += all - s.bytes() >= s.bytes();
    // no room for twice the size: as much as needed; no room for that either: an error, nothing changed, no error left behind
    const size_t had = s.bytes();
    most = had + 1;
    bad += s.reserve(had + 1) != cudaSuccess || s.bytes() != had + 1;
    void* now = s.as<void>();
    const size_t blocks = live.size();
    bad += s.reserve(had + 2) == cudaSuccess || s.bytes() != had + 1 || s.as<void>() != now || live.size() != blocks;
    bad += cudaGetLastError() != cudaSuccess;
    s.release();
    bad += !live.empty() || s.bytes() != 0 || s.as<void>() != nullptr;
    most = 1000000;
    bad += s.reserve(10) != cudaSuccess || live.size() != 1;                // and it can be used again
    s.release();
    std::printf("%d\n", bad);
    return bad;
}
"""


def _run(program, *flags):
    with tempfile.TemporaryDirectory() as tmp:
        src, exe = os.path.join(tmp, "t.cpp"), os.path.join(tmp, "t")
        open(src, "w").write(program)
        cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
        subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "makepad_b200", "csrc"), "-I", cuda, *flags, src, "-o", exe])
        out = subprocess.run([exe], capture_output=True, text=True)
        assert out.returncode == 0 and out.stdout.strip() == "0", out.stdout + out.stderr


def test_a_replaced_scratch_block_lives_until_the_context_is_destroyed():
    """A captured graph holds the addresses of the blocks that its launches were given."""
    _run(SCRATCH)
    for f in ("mpq.cu", "nvfp4_gemm.cu", "nvfp4.cuh"):         # and no growing buffer is freed anywhere else
        text = open(os.path.join(ROOT, "makepad_b200", "csrc", f)).read()
        assert not re.search(r"cudaFree\([^;]*\b(q4u_xs|swiglu_buf|q4_partial|q4_rect_partial|sfa_tiled|partial)\b", text), f


NEEDS = r"""
#include "q4_plan.h"
#include <cstdio>
using namespace mpq;
int main()
{
    int bad = 0;
    const int64_t shapes[][2] = {{57344, 8192}, {128256, 4096}, {22016, 4096}, {4096, 11008}, {8192, 28672}, {500, 1056}, {1, 32}, {33, 288}, {96, 28672}, {20000, 64}};
    for (auto& nk : shapes)
        for (int sms : {148, 132})
            for (int pairs : {74, 66, 0}) {
                const int64_t N = nk[0], K = nk[1];
                const int nrp = (int)((N + 31) / 32), nchunks = (int)((K + 63) / 64 + 3) / 4 * 4;
                const int pieces = q4_umma_plan(nrp, nchunks, sms).pieces;
                for (int64_t M : {17, 64, 65, 100, 257, 512, 700, 2100}) {
                    const Q4Needs n = q4_needs(N, K, nrp, nchunks, M, 1000, pieces, 17, 65, pairs);
                    bad += n.partial < 1000;                                    // what 2..16 rows want
                    for (int64_t m = 17; m <= M; ++m) {                         // no smaller call, by either kernel, wants more
                        const int u = (int)(m < 64 ? m : 64);
                        bad += q4_umma_need_xs(nchunks, u) > n.xs || q4_umma_need_partial(pieces, u, N) > n.partial;
                        if (m < 65 || !pairs) continue;
                        const Q4GemmPlan pl = q4_gemm_plan(nrp, nchunks, (int)std::min<int64_t>(m, q4_gemm_slab(K)), pairs);
                        bad += pl.need_xs > n.xs || pl.need_partial > n.partial;
                    }
                }
            }
    // the shapes whose 64 rows want more partial sums than 512 rows
    const int64_t wide[][3] = {{57344, 8192, 44040192}, {128256, 4096, 65667072}};
    for (auto& s : wide) {
        const int nrp = (int)(s[0] / 32), nchunks = (int)(s[1] / 64), pieces = q4_umma_plan(nrp, nchunks, 148).pieces;
        bad += q4_umma_need_partial(pieces, 64, s[0]) != (size_t)s[2] || q4_gemm_plan(nrp, nchunks, 512, 74).need_partial >= (size_t)s[2];
        bad += q4_needs(s[0], s[1], nrp, nchunks, 512, 0, pieces, 17, 65, 74).partial < (size_t)s[2];
    }
    // two slabs of 64 rows instead of tiles: up to 96 rows of a large weight, up to 128 of a very large one
    const int64_t route[][3] = {{196607, 65, 0}, {196608, 65, 1}, {196608, 96, 1}, {196608, 97, 0}, {262143, 97, 0}, {262144, 97, 1}, {262144, 128, 1},
                                {262144, 129, 0}, {1 << 30, 129, 0}, {1, 64, 1}, {1, 65, 0}, {256512, 96, 1}, {256512, 128, 0}};
    for (auto& r : route) bad += q4_slabs_of_64(r[0], r[1]) != (r[2] != 0);
    // few rows of x go to kernels with needs of their own
    bad += q4_needs(4096, 4096, 128, 64, 16, 77, 2, 17, 65, 74).xs != 0 || q4_needs(4096, 4096, 128, 64, 16, 77, 2, 17, 65, 74).partial != 77;
    bad += q4_needs(4096, 4096, 128, 64, 300, 77, 2, 0, 65, 74).xs != 0;
    std::printf("%d\n", bad);
    return bad;
}
"""


TILES = r"""
#include "q4_plan.h"
#include <cstdio>
using namespace mpq;
int main()
{
    int bad = 0;
    for (int nrp : {1, 7, 8, 9, 128, 625, 688, 1792, 4008})
        for (int nchunks : {4, 36, 64, 448})
            for (int M : {1, 64, 65, 80, 128, 129, 512, 2048})
                for (int pairs : {74, 66, 1}) {
                    const Q4GemmPlan p = q4_gemm_plan(nrp, nchunks, M, pairs);
                    const int64_t tiles = (int64_t)((nrp + 7) / 8) * p.nt, rest = (int64_t)p.rest * nchunks;
                    bad += p.Mt % 16 || p.Mt < 32 || p.Mt > Q4G_MT_MAX || (int64_t)p.nt * p.Mt < M;        // every row in a tile
                    bad += (int64_t)p.full * 2 * pairs + p.rest != tiles || p.rest >= 2 * pairs;           // every tile, whole or left over
                    bad += p.grid < 1 || p.grid > 2 * pairs || p.ranges > p.grid || (p.full && p.grid != 2 * pairs);
                    bad += (int64_t)p.ranges * p.W < rest || (p.ranges && (int64_t)(p.ranges - 1) * p.W >= rest) || p.W > nchunks;   // a range: two tiles at most
                    bad += p.need_partial != (p.cut ? (size_t)p.ranges * 2 * Q4G_SLOT * 4 : 0);
                }
    std::printf("%d\n", bad);
    return bad;
}
"""


def test_tiles_above_64_rows_cover_the_call():
    """Whole tiles and ranges of the tiles that are left over: all of them, none twice, no range over more than two tiles."""
    _run(TILES)


WALK = r"""
#include "q4_plan.h"
#include <cstdio>
#include <cstdlib>
#include <vector>
using namespace mpq;
struct Piece { int tile, c0, n, slot; };               // slot: -1 = straight to y, else the slot that the kernel writes
int main()
{
    int bad = 0, both = 0;
    for (int nrp : {1, 9, 128, 625, 938, 1792})
        for (int nchunks : {4, 8, 20, 36})
            for (int M : {65, 129, 300, 512})
                for (int pairs : {74, 66, 1}) {
                    const Q4GemmPlan p = q4_gemm_plan(nrp, nchunks, M, pairs);
                    const int tiles = p.full * p.grid + p.rest;
                    both += p.full && p.cut;
                    std::vector<int> seen((size_t)tiles * nchunks, 0);
                    std::vector<std::vector<Piece>> pieces(tiles);
                    for (int block = 0; block < p.grid; ++block) {
                        Q4GWalk w(block, p.grid, p.full, p.rest, p.W, nchunks), k = w;      // copies and MMAs; workers, piece by piece
                        while (k.left) {
                            const int n = k.rest_left ? std::min(k.rest_left, nchunks - k.c) : nchunks;
                            const bool whole = k.c == 0 && n == nchunks;
                            const int at = k.tile != p.full * p.grid + q4g_first_tile(block, p.W, nchunks);
                            if (k.tile < 0 || k.tile >= tiles || n < 1) return 1;
                            pieces[k.tile].push_back({k.tile, k.c, n, whole ? -1 : block * 2 + at});
                            for (int i = 0; i < n; ++i) {
                                bad += w.tile != k.tile || w.c != k.c + i || w.left != k.left - i;      // the same walk
                                ++seen[(size_t)w.tile * nchunks + w.c];
                                w.next(nchunks, block, p.grid);
                            }
                            k.skip(n, nchunks, block, p.grid);
                        }
                        bad += w.left != 0;
                    }
                    for (int s : seen) bad += s != 1;                                       // every chunk of every tile once
                    for (int t = 0; t < tiles; ++t) {
                        if (t < p.full * p.grid) { bad += pieces[t].size() != 1 || pieces[t][0].slot != -1; continue; }
                        const int cut = t - p.full * p.grid;                                // the sum reads, in order, what was written
                        int pf, pl;
                        q4u_pieces(cut, nchunks, p.W, &pf, &pl);
                        bad += (int)pieces[t].size() != pl - pf + 1;
                        if (pf == pl) { bad += pieces[t][0].slot != -1; continue; }
                        const bool second = cut != q4g_first_tile(pf, p.W, nchunks);
                        int c = 0;
                        for (int s = pf; s <= pl && s - pf < (int)pieces[t].size(); ++s) {
                            const Piece& q = pieces[t][s - pf];
                            bad += q.slot != s * 2 + (s == pf && second) || q.c0 != c;
                            c += q.n;
                        }
                        bad += c != nchunks;
                    }
                }
    bad += both < 20;                                                                       // the form of long prompts is among them
    std::printf("%d\n", bad);
    return bad != 0;
}
"""


def test_the_walk_over_tiles_above_64_rows_visits_every_chunk_once():
    """Cut ranges first, then whole tiles: copies, MMAs and workers walk alike, no chunk is left out or taken twice, and the sum of a cut
    tile reads the slots that its pieces were written to."""
    _run(WALK)


def test_scratch_reserved_for_a_call_is_enough_for_every_smaller_one():
    _run(NEEDS)


UPLOAD = r"""
#include "upload.h"
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
static const char *locked_lo = nullptr, *locked_hi = nullptr;              // what the fake driver has page-locked
static bool refuse_direct = false, refuse_pinned = false;
static int direct = 0, staged = 0, left_behind = 0;
static bool writer_done = true;                                            // a copy that fills the array may still be on its way
extern "C" {
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p)
{
    a->type = p >= locked_lo && p < locked_hi ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    if (!writer_done) return cudaErrorUnknown;                             // too early
    memcpy(d, s, n);
    ++staged;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind)
{
    if (refuse_direct) { left_behind = 1; return cudaErrorInvalidValue; }
    writer_done = true;                                                    // it waits for what precedes it
    memcpy(d, s, n);
    ++direct;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { writer_done = true; return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
    if (refuse_pinned) { left_behind = 1; return cudaErrorMemoryAllocation; }
    *p = malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { left_behind = 0; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
}
static int upload(mpq::StagedUpload& u, const std::vector<char>& from, size_t off, size_t n)
{
    std::vector<char> to(n + 1, 7);
    cudaError_t e = cudaErrorUnknown;
    direct = staged = 0;
    const bool ok = u.run(to.data(), from.data() + off, -1, 0, n, nullptr, &e) == mpq::StagedUpload::OK && e == cudaSuccess;
    return !ok || memcmp(to.data(), from.data() + off, n) || to[n] != 7 || left_behind;
}
int main()
{
    int bad = 0;
    std::vector<char> from(5 * mpq::StagedUpload::PIECE + 123);
    for (size_t i = 0; i < from.size(); ++i) from[i] = (char)(i * 2654435761u >> 13);
    const char *src_lo = from.data(), *src_hi = src_lo + from.size();
    const size_t n = from.size();
    mpq::StagedUpload u;
    bad += upload(u, from, 0, n) || direct != 0 || staged != 6;            // pageable: piece by piece through the slots
    bad += upload(u, from, 5, 1) || staged != 1;
    locked_lo = src_lo, locked_hi = src_hi, writer_done = false;
    bad += upload(u, from, 0, n) || direct != 1 || staged != 0;            // page-locked: one copy of it all
    bad += upload(u, from, 777, n - 777) || direct != 1;                   // and a part of it
    locked_hi = src_lo + n / 2, writer_done = false;
    bad += upload(u, from, 0, n) || direct != 0 || staged != 6;            // page-locked in part: through the slots
    locked_hi = src_hi, refuse_direct = true, writer_done = false;
    bad += upload(u, from, 0, n) || direct != 0 || staged != 6;            // a copy that the driver refuses: through the slots
    u.release();
EXTRA
    std::printf("%d\n", bad);
    return bad;
}
"""


def test_page_locked_arrays_are_uploaded_without_a_copy_on_the_host():
    _run(UPLOAD.replace("EXTRA", ""))


def test_uploads_work_where_no_pages_can_be_locked():
    _run(UPLOAD.replace("EXTRA", """
    locked_lo = locked_hi = nullptr, refuse_direct = false, refuse_pinned = true;
    mpq::StagedUpload v;
    bad += upload(v, from, 0, n) || staged != 6;
    refuse_pinned = false;
    bad += upload(v, from, 3, n - 3) || staged != 6;
    v.release();
    bad += upload(v, from, 0, n) || staged != 6;
    v.release();
"""))


PAGES = r"""
#include "host_pages.h"
#include <cstdio>
#include <cstdlib>
static int locked = 0, live = 0;
static bool refuse = false;
extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
    if (refuse) return cudaErrorMemoryAllocation;
    ++locked, ++live;
    *p = malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { --live; free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}
int main()
{
    int bad = 0;
    mpq::HostPages pages;
    const size_t most = mpq::HostPages::MOST_OUT;
    for (size_t n = 16; n <= most; n += 4096) bad += !pages.reserve(n, most) || pages.bytes < n || pages.bytes > most || live != 1;
    bad += locked > 6;                                                     // rows that grow by a page a call: 64 KB, 128 KB ... 1 MB
    bad += pages.reserve(most + 16, most) || !pages.reserve(most, most);
    bad += mpq::HostPages::MOST_IN > 524288 || mpq::HostPages::MOST_OUT_BEHIND_COPY > 786432;
    pages.release();
    refuse = true;
    bad += pages.reserve(16, most) || pages.bytes || live;
    std::printf("%d\n", bad);
    return bad;
}
"""


def test_pages_for_host_rows_grow_in_doubling_steps():
    _run(PAGES)


FP4 = r"""
#include "nvfp4_plan.h"
#include <cstdio>
using namespace mpq;
static bool rows(int M, int64_t N, int64_t K) { return nvfp4_rows_pay(rows_plan(M, N, K, 148, 0), pair_plan(M, N, K, 74), M); }
int main()
{
    int bad = 0;
    // one CTA more than a full wave, K too short for 64 rows, and their neighbours, as measured
    bad += rows(64, 33264, 2048) || !rows(64, 33152, 2048) || rows(64, 33264, 14336) || !rows(64, 28672, 4096) || !rows(64, 57344, 4096);
    bad += rows(64, 8192, 2048) || rows(64, 14336, 4096) || !rows(64, 4096, 4096) || !rows(64, 4096, 14336) || !rows(48, 14336, 4096);
    for (int64_t N = 8; N < 200000; N += 8 * 61)
        for (int64_t K = 32; K < 60000; K += 32 * 37)
            for (int M : {1, 16, 17, 32, 33, 64}) {
                const RowsPlan r = rows_plan(M, N, K, 148, 0);
                const PairPlan p = pair_plan(M, N, K, 74);
                bad += M <= 32 && !rows(M, N, K);
                bad += r.splits < 1 || (r.splits > 1 && (r.tiles * r.splits > 296 || r.k_blocks / r.splits < SPLIT_MIN_BLOCKS));
                bad += r.tiles * 96 > N + 224 || r.tiles * 128 < N || r.Mp % 16 || r.Mp < M;
                bad += rows_partial_bytes(r) > (size_t)74 * 256 * BN * 4 && r.splits > 1;          // the room that is reserved
                bad += p.splits < 1 || p.last * p.splits > 74 || (p.splits > 1 && p.k_blocks / p.splits < SPLIT_MIN_BLOCKS);
                bad += !(r.cost > 0) || !(p.cost > 0);
                const RowsPlan cut = rows_plan(M, N, K, 148, 3);
                bad += cut.splits != (r.k_blocks >= 6 ? 3 : r.k_blocks >= 4 ? 2 : 1);
            }
    std::printf("%d\n", bad);
    return bad;
}
"""


def test_few_nvfp4_rows_go_to_the_kernel_that_is_faster():
    _run(FP4)


def test_every_kernel_that_can_give_up_a_wait_settles_before_it_ends():
    """A kernel whose roles share an abort flag waits for what was in flight behind its last CTA barrier, before tensor memory is freed."""
    kernels = 0
    for f in ("q4_umma.cuh", "q4_gemm.cuh", "nvfp4_gemm.cu", "nvfp4_rows.cuh"):
        text = open(os.path.join(ROOT, "makepad_b200", "csrc", f)).read()
        for body in text.split("volatile int s_abort;")[1:]:
            kernels += 1
            end = body[:body.index("tcgen05.dealloc")]
            assert "settle_after_timeout(s_abort);" in end[end.rindex("__syncthreads();"):], f
    assert kernels == 5


def test_no_cta_of_a_cluster_leaves_while_another_may_still_store_into_it():
    """q4_rect_kernel: every CTA arrives at a cluster barrier behind its last remote store, and waits for the others there before it leaves,
    whether its own wait for the slices ran out or not; what was on its way then lands before it ends."""
    text = open(os.path.join(ROOT, "makepad_b200", "csrc", "q4_rect.cuh")).read()
    kernel = text[text.index("q4_rect_kernel(const __grid_constant__"):]
    kernel = kernel[:kernel.index("\n}")]
    last_put = kernel.rindex("put(")
    end = kernel[last_put:]
    arrive, sums, wait, settle = (end.index(t) for t in ("barrier.cluster.arrive.relaxed", "mbar_wait(sent_u32, 0,", "barrier.cluster.wait", "settle_after_timeout(!arrived)"))
    assert arrive < sums < wait < settle
    assert "return" not in kernel[kernel.index("barrier.cluster.arrive"):].replace("if (m >= p.M) return;", "")


def test_what_an_earlier_kernel_writes_is_read_by_ordinary_loads():
    """Kernels that start beside the one in front of them read its output behind griddepcontrol.wait, where only ordinary loads see it: no
    __ldg, no load that the compiler may move (pdl.cuh has those for data read once), no const __restrict__ pointer to it."""
    csrc = os.path.join(ROOT, "makepad_b200", "csrc")
    kernels = 0
    for f in sorted(os.listdir(csrc)):
        if not f.endswith((".cu", ".cuh")):
            continue
        for kernel in re.split(r"(?=__global__ )", open(os.path.join(csrc, f)).read())[1:]:
            kernel = kernel[:kernel.index("\n}")]
            if "griddepcontrol.wait" in kernel:
                kernels += 1
                assert not re.search(r"__ld(g|cs|cg|ca|lu)\(", kernel), (f, kernel[:120])
                assert not re.search(r"const \w+\* __restrict__", kernel[:kernel.index("{")]), (f, kernel[:120])
    assert kernels == 15, kernels
    rows = open(os.path.join(csrc, "nvfp4_rows.cuh")).read()               # (and in the helper of one of them)
    assert not re.search(r"__ld(g|cs)\(", rows)


def test_every_bounded_wait_has_a_code_of_its_own():
    """mpq_context_poll_status reports a word and a code: the code names the wait that ran out."""
    csrc = os.path.join(ROOT, "makepad_b200", "csrc")
    codes = []
    for f in os.listdir(csrc):
        if f.endswith((".cu", ".cuh")):
            text = open(os.path.join(csrc, f)).read()
            codes += re.findall(r"atomicExch\((?:p\.)?status, (\d+)\)", text)
            codes += set(re.findall(r"\bfail = ([1-9]\d*);", text))           # (a role with several waits for the same thing)
    assert len(codes) > 25 and len(codes) == len(set(codes)), sorted(codes, key=int)


def test_waits_for_staged_rows_begin_behind_the_kernels_before():
    """In the Q4 tcgen05 kernels the issuing warp and the workers wait for the kernels before (griddepcontrol.wait) ahead of their first
    bounded wait for what depends on the staged activations."""
    for f in ("q4_umma.cuh", "q4_gemm.cuh"):
        text = open(os.path.join(ROOT, "makepad_b200", "csrc", f)).read()
        issue = text[text.index("// ---------------- MMA issue"):]
        assert "griddepcontrol.wait" in issue[:issue.index("q4u_bar_poll<0>(")], f
        work = text[text.index("// ---------------- expansion + drain"):]
        first = work.index("df, dph)" if f == "q4_umma.cuh" else "q4u_bar_wait(df + 8, dph)")
        assert "griddepcontrol.wait" in work[:first], f


def test_waits_of_a_warp_on_several_barriers_order_memory():
    """A vote over the lanes' barriers orders no memory: where lanes look at different ones, a __syncwarp stands between the vote and
    whatever reads what was waited for, and no kernel votes on barriers in any other way."""
    csrc = os.path.join(ROOT, "makepad_b200", "csrc")
    text = open(os.path.join(csrc, "q4_umma.cuh")).read()
    for name in ("bool q4u_bar_wait(", "bool q4u_bar_look("):
        body = text[text.index(name):]
        body = body[:body.index("\n}")]
        vote = max(body.rfind("vote.sync"), body.rfind("_sync("))
        assert "__syncwarp();" in body[vote:] and "return" not in body[vote:body.index("__syncwarp();")], name
    poll = text[text.index("bool q4u_bar_poll("):]
    assert "q4u_bar_look(" in poll[:poll.index("\n}")]
    votes = [m for f in ("q4_umma.cuh", "q4_gemm.cuh") for m in re.findall(r"_sync\([^;]*q4u_bar_test", open(os.path.join(csrc, f)).read())]
    assert len(votes) == 1, votes                                      # the one of q4u_bar_look


ROUTES = r"""
#include "q4_plan.h"
#include <cstdio>
using namespace mpq;
int main()
{
    int bad = 0;
    for (int64_t units : {1, 196608, 262144})
        for (int64_t M = 1; M <= 2100; ++M) {
            bad += q4_route(units, M, 17, 65, false) != Q4Route::Slabs16;                              // no tensor map: every call still has a kernel
            bad += q4_route(units, M, 0, 65, true) != Q4Route::Slabs16;
            bad += q4_route(units, M, 17, 65, true) != (M < 17 ? Q4Route::Slabs16 : q4_slabs_of_64(units, M) ? Q4Route::Slabs64 : Q4Route::Tiles);
            bad += q4_route(units, M, 17, 0, true) != (M < 17 ? Q4Route::Slabs16 : Q4Route::Slabs64);
        }
    // ... and no scratch of kernels that it does not reach
    bad += q4_needs(4096, 4096, 128, 64, 300, 77, 2, q4_umma_from(17, false), 65, 0).xs != 0;
    std::printf("%d\n", bad);
    return bad;
}
"""


def test_a_weight_without_a_tensor_map_is_not_refused():
    """The tcgen05 kernels read weights through a tensor map of the driver's; where it made none, calls of 17 rows and more run as slabs of
    16 rows (as with MPQ_Q4_UMMA_MIN=0), and no call returns an error for the map's sake."""
    _run(ROUTES)
    text = open(os.path.join(ROOT, "makepad_b200", "csrc", "mpq.cu")).read()
    assert not re.search(r"!q\.mapped\) return fail", text)
    assert not re.search(r"ctx->q4_umma_min (>|<|>=|<=) ", text)          # routes go through q4_route, which knows of the map


def test_a_timeline_of_kernels_that_are_not_stamped_is_refused():
    """The diagnostic library returns no array when nothing was stamped: a message then, not a read of address zero."""
    import ctypes as C
    import numpy as np
    import pytest
    from makepad_b200 import timeline
    stamps = np.arange(64 * 1024 * 16, dtype=np.uint64)

    class Debug:                                                       # stands for the library's mpq_debug_trace
        def __init__(self, ptr, launches):
            self.ptr, self.launches = ptr, launches

        def __call__(self, count):
            C.cast(count, C.POINTER(C.c_int32))[0] = self.launches
            return self.ptr

    class Lib:
        def __init__(self, ptr, launches):
            self.mpq_debug_trace = Debug(ptr, launches)

    with pytest.raises(RuntimeError, match="0 of 24 launches"):
        timeline.read_trace(Lib(None, 0), 24)
    with pytest.raises(RuntimeError, match="18 of 24 launches"):       # some projections of a layer stream, others do not
        timeline.read_trace(Lib(stamps.ctypes.data, 18), 24)
    assert (timeline.read_trace(Lib(stamps.ctypes.data, 24), 24).ravel() == stamps).all()


def test_the_tcgen05_kernels_are_stamped_in_the_diagnostic_build():
    """What the timeline names, the kernels stamp: phases 0..7 in each, and their launches pass the array."""
    csrc = os.path.join(ROOT, "makepad_b200", "csrc")
    for f in ("q4_umma.cuh", "q4_gemm.cuh"):
        text = open(os.path.join(csrc, f)).read()
        assert sorted(re.findall(r"Q4U_TRACE\((\d),", text)) == list("01234567"), f
    assert open(os.path.join(csrc, "mpq.cu")).read().count("p.trace = trace_slot(") == 3
