#pragma once
// Launch shapes of the resident BiCGStab (resident.cuh, resident_two.cuh): which
// form takes a system, with how many CTAs and threads and how much shared
// memory; and which systems the resident GMRES takes.  Host code without CUDA, so that the rules are tested on the CPU.
#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace mhfem {

// Launch bounds of the kernels: threads of a CTA at most.
constexpr int kMaxThreads = 512;   // three reductions, streamed
constexpr int kPassThreads = 384;  // two reductions; elsewhere the most for a CTA whose rows are few (group_threads)
constexpr int kSums = 4;           // sums of the widest reduction
constexpr int kMaxCluster = 16;

// Rows up to which one cluster takes the system: its barrier costs half of the
// grid's, its 16 SMs have a tenth of the FP64 units.  Measured per iteration,
// cluster and grid: 6.5 and 8.7 us at 800 rows (width 4), 7.8 and 8.8 at 3,960,
// 8.6 and 8.6 at 5,376, 10.6 and 8.7 at 7,905; 9.1 and 10.6 at 2,480 (width 9),
// 12.0 and 10.9 at 5,520.
constexpr int64_t kClusterRows = 4096;
// Off-diagonal entries up to which phase B of the FP64 solve forms the
// neighbours' s itself: a barrier less against one FP64 operation per entry.
// Measured per iteration, with and without: 14.97 and 15.84 us at 0.30M
// entries (50,688 rows, width 6), 18.5 and 19.0 at 0.68M, 20.6 and 21.0 at
// 0.79M (width 4), but 22.3 and 21.4 at 1.22M (width 9), 27.1 and 26.4 at
// 1.44M.  In FP32 the operation costs nothing: always.
constexpr int64_t kRecompEntries = 1000000;

// Off-diagonal entries up to which the FP64 solve runs with two reductions
// per iteration (resident_two.cuh).  Measured per iteration against three:
// 8.6 and 10.1 us at 50,000 entries (width 4), 11.7 and 12.8 at 304,000 (width
// 6), 13.7 and 14.5 at 432,000, 15.4 and 15.4 at 537,000, but 17.0 and 16.4 at
// 683,000, 16.9 and 15.8 at 682,000 (width 10).  In FP32 wherever it fits (12.6
// and 14.7 at 788,000).
constexpr int64_t kTwoEntries = 500000;

// Matrix bytes up to which the ELL words are streamed from L2 by one CTA per
// SM (129 MB of L2 also holds the gathered vectors and x).  Measured per
// iteration against the five kernels: 48.7 and 57.3 us at 44 MB (width 6),
// 55.0 and 64.6 at 56 MB, 45.9 and 64.7 at 64 MB (width 10), but 77.0 and
// 72.9 at 84 MB (width 9), 80.4 and 76.0 at 87 MB (width 10).
// In FP32 (with half the vectors' bytes) 42.8 and 56.4 us at 73 MB.
constexpr int64_t kStreamedBytes = (int64_t)72 << 20;

// Threads of a CTA with `rc` rows: as few passes over them as `most` threads
// allow, of equal size, whole warps, and at least one warp per FP64 unit.  A
// thread more is a value more in every block sum, a pass more another round of
// gather latency.  Measured per iteration: 326 rows 12.4 us with 352 threads
// (one pass), 13.8 with 192, 14.0 with 256; 793 rows 15.8 with 288 (three),
// 17.2 with 512, 19.1 with 256; 1,115 rows 18.8 with 384, 20.1 with 512; above
// 4,096 rows the streamed ELL words want 512 threads (46.7 us against 49.3 with
// 384 at 5,116 rows, 25.2 and 27.2 in FP32).
inline int group_threads(int rc, int most)
{
    if (rc > 4096) return kMaxThreads;
    const int passes = (rc + most - 1) / most, per = (rc + passes - 1) / passes;
    return std::max(128, (per + 31) / 32 * 32);
}

// Rows up to which every FP64 system runs resident, whatever its width, and
// tests its convergence in every iteration: MHFEM_NOALLOC_MAX_ROWS, the size up
// to which mhfem_bicgstab_noalloc promises both.  The test costs the streamed
// forms 1.0 to 1.5 us per iteration there (227,556 rows of width 10 24.9 ->
// 25.9 us, 262,144 of width 13 29.1 -> 30.6).  The ELL words of the widest
// systems exceed kStreamedBytes: 45.1 us per iteration against the five
// kernels' 123.5 at 262,144 rows of width 25, 98.3 against 175.7 at width 40.
constexpr int64_t kEveryTestRows = (int64_t)1 << 18;

// Iterations between the convergence tests of the streamed forms above
// kEveryTestRows (a power of two).  There the FP64 pipe bounds the vector
// phases, and the two sums over r are two of 26 operations per row; a solve
// takes hundreds of iterations.
constexpr int kStreamedCheckEvery = 4;

// Shared memory left for the kernels' static variables: the cluster's slots
// take 2 KB of the two-reduction form's.
constexpr size_t kStaticTwo = 4096, kStaticThree = 2048;

struct ResidentPlan {
    bool ok = false, cluster = false, mats = false, recomp = false, x_in_smem = false;
    bool two = false;  // resident_two.cuh
    int check_every = 1;
    int ctas = 0, threads = 0, rc = 0;
    size_t smem = 0;
};

inline ResidentPlan plan_resident(int64_t rows, int width, size_t real, int sms, size_t smem_max)
{
    ResidentPlan P;
    if (rows < 1) return P;
    auto fill = [&](int ctas) {
        P.ctas = ctas;
        P.rc = (int)((rows + ctas - 1) / ctas);
        P.ctas = (int)((rows + P.rc - 1) / P.rc);  // no empty CTA
        P.threads = std::min(group_threads(P.rc, kPassThreads), P.two ? kPassThreads : kMaxThreads);
        const size_t vectors = 5 + (P.recomp ? 1 : 0) + (P.x_in_smem ? 1 : 0);
        P.smem = sizeof(double) * (size_t)kSums * P.threads + real * vectors * P.rc +
                 (P.two    ? (real * (1 + 4 * (size_t)width) + sizeof(int32_t) * width) * P.rc
                  : P.mats ? (real + sizeof(int32_t)) * (size_t)width * P.rc
                           : 0);
        return P.smem + (P.two ? kStaticTwo : kStaticThree) <= smem_max;
    };
    const int64_t want = (rows + 127) / 128;
    const int ctas = (int)std::min<int64_t>(want, sms);
    if (real == 4 || rows * width <= kTwoEntries) {
        // two reductions per iteration, in a cluster or the grid
        for (bool cluster : {true, false}) {
            if (cluster && rows > kClusterRows) continue;
            P = ResidentPlan{};
            P.two = P.x_in_smem = true;
            P.cluster = cluster;
            int c = 1;
            while (c < kMaxCluster && (int64_t)c * 128 < rows) c *= 2;
            P.ok = fill(cluster ? c : ctas);
            if (cluster) P.ctas = c;  // every CTA of the cluster is launched, also those left without rows
            if (P.ok) return P;
        }
    }
    const bool every = real == 8 && rows <= kEveryTestRows;
    for (int form = 0; form < 3; ++form) {  // ELL words and x in shared memory, x only, neither
        if (form > 0 && !every && (int64_t)(real + 4) * width * rows > kStreamedBytes) return ResidentPlan{};
        P = ResidentPlan{};
        P.check_every = form == 0 || every ? 1 : kStreamedCheckEvery;
        P.mats = form == 0;
        P.recomp = P.mats && (real == 4 || rows * width <= kRecompEntries);
        P.x_in_smem = form < 2;
        P.ok = fill(ctas);
        if (P.ok) return P;
    }
    return P;
}

// Whether restarted GMRES runs resident (k_gmres_resident.cu).  Above about
// 90,000 rows the basis and the ELL words are read from memory, by one CTA per
// SM against up to eight of k_gmres.cu's kernels, so the route follows the bytes
// of the matrix and of a part of the basis.  Measured per iteration, resident
// and two kernels, with restart length 5 and 30 (in brackets rows x (12 width +
// 100) in millions):
//   288,920 rows, width  4  (43): 20.3 and 45.3 us, 39.6 and 81.9
//   287,712 rows, width 21 (101): 49.1 and 76.0, 74.7 and 107.6
//   766,085 rows, width  4 (113): 48.4 and 64.1, 131.4 and 134.7
//   720,954 rows, width  6 (124): 49.9 and 67.4, 128.8 and 135.2
//   694,960 rows, width  9 (145): 62.5 and 73.9, 133.3 and 140.0
//   595,428 rows, width 13 (152): 71.3 and 74.5, 122.4 and 129.4
//   but 455,112, width 21 (160): 102.2 and 88.4, 130.0 and 130.2
//   779,040 rows, width  9 (162): 77.4 and 76.0, 153.9 and 146.3
//   726,516 rows, width 13 (186): 87.6 and 84.7, 149.3 and 145.0
//   677,376 rows, width 21 (238): 150.4 and 96.6, 198.7 and 157.3
// Up to 2^18 rows always: only a width above 40 would exceed the line there.
inline bool gmres_resident_fits(int64_t rows, int width)
{
    if (rows <= ((int64_t)1 << 18)) return true;
    return rows <= ((int64_t)3 << 18) && rows * (12 * (int64_t)width + 100) <= 155000000;
}

}  // namespace mhfem
