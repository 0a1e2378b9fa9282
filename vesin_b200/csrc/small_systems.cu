// Batches of independent small systems. Two passes (count, emit) so that every
// system owns one contiguous, exactly sized block of the output. Two kernels:
//   * molecules (no periodic direction, at most 96 points): a WARP per system,
//     two systems per CTA;
//   * everything else (periodic systems, up to 2048 points): one or more CTAs
//     per system, which list the periodic images that can reach a tile of home
//     points and stage them a batch at a time.
// Both decide like the pair kernel of large systems: a lane per home point,
// candidates broadcast from shared memory four at a time, an fp32 screen on
// coordinates relative to a point of the system (two candidates per packed
// instruction) that leaves one hit bit per candidate, and the exact fp64
// predicate inside the error band. Hits gather in a per-warp list and leave 32
// at a time through the coalesced stores of the large-system kernels. Walking
// the (i, j) of the flattened triangle instead, a square root and a few
// corrections per candidate, the 16 384 molecules of 16 to 64 atoms (float, 5.3 M
// pairs) took 64 us to count and 120 us to write; now 18 and 54 (the 230 MB of the
// list take 35 us at the copy bandwidth: half the time is the chain of a warp,
// points -> decisions -> list -> stores).
//
// Replaces, for this use, the per-system loop of the callers
// (python/vesin/vesin/metatomic/_neighbors.py:197-199) and the brute-force
// kernels of the reference (vesin/src/cuda/bruteforce.cu:241-573), which keep
// one image per pair and therefore need cutoff <= half the smallest face
// distance; here the number of images per direction follows from the box.
#include "kernels.cuh"

#include "emit.cuh"
#include "plan.hpp"

#include <algorithm>
#include <type_traits>

namespace vb200 {

namespace {

constexpr int SMALL_THREADS = 128;
constexpr int SMALL_WARPS = SMALL_THREADS / 32;
// per SM (72 registers, and 8 to 28 bytes of spills when pairs are written; 512 cells, both passes: 6 132 us, 7 131, 8 132)
constexpr int SMALL_CTAS = 7;
constexpr unsigned FULL_MASK = 0xffffffffu;

struct SystemFrame {
    double H[3][3];    // box, rows of non-periodic directions replaced by unit vectors
    double Hinv[3][3];
    double reach[3];   // fractional distance within which points can be neighbors
    int periodic[3];
    int singular;
};

__device__ __forceinline__ void cross3(const double a[3], const double b[3], double out[3]) {
    out[0] = a[1] * b[2] - a[2] * b[1];
    out[1] = a[2] * b[0] - a[0] * b[2];
    out[2] = a[0] * b[1] - a[1] * b[0];
}

__device__ __forceinline__ void unit3(double v[3]) {
    double inv = 1.0 / sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    v[0] *= inv;
    v[1] *= inv;
    v[2] *= inv;
}

/// Same normalisation of the box as the host plan (and as the reference CPU
/// path, vesin/src/types.hpp:41-97): rows of non-periodic directions become
/// unit vectors orthogonal to the periodic ones.
__device__ void normalise_box(SystemFrame& frame, const BatchInput& in, unsigned system, const bool* periodic) {
    int n_periodic = 0, first = -1, second = -1;
    for (int i = 0; i < 3; i++) {
        for (int j = 0; j < 3; j++) {
            const size_t k = 9 * static_cast<size_t>(system) + 3 * i + j;
            frame.H[i][j] = (in.boxes == nullptr) ? 0.0 : (in.is_float ? static_cast<double>(static_cast<const float*>(in.boxes)[k]) : static_cast<const double*>(in.boxes)[k]);
        }
        frame.periodic[i] = (periodic != nullptr && periodic[i]) ? 1 : 0;
        if (frame.periodic[i]) {
            n_periodic++;
            if (first < 0) {
                first = i;
            } else if (second < 0) {
                second = i;
            }
        }
    }
    if (n_periodic == 0) {
        for (int i = 0; i < 3; i++) {
            for (int j = 0; j < 3; j++) {
                frame.H[i][j] = (i == j) ? 1.0 : 0.0;
            }
        }
    } else if (n_periodic == 1) {
        double a[3] = {frame.H[first][0], frame.H[first][1], frame.H[first][2]};
        double an[3] = {a[0], a[1], a[2]};
        unit3(an);
        double helper[3] = {0, 1, 0};
        if (fabs(an[1]) > 0.9) {
            helper[1] = 0;
            helper[2] = 1;
        }
        double c[3], b[3];
        cross3(a, helper, c);
        unit3(c);
        cross3(c, a, b);
        unit3(b);
        for (int k = 0; k < 3; k++) {
            frame.H[(first + 1) % 3][k] = b[k];
            frame.H[(first + 2) % 3][k] = c[k];
        }
    } else if (n_periodic == 2) {
        double c[3];
        cross3(frame.H[first], frame.H[second], c);
        unit3(c);
        for (int k = 0; k < 3; k++) {
            frame.H[3 - first - second][k] = c[k];
        }
    }
}

/// The frame of a system by one warp: the box by its first lane, the entries of the inverse by
/// nine lanes, the reach of the images by three. Ends with a __syncwarp().
__device__ void make_frame(SystemFrame& frame, const BatchInput& in, unsigned system, int lane) {
    if (lane == 0) {
        normalise_box(frame, in, system, in.periodic != nullptr ? in.periodic + 3 * static_cast<size_t>(system) : nullptr);
    }
    __syncwarp();
    const double (*m)[3] = frame.H;
    const double det = m[0][0] * (m[1][1] * m[2][2] - m[2][1] * m[1][2]) - m[0][1] * (m[1][0] * m[2][2] - m[1][2] * m[2][0]) +
                       m[0][2] * (m[1][0] * m[2][1] - m[1][1] * m[2][0]);
    const bool singular = !(fabs(det) >= 1e-30);
    if (lane < 9 && !singular) {
        const int r = lane / 3;
        const int c = lane % 3;
        const int r1 = (r + 1) % 3, r2 = (r + 2) % 3;
        const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
        frame.Hinv[r][c] = (m[c1][r1] * m[c2][r2] - m[c1][r2] * m[c2][r1]) / det;
    }
    __syncwarp();
    double images = 1.0;
    if (lane < 3 && !singular) {
        frame.reach[lane] = 0.0;
        if (frame.periodic[lane]) {
            // |fractional distance| * face distance <= |v| < cutoff
            const double (*inv)[3] = frame.Hinv;
            const double inv_face = sqrt(inv[0][lane] * inv[0][lane] + inv[1][lane] * inv[1][lane] + inv[2][lane] * inv[2][lane]);
            frame.reach[lane] = in.cutoff * inv_face * (1.0 + 1e-9);
            // images within cutoff / d + 1/2 of the nearest one, which is at most half a cell away
            images = 2.0 * fmin(floor(frame.reach[lane] + 0.5 + 1e-9), 1.0e6) + 1.0;
        } else {
            frame.reach[lane] = in.cutoff * (1.0 + 1e-9); // the row is a unit vector orthogonal to the others
        }
    }
    images *= __shfl_sync(FULL_MASK, images, 1) * __shfl_sync(FULL_MASK, images, 2);
    if (lane == 0) {
        // beyond the limit of images per pair the system is refused (2: "cutoff too large for the box")
        frame.singular = singular ? 1 : ((images > static_cast<double>(MAX_STENCIL_CELLS)) ? 2 : 0);
    }
    __syncwarp();
}

__device__ __forceinline__ bool half_rule_small(int s0, int s1, int s2) {
    // vesin/src/cpu_cell_list.cpp:107-132
    int sum = s0 + s1 + s2;
    if (sum < 0) {
        return false;
    }
    if (sum == 0 && (s2 < 0 || (s2 == 0 && s1 < 0))) {
        return false;
    }
    return true;
}

constexpr int MOLECULE_MAX_POINTS = 96;  // largest system the warp-per-system kernel takes
// A CTA is done when its largest system is: 16 384 molecules of 16 to 64 atoms, both passes, with 8
// systems per CTA 79 us, 4 75, 2 72 (1, where 32 CTAs fill an SM: 70, but 16 000 of 4 to 10 atoms 26 instead of 23)
constexpr int MOLECULE_WARPS = 2;

template <class Kind>
__device__ __forceinline__ double batch_coordinate(const BatchInput& in, size_t k) {
    // float -> double is exact: fp32 inputs are decided with the same fp64 arithmetic
    return Kind::FLOAT ? static_cast<double>(static_cast<const float*>(in.points)[k]) : static_cast<const double*>(in.points)[k];
}

/// Systems without a periodic direction and with few points go to the
/// warp-per-system kernel.
__device__ __forceinline__ bool taken_by_warp_kernel(const BatchInput& in, unsigned system, int n) {
    if (n > MOLECULE_MAX_POINTS) {
        return false;
    }
    if (in.periodic == nullptr) {
        return true;
    }
    const bool* periodic = in.periodic + 3 * static_cast<size_t>(system);
    return !(periodic[0] || periodic[1] || periodic[2]);
}

// ---- the fp32 screen -------------------------------------------------------

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long packed;
    asm("mov.b64 %0, {%1, %2};" : "=l"(packed) : "f"(lo), "f"(hi));
    return packed;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

/// Squared distances further than `half` from `mid` are decided by the screen.
struct ScreenBand {
    float mid, half;
};

/// The band for home points within `m` of the origin of the local frame. A candidate within the
/// cutoff of one of them is then within M = m + cutoff of it: the band covers the rounding of the
/// coordinates (relative error 2^-24 of values up to M), of the differences and of the sum. A
/// candidate further out is at more than the cutoff by more than its own rounding error, as long
/// as m is not thousands of times the cutoff; beyond that (or with m not finite) every candidate
/// goes to the exact predicate.
__device__ __forceinline__ ScreenBand everything_exact() {
    return ScreenBand{0.0f, __int_as_float(0x7f800000)};
}
__device__ __forceinline__ ScreenBand screen_band(float m, double cutoff_exact, double cutoff2_exact) {
    const float c = static_cast<float>(cutoff_exact) * 1.01f;
    const float M = (m + c) * 1.0001f;
    const float eps = 5.9604644775390625e-08f;
    float band = 4.0f * eps * (2.0f * 1.7320508f * c * (2.0f * M + c) + 3.0f * c * c) + 40.0f * eps * eps * M * M + 4.0f * eps * c * c;
    band *= 1.05f; // this expression is itself evaluated in fp32, and the sum starts from -mid
    const float cutoff2 = static_cast<float>(cutoff2_exact);
    if (!(m < 5.0e3f * c) || !(cutoff2 + band < 3.0e38f) || !(c > 1.0e-12f)) {
        return everything_exact();
    }
    return ScreenBand{cutoff2, band};
}

/// Decisions on candidates [0, 4 * quads) of a word for the home point whose negated coordinates are
/// (ax, ay, az), as far as `keep` has bits: the sign of d2 - mid, or exact(bit) for a candidate too
/// close to the cutoff for fp32 (the minimum over the word tells whether there is one). x, y, z:
/// 16-byte aligned arrays in shared memory, the same addresses for every lane.
template <class Exact>
__device__ __forceinline__ unsigned screen_word(
    const float* x, const float* y, const float* z, int quads, float ax, float ay, float az, const ScreenBand& band, unsigned keep, Exact exact
) {
    const unsigned long long ax2 = pack2(ax, ax), ay2 = pack2(ay, ay), az2 = pack2(az, az), mid2 = pack2(-band.mid, -band.mid);
    unsigned inside = 0;
    float closest = __int_as_float(0x7f800000);
#pragma unroll
    for (int k = 7; k >= 0; k--) {
        if (k >= quads) {
            continue;
        }
        const ulonglong2 x4 = reinterpret_cast<const ulonglong2*>(x)[k];
        const ulonglong2 y4 = reinterpret_cast<const ulonglong2*>(y)[k];
        const ulonglong2 z4 = reinterpret_cast<const ulonglong2*>(z)[k];
        const unsigned long long dx0 = add2(x4.x, ax2), dy0 = add2(y4.x, ay2), dz0 = add2(z4.x, az2);
        const unsigned long long dx1 = add2(x4.y, ax2), dy1 = add2(y4.y, ay2), dz1 = add2(z4.y, az2);
        const unsigned long long d0 = fma2(dx0, dx0, fma2(dy0, dy0, fma2(dz0, dz0, mid2)));
        const unsigned long long d1 = fma2(dx1, dx1, fma2(dy1, dy1, fma2(dz1, dz1, mid2)));
        float d2[4];
        asm("mov.b64 {%0, %1}, %2;" : "=f"(d2[0]), "=f"(d2[1]) : "l"(d0));
        asm("mov.b64 {%0, %1}, %2;" : "=f"(d2[2]), "=f"(d2[3]) : "l"(d1));
#pragma unroll
        for (int c = 3; c >= 0; c--) {
            inside = __funnelshift_l(__float_as_uint(d2[c]), inside, 1);
        }
        closest = fminf(closest, fminf(fabsf(d2[0]), fabsf(d2[1])));
        closest = fminf(closest, fminf(fabsf(d2[2]), fabsf(d2[3])));
    }
    if (!(closest > band.half)) {
#pragma unroll 1
        for (unsigned left = keep; left != 0; left &= left - 1) {
            const int b = __ffs(left) - 1;
            const float dx = x[b] + ax, dy = y[b] + ay, dz = z[b] + az;
            if (!(fabsf(fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, -band.mid)))) > band.half)) { // (NaN: the exact predicate decides)
                inside &= ~(1u << b);
                if (exact(b)) {
                    inside |= 1u << b;
                }
            }
        }
    }
    return inside & keep;
}

/// Bits `first` and above of a word.
__device__ __forceinline__ unsigned bits_from(int first) {
    return (first <= 0) ? 0xffffffffu : ((first >= 32) ? 0u : (0xffffffffu << first));
}

constexpr int HIT_WINDOW = 224;                // hits a warp lists at a time
constexpr int HIT_LIST = HIT_WINDOW + 32;      // ... behind fewer than 32 that wait for company

/// Lists the hits of a word (bit b of lane l -> entry + b) behind the `listed` entries that are
/// waiting, and hands them on in multiples of 32: write(n) writes entries [0, n) of the list.
/// Lanes hold different numbers of hits; their order is that of the lanes.
template <class Write>
__device__ __forceinline__ void list_hits(unsigned bits, unsigned entry, unsigned short* list, int& listed, int lane, Write write) {
    const int mine = __popc(bits);
    int position = mine;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
        const int up = __shfl_up_sync(FULL_MASK, position, offset);
        if (lane >= offset) {
            position += up;
        }
    }
    const int total = __shfl_sync(FULL_MASK, position, 31);
    position -= mine;
    for (int window = 0; window < total; window += HIT_WINDOW) {
        while (bits != 0 && position < window + HIT_WINDOW) {
            const int b = __ffs(bits) - 1;
            bits &= bits - 1;
            list[listed + position - window] = static_cast<unsigned short>(entry + b);
            position++;
        }
        listed += min(HIT_WINDOW, total - window);
        __syncwarp();
        const int whole = listed & ~31;
        if (whole != 0) {
            write(whole);
            listed -= whole;
            // what is left moves to the front of the list
            unsigned short moved = 0;
            if (lane < listed) {
                moved = list[whole + lane];
            }
            __syncwarp();
            if (lane < listed) {
                list[lane] = moved;
            }
            __syncwarp();
        }
    }
}

struct MoleculeShared {
    alignas(16) float fx[MOLECULE_WARPS][MOLECULE_MAX_POINTS]; // relative to the first point of the system
    alignas(16) float fy[MOLECULE_WARPS][MOLECULE_MAX_POINTS];
    alignas(16) float fz[MOLECULE_WARPS][MOLECULE_MAX_POINTS];
    double x[MOLECULE_WARPS][MOLECULE_MAX_POINTS]; // original positions
    double y[MOLECULE_WARPS][MOLECULE_MAX_POINTS];
    double z[MOLECULE_WARPS][MOLECULE_MAX_POINTS];
    alignas(16) double transpose[MOLECULE_WARPS][TRANSPOSE_DOUBLES];
    unsigned short list[MOLECULE_WARPS][HIT_LIST]; // hits waiting to be written: (i << 8) | j
};
static_assert(MOLECULE_MAX_POINTS % 32 == 0 && MOLECULE_MAX_POINTS <= 256, "whole words of candidates, indices of 8 bits");
static_assert(sizeof(MoleculeShared) <= SHARED_WITHOUT_ASKING, "no launch has to ask for its shared memory");

/// The reference's arithmetic for S = 0 (vesin/src/cpu_cell_list.cpp:135-138), operation for
/// operation: the shift term is an exact zero.
__device__ __forceinline__ double molecule_pair(const MoleculeShared& sh, int warp, int i, int j, double& vx, double& vy, double& vz) {
    vx = __dadd_rn(__dsub_rn(sh.x[warp][j], sh.x[warp][i]), 0.0);
    vy = __dadd_rn(__dsub_rn(sh.y[warp][j], sh.y[warp][i]), 0.0);
    vz = __dadd_rn(__dsub_rn(sh.z[warp][j], sh.z[warp][i]), 0.0);
    return __dadd_rn(__dadd_rn(__dmul_rn(vx, vx), __dmul_rn(vy, vy)), __dmul_rn(vz, vz));
}

/// What a launch of the batch kernels does is compiled in: counts or writes, full or half lists, points
/// and values in float or double, arrays that are aligned for paired stores. Looked at while the
/// kernels ran it took registers, which decide how many CTAs share an SM: both passes over 16 384
/// molecules 83 -> 79 us, over 512 cells 149 -> 131.
template <bool EMIT_, bool FULL_, bool FLOAT_, bool PAIRED_>
struct BatchKind {
    static constexpr bool EMIT = EMIT_;
    static constexpr bool FULL = FULL_;
    static constexpr bool FLOAT = FLOAT_;
    static constexpr int VALUES = FLOAT_ ? 1 : 0;
    static constexpr bool PAIRED = PAIRED_;
};

/// Writes the hits of up to 32 lanes from element `first` of the output on, both orientations
/// side by side for full lists.
template <class Kind>
__device__ __forceinline__ void write_hits(
    double* transpose, const PairOutput& out, int lane, unsigned long long first, int n_valid, unsigned long long gi,
    unsigned long long gj, int s0, int s1, int s2, double d, double vx, double vy, double vz, bool shifted
) {
    if (!Kind::FULL) {
        // half lists keep i <= j: the forward pair
        store_pairs<Kind::VALUES>(transpose, out, lane, first, n_valid, gi, gj, s0, s1, s2, d, vx, vy, vz, shifted);
    } else if (Kind::PAIRED) {
        store_both<Kind::VALUES>(transpose, out, lane, first, n_valid, gi, gj, s0, s1, s2, d, vx, vy, vz, shifted);
    } else {
        store_pairs<Kind::VALUES>(transpose, out, lane, first, n_valid, gi, gj, s0, s1, s2, d, vx, vy, vz, shifted);
        store_pairs<Kind::VALUES>(transpose, out, lane, first + n_valid, n_valid, gj, gi, -s0, -s1, -s2, d, -vx, -vy, -vz, shifted);
    }
}

constexpr int FRONT_THREADS = 256;

/// Header of a batch: nothing found yet. And the frames of the systems of the CTA kernel, a warp each:
/// the box, its inverse and the reach are a chain of divisions and roots that every CTA of both
/// passes went through before it did anything else (512 cells, both passes: 108.5 -> 98.4 us, and 1.8 here).
__global__ void __launch_bounds__(FRONT_THREADS) batch_front_kernel(const BatchInput in, SystemFrame* __restrict__ frames, DeviceHeader* header) {
    __shared__ SystemFrame sh_frames[FRONT_THREADS / 32];
    let_next_kernel_start();
    if (blockIdx.x == 0) {
        if (threadIdx.x < sizeof(DeviceHeader) / 4) {
            reinterpret_cast<unsigned*>(header)[threadIdx.x] = 0;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            header->first_bad = NO_BAD_POINT;
            header->mask_cursor = ~0ull; // first singular system
        }
    }
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const unsigned warps_in_grid = gridDim.x * (FRONT_THREADS / 32);
    for (unsigned system = blockIdx.x * (FRONT_THREADS / 32) + warp; frames != nullptr && system < in.n_systems; system += warps_in_grid) {
        const int n = static_cast<int>(in.offsets[system + 1] - in.offsets[system]);
        if (taken_by_warp_kernel(in, system, n)) {
            continue;
        }
        SystemFrame& frame = sh_frames[warp];
        make_frame(frame, in, system, lane);
        for (int k = lane; k < static_cast<int>(sizeof(SystemFrame) / 4); k += 32) {
            reinterpret_cast<unsigned*>(frames + system)[k] = reinterpret_cast<const unsigned*>(&frame)[k];
        }
        __syncwarp();
    }
}

template <class Kind>
__global__ void __launch_bounds__(MOLECULE_WARPS * 32, Kind::EMIT ? 16 : 20) molecules_kernel(
    const BatchInput in, unsigned long long* __restrict__ system_count, const unsigned long long* __restrict__ system_start, PairOutput out,
    DeviceHeader* header, const unsigned long long capacity, DeviceHeader* mirror
) {
    constexpr bool EMIT = Kind::EMIT;
    let_next_kernel_start();
    wait_for_previous_kernel();
    extern __shared__ __align__(16) unsigned char molecule_smem[];
    MoleculeShared& sh = *reinterpret_cast<MoleculeShared*>(molecule_smem);
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const unsigned warps_in_grid = gridDim.x * MOLECULE_WARPS;
    if (EMIT && mirror != nullptr && blockIdx.x == 0 && warp == 0) {
        export_header(header, mirror, lane); // (the writing pass adds nothing to the header)
    }

    for (unsigned system = blockIdx.x * MOLECULE_WARPS + warp; system < in.n_systems; system += warps_in_grid) {
        const unsigned long long begin = in.offsets[system];
        const int n = static_cast<int>(in.offsets[system + 1] - begin);
        if (!taken_by_warp_kernel(in, system, n)) {
            if (!EMIT && lane == 0) {
                system_count[system] = 0; // the CTAs of the other kernel add to it
            }
            continue;
        }
        if (EMIT && system_start[system + 1] > capacity) {
            continue; // written before the host knew the total: the arrays are too short, the host will grow them
        }
        __syncwarp();
        // ---- the system's points: originals for the exact arithmetic, fp32 copies relative to the
        //      first point for the screen ----
        const double ox = (n > 0) ? batch_coordinate<Kind>(in, 3 * begin + 0) : 0.0;
        const double oy = (n > 0) ? batch_coordinate<Kind>(in, 3 * begin + 1) : 0.0;
        const double oz = (n > 0) ? batch_coordinate<Kind>(in, 3 * begin + 2) : 0.0;
        float reach = 0.0f;
        bool finite = true;
        for (int k = lane; k < ((n + 3) & ~3); k += 32) {
            double x = ox, y = oy, z = oz;
            if (k < n) {
                x = batch_coordinate<Kind>(in, 3 * (begin + k) + 0);
                y = batch_coordinate<Kind>(in, 3 * (begin + k) + 1);
                z = batch_coordinate<Kind>(in, 3 * (begin + k) + 2);
            }
            sh.x[warp][k] = x;
            sh.y[warp][k] = y;
            sh.z[warp][k] = z;
            const float fx = static_cast<float>(x - ox);
            const float fy = static_cast<float>(y - oy);
            const float fz = static_cast<float>(z - oz);
            sh.fx[warp][k] = fx;
            sh.fy[warp][k] = fy;
            sh.fz[warp][k] = fz;
            reach = fmaxf(reach, fmaxf(fabsf(fx), fmaxf(fabsf(fy), fabsf(fz))));
            if (!(isfinite(x) && isfinite(y) && isfinite(z))) {
                finite = false;
                if (!EMIT) {
                    atomicOr(&header->status, STATUS_BAD_POINT);
                    atomicMin(&header->first_bad, begin + k);
                }
            }
        }
        if (__any_sync(FULL_MASK, !finite)) {
            reach = __int_as_float(0x7f800000);
        }
#pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) {
            reach = fmaxf(reach, __shfl_xor_sync(FULL_MASK, reach, offset));
        }
        __syncwarp();
        const ScreenBand band = screen_band(reach * 1.7320508f, in.cutoff, in.cutoff2);

        const unsigned long long index_offset = in.global_indices ? begin : 0ull;
        constexpr unsigned per_hit = Kind::FULL ? 2u : 1u;
        unsigned long long next = EMIT ? system_start[system] : 0ull; // where the next hits go
        int listed = 0;                                               // hits waiting in the list (the same value in every lane)
        int hits = 0;
        const auto write = [&](int count) {
            for (int c0 = 0; c0 < count; c0 += 32) {
                const int n_valid = min(32, count - c0);
                int i = 0, j = 0;
                if (lane < n_valid) {
                    const unsigned entry = sh.list[warp][c0 + lane];
                    i = entry >> 8;
                    j = entry & 255;
                }
                double vx, vy, vz;
                const double d = __dsqrt_rn(molecule_pair(sh, warp, i, j, vx, vy, vz));
                write_hits<Kind>(sh.transpose[warp], out, lane, next, n_valid, index_offset + i, index_offset + j, 0, 0, 0, d, vx, vy, vz, false);
                next += static_cast<unsigned long long>(n_valid) * per_hit;
            }
        };
        // a lane per home point i, words of 32 candidates j; only j > i
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane;
            const int own = min(i, n - 1);
            const float ax = -sh.fx[warp][own];
            const float ay = -sh.fy[warp][own];
            const float az = -sh.fz[warp][own];
            for (int j0 = i0; j0 < n; j0 += 32) {
                const unsigned keep = (i < n) ? bits_from(i + 1 - j0) & ~bits_from(n - j0) : 0u;
                const unsigned inside = screen_word(
                    sh.fx[warp] + j0, sh.fy[warp] + j0, sh.fz[warp] + j0, min(8, (n - j0 + 3) >> 2), ax, ay, az, band, keep,
                    [&](int b) {
                        double vx, vy, vz;
                        return molecule_pair(sh, warp, i, j0 + b, vx, vy, vz) < in.cutoff2;
                    }
                );
                if (EMIT) {
                    list_hits(inside, static_cast<unsigned>((i << 8) | j0), sh.list[warp], listed, lane, write);
                } else {
                    hits += __popc(inside);
                }
            }
        }
        if (EMIT) {
            if (listed > 0) {
                write(listed);
            }
        } else {
            hits = __reduce_add_sync(FULL_MASK, hits);
            if (lane == 0) {
                system_count[system] = static_cast<unsigned long long>(hits) * per_hit;
            }
        }
    }
}

// ---- periodic systems, and larger ones -------------------------------------
// Candidates of a tile of 32 home points are the images of the points j >= i0
// whose fractional coordinates lie within the cutoff of the tile's bounding
// box: a cell as wide as two cutoffs has eight images per point there, not the
// 27 around every pair. A chunk of 128 points (one per thread) counts its
// images, a scan numbers them, and the images are staged 256 at a time; warps
// take words of 32 of them. What bounds it: the latency of the short chain
// (box, points, scan, stage) for the few thousand tiles that a batch of
// hundreds of cells has; the work itself is the emission of the hits.
// Several CTAs share the tiles of a system when the systems alone would not
// fill the GPU. 512 cells of 4 to 200 atoms (5 A cutoff, 2.8 M pairs): 31 us to
// count and 67 us to write; exact arithmetic on every image of every pair, a CTA
// per system, took 640 and 954.

constexpr int SMALL_CHUNK = SMALL_THREADS; // points whose images are listed at a time
constexpr int SMALL_BATCH = 256;           // images staged at a time
constexpr int SMALL_TILE = 32;             // home points per tile

struct SmallShared {
    alignas(16) float near_x[SMALL_BATCH]; // images relative to the first home point of the tile
    alignas(16) float near_y[SMALL_BATCH];
    alignas(16) float near_z[SMALL_BATCH];
    int4 image[SMALL_BATCH];               // x, y, z: image shift minus wrap shift of the point; w: the point in the chunk
    alignas(16) double transpose[SMALL_WARPS][TRANSPOSE_DOUBLES];
    SystemFrame frame;
    double x[SMALL_CHUNK];                 // original positions of the chunk
    double y[SMALL_CHUNK];
    double z[SMALL_CHUNK];
    int wrap[3][SMALL_CHUNK];              // wrap shift, seen from the first home point
    int low[3][SMALL_CHUNK];               // first image in each direction
    int count[2][SMALL_CHUNK];             // images in the first two directions
    int first_slot[SMALL_CHUNK + 1];       // exclusive scan of the images per point
    double home[3][SMALL_TILE];
    int home_wrap[3][SMALL_TILE];
    double box_lo[3], box_hi[3];           // fractional coordinates images of this tile can have
    ScreenBand band;
    int warp_sum[SMALL_WARPS];
    unsigned self_word[SMALL_BATCH / 32];  // images a point may pair with itself in
    unsigned short list[SMALL_WARPS][HIT_LIST]; // (home point << 8) | slot
    unsigned long long counter;            // output elements counted (pass 1) / handed out (pass 2)
};

/// The reference's arithmetic, operation for operation (vesin/src/cpu_cell_list.cpp:135-138, types.hpp:232-243).
__device__ __forceinline__ double small_pair(
    const SystemFrame& frame, double rix, double riy, double riz, double rjx, double rjy, double rjz, int s0, int s1, int s2, double& vx,
    double& vy, double& vz
) {
    const double f0 = static_cast<double>(s0), f1 = static_cast<double>(s1), f2 = static_cast<double>(s2);
    const double shx = __dadd_rn(__dadd_rn(__dmul_rn(f0, frame.H[0][0]), __dmul_rn(f1, frame.H[1][0])), __dmul_rn(f2, frame.H[2][0]));
    const double shy = __dadd_rn(__dadd_rn(__dmul_rn(f0, frame.H[0][1]), __dmul_rn(f1, frame.H[1][1])), __dmul_rn(f2, frame.H[2][1]));
    const double shz = __dadd_rn(__dadd_rn(__dmul_rn(f0, frame.H[0][2]), __dmul_rn(f1, frame.H[1][2])), __dmul_rn(f2, frame.H[2][2]));
    vx = __dadd_rn(__dsub_rn(rjx, rix), shx);
    vy = __dadd_rn(__dsub_rn(rjy, riy), shy);
    vz = __dadd_rn(__dsub_rn(rjz, riz), shz);
    return __dadd_rn(__dadd_rn(__dmul_rn(vx, vx), __dmul_rn(vy, vy)), __dmul_rn(vz, vz));
}

template <class Kind>
__global__ void __launch_bounds__(SMALL_THREADS, SMALL_CTAS) small_systems_kernel(
    const BatchInput in, const unsigned splits, unsigned long long* __restrict__ system_count, unsigned long long* __restrict__ share_count,
    const unsigned long long* __restrict__ system_start, PairOutput out, DeviceHeader* header, const unsigned long long capacity
) {
    constexpr bool EMIT = Kind::EMIT;
    let_next_kernel_start();
    wait_for_previous_kernel();
    __shared__ SmallShared sh;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    constexpr unsigned per_hit = Kind::FULL ? 2u : 1u;

    const unsigned long long n_items = static_cast<unsigned long long>(in.n_systems) * splits;
    for (unsigned long long item = blockIdx.x; item < n_items; item += gridDim.x) {
        // (the first tiles of all systems come first: they see the most candidates, and the light ones
        // behind them even out when the SMs run dry: 512 cells of 4 to 200 atoms, both passes, 131 -> 111 us)
        const int share = static_cast<int>(item / in.n_systems);
        const unsigned system = static_cast<unsigned>(item - static_cast<unsigned long long>(share) * in.n_systems);
        const unsigned long long begin = in.offsets[system];
        const int n = static_cast<int>(in.offsets[system + 1] - begin);
        if (taken_by_warp_kernel(in, system, n)) {
            continue;
        }
        const int n_tiles = (n + SMALL_TILE - 1) / SMALL_TILE;
        if (share >= max(n_tiles, 1)) {
            continue; // (only shares of earlier tiles are ever added up)
        }
        if (EMIT && system_start[system + 1] > capacity) {
            continue; // as in the warp kernel
        }
        __syncthreads(); // previous item done with shared memory
        if (threadIdx.x >= 32 && threadIdx.x < 32 + sizeof(SystemFrame) / 4) {
            reinterpret_cast<unsigned*>(&sh.frame)[threadIdx.x - 32] = reinterpret_cast<const unsigned*>(static_cast<const SystemFrame*>(in.frames) + system)[threadIdx.x - 32];
        }
        if (warp == 0) {
            unsigned long long before = 0;
            if (EMIT) {
                before = system_start[system];
                for (int s = 0; s < share; s++) {
                    before += share_count[system * static_cast<unsigned long long>(splits) + s];
                }
            }
            if (lane == 0) {
                sh.counter = before;
            }
        }
        __syncthreads();
        const SystemFrame& frame = sh.frame;
        const bool usable = frame.singular == 0;
        if (!EMIT && !usable && threadIdx.x == 0) {
            atomicOr(&header->status, frame.singular == 2 ? STATUS_STENCIL_TOO_LARGE : STATUS_SINGULAR_BOX);
            atomicMin(&header->mask_cursor, static_cast<unsigned long long>(system)); // first offending system
        }
        if (!EMIT && share == 0) {
            for (int k = threadIdx.x; k < n; k += SMALL_THREADS) {
                const bool finite = isfinite(batch_coordinate<Kind>(in, 3 * (begin + k) + 0)) && isfinite(batch_coordinate<Kind>(in, 3 * (begin + k) + 1)) &&
                                    isfinite(batch_coordinate<Kind>(in, 3 * (begin + k) + 2));
                if (!finite) {
                    atomicOr(&header->status, STATUS_BAD_POINT);
                    atomicMin(&header->first_bad, begin + k);
                }
            }
        }
        const unsigned long long index_offset = in.global_indices ? begin : 0ull;
        unsigned long long my_count = 0;

        for (int i0 = share * SMALL_TILE; usable && i0 < n; i0 += static_cast<int>(splits) * SMALL_TILE) {
            const int n_home = min(SMALL_TILE, n - i0);
            // everything is seen from the first home point: fractional coordinates, wrap shifts
            // (what they have in common cancels in the shift of a pair) and fp32 positions
            const double ox = batch_coordinate<Kind>(in, 3 * (begin + i0) + 0);
            const double oy = batch_coordinate<Kind>(in, 3 * (begin + i0) + 1);
            const double oz = batch_coordinate<Kind>(in, 3 * (begin + i0) + 2);
            float hx = 0, hy = 0, hz = 0; // the lane's home point, negated
            bool exact_only = false;
            for (int chunk0 = i0; chunk0 < n; chunk0 += SMALL_CHUNK) {
                const int j = chunk0 + static_cast<int>(threadIdx.x);
                bool have = j < n;
                double rx = ox, ry = oy, rz = oz;
                if (have) {
                    rx = batch_coordinate<Kind>(in, 3 * (begin + j) + 0);
                    ry = batch_coordinate<Kind>(in, 3 * (begin + j) + 1);
                    rz = batch_coordinate<Kind>(in, 3 * (begin + j) + 2);
                    have = isfinite(rx) && isfinite(ry) && isfinite(rz); // others are reported by the counting pass
                }
                const double dx = rx - ox, dy = ry - oy, dz = rz - oz;
                double f[3];
                int wrap[3];
                double slack = 0.0; // covers the rounding of the fractional coordinates
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const double ax = dx * frame.Hinv[0][k], ay = dy * frame.Hinv[1][k], az = dz * frame.Hinv[2][k];
                    const double t = fmin(fmax(ax + ay + az, -1.0e9), 1.0e9);
                    slack = fmax(slack, 1.0e-14 * (fabs(ax) + fabs(ay) + fabs(az)));
                    const double w = frame.periodic[k] ? floor(t) : 0.0;
                    wrap[k] = static_cast<int>(w);
                    f[k] = t - w;
                }
                const double image_slack = fmin(slack, 1.0e-3); // bounds the images of a point absurdly far out
                __syncthreads(); // the previous chunk has been consumed
                sh.x[threadIdx.x] = rx;
                sh.y[threadIdx.x] = ry;
                sh.z[threadIdx.x] = rz;
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    sh.wrap[k][threadIdx.x] = wrap[k];
                }
                if (chunk0 == i0 && warp == 0) {
                    // the home points open the first chunk: what images can reach them?
                    const bool home = lane < n_home;
                    sh.home[0][lane] = rx;
                    sh.home[1][lane] = ry;
                    sh.home[2][lane] = rz;
                    float reach = 0.0f;
                    float rel[3];
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        sh.home_wrap[k][lane] = wrap[k];
                        const double r = ((k == 0) ? dx : ((k == 1) ? dy : dz)) -
                                         (wrap[0] * frame.H[0][k] + wrap[1] * frame.H[1][k] + wrap[2] * frame.H[2][k]);
                        rel[k] = static_cast<float>(r);
                        reach += rel[k] * rel[k];
                    }
                    reach = sqrtf(reach);
                    if (!home) {
                        reach = 0.0f;
                    } else if (!(reach < 3.0e38f)) {
                        reach = __int_as_float(0x7f800000);
                    }
                    double most_slack = home ? fmin(slack, 1.0e9) : 0.0;
#pragma unroll
                    for (int offset = 16; offset > 0; offset >>= 1) {
                        reach = fmaxf(reach, __shfl_xor_sync(FULL_MASK, reach, offset));
                        most_slack = fmax(most_slack, __shfl_xor_sync(FULL_MASK, most_slack, offset));
                    }
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        double lo = home ? f[k] : 1.0e300;
                        double hi = home ? f[k] : -1.0e300;
#pragma unroll
                        for (int offset = 16; offset > 0; offset >>= 1) {
                            lo = fmin(lo, __shfl_xor_sync(FULL_MASK, lo, offset));
                            hi = fmax(hi, __shfl_xor_sync(FULL_MASK, hi, offset));
                        }
                        if (lane == 0) {
                            const double margin = frame.reach[k] + 1.0e-9 + (frame.periodic[k] ? fmin(most_slack, 1.0e-3) : most_slack);
                            sh.box_lo[k] = lo - margin;
                            sh.box_hi[k] = hi + margin;
                        }
                    }
                    if (lane == 0) {
                        sh.band = screen_band(reach * 1.0001f, in.cutoff, in.cutoff2);
                    }
                }
                if (chunk0 == i0) {
                    __syncthreads();
                    const int h = lane;
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        const double r = sh.home[k][h] - ((k == 0) ? ox : ((k == 1) ? oy : oz));
                        const double rel = r - (sh.home_wrap[0][h] * frame.H[0][k] + sh.home_wrap[1][h] * frame.H[1][k] + sh.home_wrap[2][h] * frame.H[2][k]);
                        (k == 0 ? hx : (k == 1 ? hy : hz)) = -static_cast<float>(rel);
                    }
                }
                // ---- images of the thread's point inside the reach of the tile ----
                int images = have ? 1 : 0;
                bool far = false; // so far out that fp64 rounding of the shift products shows
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    int low = 0;
                    int count = 1;
                    if (frame.periodic[k]) {
                        low = static_cast<int>(ceil(sh.box_lo[k] - image_slack - f[k]));
                        count = max(0, static_cast<int>(floor(sh.box_hi[k] + image_slack - f[k])) - low + 1);
                    } else if (f[k] < sh.box_lo[k] - slack || f[k] > sh.box_hi[k] + slack) {
                        count = 0;
                    }
                    far = far || wrap[k] > 100000 || wrap[k] < -100000;
                    sh.low[k][threadIdx.x] = low;
                    if (k < 2) {
                        sh.count[k][threadIdx.x] = count;
                    }
                    images *= count;
                }
                int inclusive = images;
#pragma unroll
                for (int offset = 1; offset < 32; offset <<= 1) {
                    const int up = __shfl_up_sync(FULL_MASK, inclusive, offset);
                    if (lane >= offset) {
                        inclusive += up;
                    }
                }
                if (lane == 31) {
                    sh.warp_sum[warp] = inclusive;
                }
                exact_only = __syncthreads_or(far) != 0 || exact_only;
                int before = 0;
                int total = 0;
#pragma unroll
                for (int w = 0; w < SMALL_WARPS; w++) {
                    before += (w < warp) ? sh.warp_sum[w] : 0;
                    total += sh.warp_sum[w];
                }
                sh.first_slot[threadIdx.x] = before + inclusive - images;
                if (threadIdx.x == 0) {
                    sh.first_slot[SMALL_CHUNK] = total;
                }
                ScreenBand band = sh.band;
                if (exact_only) {
                    band = everything_exact();
                }

                for (int batch0 = 0; batch0 < total; batch0 += SMALL_BATCH) {
                    const int slots = min(SMALL_BATCH, total - batch0);
                    const int words = (slots + 31) >> 5;
                    __syncthreads(); // the scan is visible; the previous batch has been consumed
                    for (int s = threadIdx.x; s < 32 * words; s += SMALL_THREADS) {
                        bool self = false;
                        float nx = 0.0f, ny = 0.0f, nz = 0.0f;
                        int4 image = make_int4(0, 0, 0, 0);
                        if (s < slots) {
                            const int slot = batch0 + s;
                            int t = 0; // last point whose images start at or before the slot
#pragma unroll
                            for (int step = SMALL_CHUNK / 2; step > 0; step >>= 1) {
                                if (sh.first_slot[t + step] <= slot) {
                                    t += step;
                                }
                            }
                            const int number = slot - sh.first_slot[t];
                            const int c0 = sh.count[0][t];
                            const int c1 = sh.count[1][t];
                            const int row = number / c0;
                            const int t0 = sh.low[0][t] + (number - row * c0);
                            const int plane = row / c1;
                            const int t1 = sh.low[1][t] + (row - plane * c1);
                            const int t2 = sh.low[2][t] + plane;
                            image = make_int4(t0 - sh.wrap[0][t], t1 - sh.wrap[1][t], t2 - sh.wrap[2][t], t);
                            nx = static_cast<float>((sh.x[t] - ox) + (image.x * frame.H[0][0] + image.y * frame.H[1][0] + image.z * frame.H[2][0]));
                            ny = static_cast<float>((sh.y[t] - oy) + (image.x * frame.H[0][1] + image.y * frame.H[1][1] + image.z * frame.H[2][1]));
                            nz = static_cast<float>((sh.z[t] - oz) + (image.x * frame.H[0][2] + image.y * frame.H[1][2] + image.z * frame.H[2][2]));
                            // a point with itself: only images, and only one of S / -S (the other
                            // one is written as the reversed pair)
                            self = (t0 | t1 | t2) != 0 && half_rule_small(t0, t1, t2);
                        }
                        sh.near_x[s] = nx;
                        sh.near_y[s] = ny;
                        sh.near_z[s] = nz;
                        sh.image[s] = image;
                        const unsigned word = __ballot_sync(FULL_MASK, self);
                        if (lane == 0) {
                            sh.self_word[s >> 5] = word;
                        }
                    }
                    __syncthreads();

                    int listed = 0;
                    const auto write = [&](int count) {
                        unsigned long long first = 0;
                        if (lane == 0) {
                            first = atomicAdd(&sh.counter, static_cast<unsigned long long>(count) * per_hit);
                        }
                        first = __shfl_sync(FULL_MASK, first, 0);
                        for (int c0 = 0; c0 < count; c0 += 32) {
                            const int n_valid = min(32, count - c0);
                            int h = 0, s = 0;
                            if (lane < n_valid) {
                                const unsigned entry = sh.list[warp][c0 + lane];
                                h = entry >> 8;
                                s = entry & 255;
                            }
                            const int4 image = sh.image[s];
                            const int s0 = image.x + sh.home_wrap[0][h];
                            const int s1 = image.y + sh.home_wrap[1][h];
                            const int s2 = image.z + sh.home_wrap[2][h];
                            double vx, vy, vz;
                            const double d = __dsqrt_rn(small_pair(
                                frame, sh.home[0][h], sh.home[1][h], sh.home[2][h], sh.x[image.w], sh.y[image.w], sh.z[image.w], s0, s1, s2, vx, vy, vz
                            ));
                            write_hits<Kind>(
                                sh.transpose[warp], out, lane, first + static_cast<unsigned long long>(c0) * per_hit, n_valid, index_offset + i0 + h,
                                index_offset + chunk0 + image.w, s0, s1, s2, d, vx, vy, vz,
                                __any_sync(FULL_MASK, (s0 | s1 | s2) != 0) != 0
                            );
                        }
                    };
                    for (int w = warp; w < words; w += SMALL_WARPS) {
                        const int in_word = min(32, slots - 32 * w);
                        unsigned keep = (lane < n_home) ? ~bits_from(in_word) : 0u;
                        if (chunk0 == i0) {
                            // of the points of the tile only those after the home point, and its own images
                            const int own_first = sh.first_slot[lane] - batch0 - 32 * w;
                            const int own_end = sh.first_slot[lane + 1] - batch0 - 32 * w;
                            keep &= bits_from(own_end) | (sh.self_word[w] & bits_from(own_first));
                        }
                        const unsigned inside = screen_word(
                            sh.near_x + 32 * w, sh.near_y + 32 * w, sh.near_z + 32 * w, (in_word + 3) >> 2, hx, hy, hz, band, keep,
                            [&](int b) {
                                const int4 image = sh.image[32 * w + b];
                                double vx, vy, vz;
                                return small_pair(
                                           frame, sh.home[0][lane], sh.home[1][lane], sh.home[2][lane], sh.x[image.w], sh.y[image.w], sh.z[image.w],
                                           image.x + sh.home_wrap[0][lane], image.y + sh.home_wrap[1][lane], image.z + sh.home_wrap[2][lane], vx, vy, vz
                                       ) < in.cutoff2;
                            }
                        );
                        if (EMIT) {
                            list_hits(inside, static_cast<unsigned>((lane << 8) | (32 * w)), sh.list[warp], listed, lane, write);
                        } else {
                            my_count += static_cast<unsigned>(__popc(inside));
                        }
                    }
                    if (EMIT && listed > 0) {
                        write(listed);
                    }
                }
            }
        }
        if (!EMIT) {
#pragma unroll
            for (int offset = 16; offset > 0; offset >>= 1) {
                my_count += __shfl_xor_sync(FULL_MASK, my_count, offset);
            }
            if (lane == 0 && my_count != 0) {
                atomicAdd(&sh.counter, my_count * per_hit);
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                const unsigned long long counted = sh.counter;
                share_count[system * static_cast<unsigned long long>(splits) + share] = counted;
                if (counted != 0) {
                    atomicAdd(&system_count[system], counted);
                }
            }
        }
    }
}

} // namespace

size_t small_systems_max_points() {
    return 2048;
}

/// Calls use(kind) with the kind of the launch.
template <bool EMIT, class Use>
static void with_kind(const BatchInput& in, bool paired, Use use) {
    const auto with_type = [&](auto full, auto aligned) {
        if (in.is_float) {
            use(BatchKind<EMIT, decltype(full)::value, true, decltype(aligned)::value>{});
        } else {
            use(BatchKind<EMIT, decltype(full)::value, false, decltype(aligned)::value>{});
        }
    };
    // (half lists and counts store no pairs side by side)
    if constexpr (EMIT) {
        if (in.full && paired) {
            with_type(std::true_type{}, std::true_type{});
            return;
        }
    }
    in.full ? with_type(std::true_type{}, std::false_type{}) : with_type(std::false_type{}, std::false_type{});
}

static unsigned multiprocessors() {
    int device = 0, sms = 148;
    if (cudaGetDevice(&device) == cudaSuccess) {
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    }
    return static_cast<unsigned>(sms);
}

unsigned small_splits(unsigned n_systems, size_t max_points) {
    // about four waves of CTAs, so that systems of different sizes even out; never more than tiles
    const unsigned tiles = static_cast<unsigned>((max_points + SMALL_TILE - 1) / SMALL_TILE);
    const unsigned wanted = 4 * SMALL_CTAS * multiprocessors() / std::max(n_systems, 1u);
    return std::max(1u, std::min(wanted, tiles));
}

static unsigned small_grid(unsigned n_systems, unsigned splits) {
    return static_cast<unsigned>(std::min<unsigned long long>(static_cast<unsigned long long>(n_systems) * splits, 1ull << 20));
}

static unsigned molecules_grid(unsigned n_systems) {
    const unsigned wanted = (n_systems + MOLECULE_WARPS - 1) / MOLECULE_WARPS;
    return std::max(1u, std::min(wanted, 1u << 20));
}

size_t small_frame_bytes() {
    return sizeof(SystemFrame);
}

void launch_batch_front(const BatchInput& in, bool any_for_cta_kernel, DeviceHeader* header, cudaStream_t stream) {
    static_assert(sizeof(DeviceHeader) % 4 == 0 && sizeof(DeviceHeader) <= 4 * FRONT_THREADS, "a thread per word");
    static_assert(sizeof(SystemFrame) % 4 == 0 && sizeof(SystemFrame) <= 4 * (SMALL_THREADS - 32), "copied word by word");
    constexpr unsigned per_block = FRONT_THREADS / 32;
    const unsigned blocks = any_for_cta_kernel ? std::min((in.n_systems + per_block - 1) / per_block, 1u << 16) : 1u;
    batch_front_kernel<<<std::max(blocks, 1u), FRONT_THREADS, 0, stream>>>(in, any_for_cta_kernel ? static_cast<SystemFrame*>(in.frames) : nullptr, header);
}

void launch_small_count(
    const BatchInput& in, size_t max_points, bool any_for_cta_kernel, unsigned long long* system_count, unsigned long long* share_count,
    DeviceHeader* header, cudaStream_t stream
) {
    const PairOutput nothing{};
    with_kind<false>(in, false, [&](auto kind) {
        using Kind = decltype(kind);
        launch_chained(
            molecules_kernel<Kind>, molecules_grid(in.n_systems), MOLECULE_WARPS * 32, sizeof(MoleculeShared), stream, in, system_count, nullptr, nothing,
            header, 0ull, nullptr
        );
        if (any_for_cta_kernel) {
            const unsigned splits = small_splits(in.n_systems, max_points);
            launch_chained(
                small_systems_kernel<Kind>, small_grid(in.n_systems, splits), SMALL_THREADS, 0, stream, in, splits, system_count, share_count, nullptr,
                nothing, header, 0ull
            );
        }
    });
}

void launch_small_emit(
    const BatchInput& in, size_t max_points, bool any_for_cta_kernel, const unsigned long long* system_start,
    unsigned long long* share_count, PairOutput out, DeviceHeader* header, cudaStream_t stream, unsigned long long capacity,
    DeviceHeader* mirror
) {
    // paired stores of full lists need aligned arrays (every system of a full list starts on an even element)
    with_kind<true>(in, paired_stores_fit(out) != 0, [&](auto kind) {
        using Kind = decltype(kind);
        launch_chained(
            molecules_kernel<Kind>, molecules_grid(in.n_systems), MOLECULE_WARPS * 32, sizeof(MoleculeShared), stream, in, nullptr, system_start, out, header,
            capacity, mirror
        );
        if (any_for_cta_kernel) {
            const unsigned splits = small_splits(in.n_systems, max_points);
            launch_chained(
                small_systems_kernel<Kind>, small_grid(in.n_systems, splits), SMALL_THREADS, 0, stream, in, splits, nullptr, share_count, system_start, out,
                header, capacity
            );
        }
    });
}

size_t molecules_max_points() {
    return MOLECULE_MAX_POINTS;
}

} // namespace vb200
