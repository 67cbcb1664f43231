#include "runtime.hpp"

#include "columns_warp.hpp"
#include "simt_tiles.hpp"

#include <algorithm>
#include <array>
#include <cstring>

#include "util.hpp"

namespace skb {

void throw_cuda(cudaError_t err, const char* what) {
    // The failure is reported by this exception: the code that the runtime keeps for
    // the thread would fail the next plain launch's cudaGetLastError() as well.
    cudaGetLastError();
    const int code = err == cudaErrorMemoryAllocation ? -4 : -2;
    throw Error(code, std::string(what) + ": " + cudaGetErrorName(err) + " (" + cudaGetErrorString(err) + ")");
}

void DeviceBuffer::allocate(size_t bytes) {
    release();
    if (bytes == 0) return;
    check_cuda(cudaMalloc(&ptr_, bytes), "cudaMalloc");
    bytes_ = bytes;
}

void DeviceBuffer::release() noexcept {
    if (ptr_ != nullptr) cudaFree(ptr_);
    ptr_ = nullptr;
    bytes_ = 0;
}

void DeviceBuffer::upload(const void* src, size_t bytes, cudaStream_t stream) {
    if (bytes > bytes_) throw Error(-1, "upload larger than the device buffer");
    if (stream == nullptr) {
        check_cuda(cudaMemcpy(ptr_, src, bytes, cudaMemcpyHostToDevice), "cudaMemcpy H2D");
    } else {
        check_cuda(cudaMemcpyAsync(ptr_, src, bytes, cudaMemcpyHostToDevice, stream), "cudaMemcpyAsync H2D");
    }
}

int sm_count() {
    int device = 0, count = 0;
    check_cuda(cudaGetDevice(&device), "cudaGetDevice");
    check_cuda(cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device), "cudaDeviceGetAttribute");
    return count;
}

size_t element_bytes(Precision p) { return p == Precision::f64 ? sizeof(double) : sizeof(float); }

std::vector<double> regs_table(const std::vector<double>& natural, int perThread, int first) {
    const int n = static_cast<int>(natural.size() / 2);
    std::vector<double> out;
    for (int i = 0; i < regs_table_size(n, perThread, first); ++i) {
        const int k = regs_table_index(n, perThread, first, i);
        out.push_back(natural[2 * k]);
        out.push_back(natural[2 * k + 1]);
    }
    return out;
}

DeviceBuffer upload_real_table(const std::vector<double>& values, Precision p) {
    if (p == Precision::f64) return upload_vector(values);
    std::vector<float> f(values.begin(), values.end());
    return upload_vector(f);
}

std::uint64_t active_columns(const std::vector<RetainedMode>& modes) {
    std::uint64_t active = 0;
    for (const auto& m : modes) active = std::max<std::uint64_t>(active, m.kx + 1);
    return active;
}

HorizontalPlan::HorizontalPlan(const Workload& w, Precision p, bool pruned, std::uint64_t maxPlanes, bool fused)
    : w_(w), p_(p), maxPlanes_(maxPlanes) {
    validate_workload(w);
    if (!supported_length(static_cast<long long>(w.nx)) || !supported_length(static_cast<long long>(w.ny)))
        throw Error(-2, "unsupported: the cuda provider transforms power-of-two Nx and Ny in [2, 1024]; got " +
                            std::to_string(w.nx) + "x" + std::to_string(w.ny));
    const auto planStart = Clock::now();
    const auto modes = retained_modes(w);
    modeCount_ = modes.size();
    if (pruned && modes.empty()) throw Error(-1, "pruned provider: the workload retains no modes");
    keep_ = static_cast<int>(pruned ? active_columns(modes) : w.nxHalf());
    const auto columnsForTables = pruned ? static_cast<std::uint64_t>(keep_) : w.nxHalf();
    const auto tables = column_tables(w, modes, columnsForTables);
    const auto twHalf = twiddle_table(std::max<std::uint64_t>(1, w.nx / 2));
    const auto twFull = twiddle_table(w.nx);
    const auto twCol = twiddle_table(w.ny);
    planningSeconds = seconds_since(planStart);

    const auto allocStart = Clock::now();
    // The twiddle tables that the path reads, in one buffer and one copy.
    const int half = static_cast<int>(std::max<std::uint64_t>(1, w.nx / 2));
    std::vector<double> twiddles;
    std::vector<std::pair<const void**, size_t>> placed;
    auto place = [&](const void** table, const std::vector<double>& values) {
        placed.push_back({table, twiddles.size() * element_bytes(p)});
        twiddles.insert(twiddles.end(), values.begin(), values.end());
    };
    place(&twFull_, twFull);
    place(&colTable_, regs_table(twCol, column_regs_per_thread(static_cast<int>(w.ny), p == Precision::f64)));
    if (fused) {
        place(&twHalf_, twHalf);
        place(&twCol_, twCol);
    } else {
        place(&rowForward_, regs_table(twHalf, row_regs_per_thread(half)));
        place(&rowInverse_, regs_table(twHalf, row_regs_per_thread(half), row_plane_radix(half)));
    }
    twiddles_ = upload_real_table(twiddles, p);
    for (const auto& [table, offset] : placed) *table = twiddles_.get<unsigned char>() + offset;
    cellMap_ = upload_vector(tables.cellMap);
    gatherMap_ = upload_vector(tables.gatherMap);
    colStart_ = upload_vector(tables.colStart);
    colKy_ = upload_vector(tables.colKy);
    colMode_ = upload_vector(tables.colMode);
    modeKx_ = upload_vector(tables.modeKx);
    modeKy_ = upload_vector(tables.modeKy);
    modeConj_ = upload_vector(tables.modeConj);
    bins_.allocate(bin_bytes(maxPlanes));
    {
        // Per-column band of the retained cells, and whether it is exact.
        std::vector<int> band(static_cast<size_t>(keep_), -1);
        for (int kx = 0; kx < keep_; ++kx)
            for (std::uint64_t ky = 0; ky < w.ny; ++ky)
                if (tables.cellMap[kx * w.ny + ky] >= 0)
                    band[kx] = std::max(band[kx], static_cast<int>(std::min<std::uint64_t>(ky, w.ny - ky)));
        bandExact_ = true;
        for (int kx = 0; kx < keep_ && bandExact_; ++kx)
            for (std::uint64_t ky = 0; ky < w.ny; ++ky) {
                const bool cell = tables.cellMap[kx * w.ny + ky] >= 0;
                const bool inBand = static_cast<int>(std::min<std::uint64_t>(ky, w.ny - ky)) <= band[kx];
                if (cell != inBand) {
                    bandExact_ = false;
                    break;
                }
            }
        band_ = upload_vector(band);
    }
    allocationSeconds = seconds_since(allocStart);
    persistentBytes = twiddles_.bytes() + cellMap_.bytes() + gatherMap_.bytes() + colStart_.bytes() +
                      colKy_.bytes() + colMode_.bytes() + modeKx_.bytes() + modeKy_.bytes() + modeConj_.bytes();
    scratchBytes = bins_.bytes();
}

ModeTables HorizontalPlan::tables() const {
    return {cellMap_.get<int>(), colStart_.get<int>(), colKy_.get<int>(), colMode_.get<int>(), gatherMap_.get<int>()};
}

void HorizontalPlan::forward_rows(const void* real, std::uint64_t planes, cudaStream_t s) const {
    if (planes > maxPlanes_) throw Error(-1, "plane count exceeds the plan's scratch");
    check_cuda(launch_rows_forward(p_, static_cast<int>(w_.nx), static_cast<int>(w_.ny),
                                   static_cast<long long>(planes), keep_, real, scratch(), rowForward_,
                                   twFull_, s),
               "row r2c kernel");
}

void HorizontalPlan::forward_columns(const ViewSet& views, double scale, cudaStream_t s) const {
    if (static_cast<std::uint64_t>(views.count) * w_.nz > maxPlanes_)
        throw Error(-1, "plane count exceeds the plan's scratch");
    forward_columns(scratch(), views, scale, s);
}

void HorizontalPlan::forward_columns(DenseBins in, const ViewSet& views, double scale, cudaStream_t s) const {
    check_cuda(launch_columns_gather(p_, static_cast<int>(w_.ny), static_cast<int>(w_.nz), keep_, in, views, tables(),
                                     scale, colTable_, s),
               "column c2c + retention kernel");
}

void HorizontalPlan::product_rows(const void* velocity, std::uint64_t members, double scale, DenseBins target,
                                  cudaStream_t s) const {
    if (3 * members * w_.nz > maxPlanes_) throw Error(-1, "plane count exceeds the plan's scratch");
    check_cuda(launch_rows_product(p_, static_cast<int>(w_.nx), static_cast<int>(w_.ny), static_cast<int>(w_.nz),
                                   static_cast<int>(members), keep_, scale, velocity, scratch(), target,
                                   rowInverse_, rowForward_, twFull_, s),
               "row product kernel");
}

void HorizontalPlan::inverse_columns(const ViewSet& views, cudaStream_t s) const {
    const auto planes = static_cast<std::uint64_t>(views.count) * w_.nz;
    if (planes > maxPlanes_) throw Error(-1, "plane count exceeds the plan's scratch");
    check_cuda(launch_columns_embed(p_, static_cast<int>(w_.ny), static_cast<int>(w_.nz), keep_, views, tables(),
                                    scratch(), colTable_, s),
               "embedding + column c2c kernel");
}

void HorizontalPlan::inverse_columns_into(const ViewSet& views, DenseBins out, cudaStream_t s, int zStride) const {
    if (out.kxStride != keep_) throw Error(-1, "bin array must hold keep() columns per row");
    const int nz = static_cast<int>(w_.nz);
    if (zStride == 0) zStride = nz;
    if (p_ == Precision::f32 && columns_warp_supported(static_cast<long long>(w_.ny))) {
        check_cuda(launch_columns_embed_warp(static_cast<int>(w_.ny), nz, zStride, keep_, views, tables(), out,
                                             twCol_, s),
                   "warp embedding + column c2c kernel");
        return;
    }
    if (zStride != nz) throw Error(-3, "padded bin planes need the FP32 warp column kernels");
    check_cuda(launch_columns_embed(p_, static_cast<int>(w_.ny), static_cast<int>(w_.nz), keep_, views, tables(), out,
                                    colTable_, s),
               "embedding + column c2c kernel");
}

void HorizontalPlan::forward_columns_from(DenseBins in, const ViewSet& views, double scale, cudaStream_t s,
                                          int zStride) const {
    if (in.kxStride != keep_) throw Error(-1, "bin array must hold keep() columns per row");
    const int nz = static_cast<int>(w_.nz);
    if (zStride == 0) zStride = nz;
    if (p_ == Precision::f32 && columns_warp_supported(static_cast<long long>(w_.ny))) {
        check_cuda(launch_columns_gather_warp(static_cast<int>(w_.ny), nz, zStride, keep_, in, views, tables(), scale,
                                              twCol_, s),
                   "warp column c2c + retention kernel");
        return;
    }
    if (zStride != nz) throw Error(-3, "padded bin planes need the FP32 warp column kernels");
    check_cuda(launch_columns_gather(p_, static_cast<int>(w_.ny), static_cast<int>(w_.nz), keep_, in, views,
                                     tables(), scale, colTable_, s),
               "column c2c + retention kernel");
}

void HorizontalPlan::inverse_columns_band(DenseBins bins, int slots, int zStride, cudaStream_t s) const {
    if (!bandExact_ || p_ != Precision::f32 || !columns_warp_supported(static_cast<long long>(w_.ny)))
        throw Error(-3, "band column stage needs FP32, an exact retained band and Ny in [32, 512]");
    check_cuda(launch_columns_inverse_band(static_cast<int>(w_.ny), static_cast<int>(w_.nz), zStride, slots, keep_,
                                           bins, band_.get<int>(), twCol_, colTable_, bandFormInverse_, s),
               "band inverse column kernel");
}

void HorizontalPlan::forward_columns_band(DenseBins bins, int slots, double scale, int zStride, cudaStream_t s) const {
    if (!bandExact_ || p_ != Precision::f32 || !columns_warp_supported(static_cast<long long>(w_.ny)))
        throw Error(-3, "band column stage needs FP32, an exact retained band and Ny in [32, 512]");
    check_cuda(launch_columns_forward_band(static_cast<int>(w_.ny), static_cast<int>(w_.nz), zStride, slots, keep_,
                                           bins, band_.get<int>(), scale, twCol_, colTable_, bandFormForward_,
                                           s),
               "band forward column kernel");
}

void HorizontalPlan::inverse_rows(void* real, std::uint64_t planes, cudaStream_t s) const {
    if (planes > maxPlanes_) throw Error(-1, "plane count exceeds the plan's scratch");
    check_cuda(launch_rows_inverse(p_, static_cast<int>(w_.nx), static_cast<int>(w_.ny),
                                   static_cast<long long>(planes), keep_, scratch(), real, rowInverse_,
                                   twFull_, s),
               "row c2r kernel");
}

void HorizontalPlan::forward(const void* real, std::uint64_t planes, const ViewSet& views, double scale,
                             cudaStream_t s) const {
    if (planes != static_cast<std::uint64_t>(views.count) * w_.nz)
        throw Error(-1, "field views must cover every real plane");
    forward_rows(real, planes, s);
    forward_columns(views, scale, s);
}

void HorizontalPlan::inverse(const ViewSet& views, void* real, cudaStream_t s) const {
    inverse_columns(views, s);
    inverse_rows(real, static_cast<std::uint64_t>(views.count) * w_.nz, s);
}

void HorizontalPlan::forward_dense(const void* real, void* wvm, std::uint64_t planes, cudaStream_t s) const {
    if (keep_ != static_cast<int>(w_.nxHalf())) throw Error(-3, "dense transform requested from a pruned plan");
    const DenseBins out{wvm, static_cast<long long>(planes), static_cast<long long>(w_.nxHalf())};
    check_cuda(launch_rows_forward(p_, static_cast<int>(w_.nx), static_cast<int>(w_.ny),
                                   static_cast<long long>(planes), keep_, real, out, rowForward_, twFull_, s),
               "row r2c kernel");
    check_cuda(launch_columns_dense(p_, -1, static_cast<int>(w_.ny), keep_, static_cast<long long>(planes), out, out,
                                    colTable_, s),
               "column c2c kernel");
}

void HorizontalPlan::inverse_dense(const void* wvm, void* real, std::uint64_t planes, cudaStream_t s) const {
    if (keep_ != static_cast<int>(w_.nxHalf())) throw Error(-3, "dense transform requested from a pruned plan");
    if (planes > maxPlanes_) throw Error(-1, "plane count exceeds the plan's scratch");
    const DenseBins in{const_cast<void*>(wvm), static_cast<long long>(planes), static_cast<long long>(w_.nxHalf())};
    check_cuda(launch_columns_dense(p_, +1, static_cast<int>(w_.ny), keep_, static_cast<long long>(planes), in,
                                    scratch(), colTable_, s),
               "column c2c kernel");
    check_cuda(launch_rows_inverse(p_, static_cast<int>(w_.nx), static_cast<int>(w_.ny),
                                   static_cast<long long>(planes), keep_, scratch(), real, rowInverse_,
                                   twFull_, s),
               "row c2r kernel");
}

void HorizontalPlan::gather_dense(const void* wvm, std::uint64_t planes, const ViewSet& views, double scale,
                                  cudaStream_t s) const {
    const DenseBins in{const_cast<void*>(wvm), static_cast<long long>(planes), static_cast<long long>(w_.nxHalf())};
    check_cuda(launch_gather_dense(p_, static_cast<int>(w_.ny), static_cast<int>(w_.nz),
                                   static_cast<long long>(modeCount_), modeKx_.get<int>(), modeKy_.get<int>(),
                                   modeConj_.get<unsigned char>(), in, views, scale, s),
               "retention kernel");
}

void HorizontalPlan::embed_dense(const ViewSet& views, void* wvm, std::uint64_t planes, cudaStream_t s) const {
    if (keep_ != static_cast<int>(w_.nxHalf())) throw Error(-3, "dense embedding requested from a pruned plan");
    const DenseBins out{wvm, static_cast<long long>(planes), static_cast<long long>(w_.nxHalf())};
    check_cuda(launch_embed_dense(p_, static_cast<int>(w_.ny), static_cast<int>(w_.nz), keep_, views, tables(), out,
                                  s),
               "embedding kernel");
}

// Which split-TF32x3 form serves a plan: tiles of 32 columns on mma.sync
// (vertical_tf32.cu) or the tcgen05 pipeline (tc_gemm.cu).  The estimates, in
// microseconds, are fits to both kernels at the 22 shapes of 64^2 to 512^2, Nz 17 to
// 129 and 1 to 8 members that were timed (within 12 % where the time is above 50 us):
// mma.sync pays by column, 0.18 ns for its loads and stores and 14 ps per 16 x 8 block
// of the padded matrix; the pipeline pays by 64-column tile on one of 148 SMs, however
// full the tile.  Measured, mma.sync / tcgen05 us: 256^2, Nz 65: 3-field forward of
// one member 41 / 71, of 4 97 / 96, 4 fields of 8 223 / 174, 12-field inverse 95 / 81;
// 512^2, Nz 129: 4-field forward 320 / 401, of 2 members 569 / 449, 15-field inverse
// 1000 / 472; 128^2, Nz 33: 3-field forward 12 / 20, of 8 members 29 / 36, 12-field
// inverse 18 / 22, of 8 members 91 / 75.  The pipeline has to be 10 % behind.
//
// The two forms round differently, so a plan whose members may run in batches of any
// size must choose the same form for every batch: `batch` is the size that the choice
// is made for, whatever the plan's own.
static bool tf32_small_groups(int R, int S, const std::vector<ModeGroup>& groups, std::uint64_t fields,
                              std::uint64_t batch) {
    if (R > kGemmTf32MaxRows) return false;
    double columns = 0.0, tiles = 0.0;
    for (const auto& g : groups) {
        const std::uint64_t c = g.count * fields * batch;
        columns += static_cast<double>(c);
        tiles += static_cast<double>((c + 63) / 64);
    }
    const int rows = (R + 15) / 16;
    const double small = 8.2 + columns * (0.18e-3 + 14e-6 * rows * ((S + 7) / 8));
    const double pipeline = 10.8 + tiles * (0.28 + 0.23 * rows + 1.1 * ((S + 31) / 32)) / 148.0;
    return 1.1 * small < pipeline;
}

VerticalPlan::VerticalPlan(GemmPrecision p, int rowsOut, int inner, const std::vector<ModeGroup>& groups,
                           std::uint64_t fields, std::uint64_t members, const std::vector<double>& natural,
                           std::uint64_t batch)
    : p_(p), R_(rowsOut), S_(inner) {
    if (groups.empty() || fields == 0 || members == 0) throw Error(-1, "Vertical GEMM requires groups and fields.");
    const auto matrixElems = static_cast<std::uint64_t>(rowsOut) * inner;
    if (natural.size() != groups.size() * matrixElems && natural.size() != matrixElems)
        throw Error(-1, "Vertical GEMM matrix family size does not match the groups.");
    const bool common = natural.size() == matrixElems && groups.size() > 1;
    std::uint64_t expected = 0;
    for (const auto& g : groups) {
        if (g.count == 0 || g.first != expected) throw Error(-1, "Vertical GEMM groups must be nonempty and contiguous.");
        expected += g.count;
    }
    const std::uint64_t perMember = expected * fields;
    if (members * perMember > static_cast<std::uint64_t>(INT32_MAX)) throw Error(-1, "too many GEMM columns");
    columns_ = members * perMember;
    members_ = members;
    memberColumns_ = static_cast<long long>(perMember);
    const std::uint64_t groupsCount = common ? 1 : groups.size();

    if (p == GemmPrecision::tf32x3 || p == GemmPrecision::bf16x3) {
        if (!tc_gemm_supported(rowsOut, inner))
            throw Error(-2, "unsupported: tensor-core GEMM needs the padded group matrix and two data stages in "
                            "227 KB of shared memory (R=" + std::to_string(rowsOut) + ", S=" + std::to_string(inner) +
                            ")");
        smallGroups_ = p == GemmPrecision::tf32x3 && tf32_small_groups(rowsOut, inner, groups, fields, batch);
    }
    std::vector<int> gc(groups.size()), gf(groups.size());
    for (std::uint64_t gi = 0; gi < groups.size(); ++gi) {
        gc[gi] = static_cast<int>(groups[gi].count * fields);
        gf[gi] = static_cast<int>(groups[gi].first * fields);
    }
    groupColumnsHost_ = gc;
    groupColumns_ = upload_vector(gc);
    groupFirst_ = upload_vector(gf);
    if (tensor_core() && !smallGroups_) {
        unitTiles_ = tc_gemm_unit_tiles();
        build_pipeline(std::vector<float>(natural.begin(), natural.end()));
        return;
    }

    const int width = gemm_tile_columns(p);
    // Member tiles unless they would run under 90 % full in a plan of several
    // members; then virtual tiles over each group's member-concatenated columns
    // (measured at 512², Nz 129, 8 members, FP64: forward 6.1 -> 4.5 ms with 4
    // targets, the two-family GEMMs 23.2 / 11.3 -> 21.9 / 4.6 ms; the 15-field
    // inverse, 94 % full as member tiles, ran 17.0 ms as member tiles and 20.4
    // as virtual ones).  Member tiles: one table whose prefixes serve smaller
    // member counts; virtual tiles: one table per member count.
    virtualTiles_ = simt_virtual_tiles(gc, members, width);
    const std::uint64_t tables = virtualTiles_ ? members : 1;
    tileTables_.resize(tables);
    tilePrefix_.assign(members, 0);
    for (std::uint64_t ti = 0; ti < tables; ++ti) {
        const std::uint64_t m = virtualTiles_ ? ti + 1 : members;
        const SimtTileTable h = simt_tiles(gc, gf, perMember, m, width, virtualTiles_, &tilePrefix_);
        TileTable& t = tileTables_[ti];
        t.group = upload_vector(h.group);
        t.column = upload_vector(h.column);
        t.count = upload_vector(h.count);
        t.per = upload_vector(h.per);
        t.first = upload_vector(h.first);
        t.tiles = static_cast<int>(h.group.size());
        if (virtualTiles_) tilePrefix_[m - 1] = t.tiles;
    }
    if (p == GemmPrecision::f64) {
        // Chunks of s, [chunk][r][s of the chunk] (vertical.hpp).
        const int padded = gemm_f64_row(inner);
        const std::uint64_t imageElems = static_cast<std::uint64_t>(rowsOut) * padded;
        std::vector<double> images(groupsCount * imageElems, 0.0);
        for (std::uint64_t g = 0; g < groupsCount; ++g)
            for (int s0 = 0; s0 < inner; s0 += kGemmF64Chunk) {
                const int chunk = gemm_f64_chunk_row(inner - s0);
                double* to = images.data() + g * imageElems + static_cast<std::uint64_t>(s0) * rowsOut;
                for (int r = 0; r < rowsOut; ++r)
                    std::copy_n(natural.data() + g * matrixElems + static_cast<std::uint64_t>(r) * inner + s0,
                                std::min(chunk, inner - s0), to + static_cast<std::uint64_t>(r) * chunk);
            }
        matrices_ = upload_vector(images);
        matrixStride_ = common ? 0 : static_cast<long long>(imageElems);
    } else if (smallGroups_) {
        const std::uint64_t imageElems = static_cast<std::uint64_t>(rowsOut) * gemm_tf32_row(inner);
        const DeviceBuffer staged = upload_vector(std::vector<float>(natural.begin(), natural.end()));
        matrices_.allocate(groupsCount * imageElems * sizeof(float));
        check_cuda(gemm_tf32_build_images(staged.get<float>(), static_cast<long long>(groupsCount), rowsOut, inner,
                                          matrices_.get<float>(), nullptr),
                   "split-TF32x3 GEMM images");
        check_cuda(cudaStreamSynchronize(nullptr), "split-TF32x3 GEMM images");
        matrixStride_ = common ? 0 : static_cast<long long>(imageElems);
        unitTiles_ = tc_gemm_unit_tiles();
    } else {
        // The FP32 form reads the transposed matrices At[g][s][r].
        std::vector<float> At(groupsCount * matrixElems);
        for (std::uint64_t g = 0; g < groupsCount; ++g)
            for (int r = 0; r < rowsOut; ++r)
                for (int s = 0; s < inner; ++s)
                    At[g * matrixElems + static_cast<std::uint64_t>(s) * rowsOut + r] =
                        static_cast<float>(natural[g * matrixElems + static_cast<std::uint64_t>(r) * inner + s]);
        matrices_ = upload_vector(At);
        matrixStride_ = common ? 0 : static_cast<long long>(matrixElems);
    }
}

// The tcgen05 form's part of a plan: FP32 matrices (one, if common to all
// groups) -> the kernel's operand images, split into TF32 hi/lo or BF16 h/m/l and
// swizzled once here; the work units; the word that an expired wait sets.
void VerticalPlan::build_pipeline(const std::vector<float>& natural) {
    const auto matrixElems = static_cast<size_t>(R_) * S_;
    const int images = static_cast<int>(natural.size() / matrixElems);
    const DeviceBuffer staged = upload_vector(natural);
    imageStride_ = images == 1 && groups() > 1 ? 0 : static_cast<long long>(tc_gemm_image_bytes(R_, S_));
    matrices_.allocate(static_cast<size_t>(images) * tc_gemm_image_bytes(R_, S_));
    check_cuda(tc_gemm_build_images(staged.get<float>(), images, R_, S_, p_ == GemmPrecision::bf16x3 ? 1 : 0,
                                    matrices_.get(), nullptr),
               "tensor-core GEMM operand images");
    check_cuda(cudaStreamSynchronize(nullptr), "tensor-core GEMM operand images");
    build_units(unitTiles_);
    error_.allocate(sizeof(int));
    check_cuda(cudaMemset(error_.get(), 0, sizeof(int)), "cudaMemset");
}

void VerticalPlan::use_pipeline_for_test() {
    if (!tensor_core()) throw Error(-1, "the tcgen05 pipeline serves the tensor-core GEMM forms");
    if (!smallGroups_) return;
    // The matrices back from their chunks [chunk][r][s of the chunk].
    const size_t imageElems = static_cast<size_t>(R_) * gemm_tf32_row(S_), count = matrices_.bytes() / sizeof(float);
    std::vector<float> stored(count), natural;
    check_cuda(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
    check_cuda(cudaMemcpy(stored.data(), matrices_.get(), matrices_.bytes(), cudaMemcpyDeviceToHost), "cudaMemcpy D2H");
    for (size_t image = 0; image < count; image += imageElems)
        for (int r = 0; r < R_; ++r)
            for (int s = 0; s < S_; ++s) {
                const int chunk = s / kGemmTf32Chunk, left = S_ - chunk * kGemmTf32Chunk;
                natural.push_back(stored[image + static_cast<size_t>(chunk) * gemm_tf32_chunk_row(kGemmTf32Chunk) * R_ +
                                         static_cast<size_t>(r) * gemm_tf32_chunk_row(left) + s % kGemmTf32Chunk]);
            }
    build_pipeline(natural);
    tileTables_.clear();
    smallGroups_ = false;
}

void VerticalPlan::set_expire_wait_for_test(bool on) {
    if (on) use_pipeline_for_test();
    expireWaitForTest_ = on;
}

// Units: runs of up to tiles * 64 virtual (member, column) pairs of one
// group, largest first so the long units start early.  One table per active
// member count so partial batches launch only their units.
void VerticalPlan::build_units(int tiles) {
    if (tiles < 1) throw Error(-1, "work units need at least one tile");
    struct Unit {
        int g, col, count;
    };
    int device = 0, sms = 0;
    check_cuda(cudaGetDevice(&device), "cudaGetDevice");
    check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "cudaDeviceGetAttribute");
    const int span = tiles * 64;
    std::vector<UnitTable> tables;
    for (std::uint64_t active = 1; active <= members_; ++active) {
        // A group's units (runs of <= `tiles` M-tiles of its member columns)
        // go to one CTA, so the CTA loads the group's operand image once; a
        // group with more than a CTA's share of the work is cut into pieces of
        // at most that share.  Pieces are dealt largest first to the CTA with
        // the least work so far (one tile of work per piece stands for its
        // image load), and each CTA walks its units as one contiguous range.
        struct Piece {
            std::vector<Unit> units;
            long long work = 0;
        };
        const int groups = static_cast<int>(groupColumnsHost_.size());
        long long totalTiles = 0;
        int unitCount = 0;
        for (int gi = 0; gi < groups; ++gi) {
            const int total = static_cast<int>(active) * groupColumnsHost_[gi];
            totalTiles += (total + 63) / 64;
            unitCount += (total + span - 1) / span;
        }
        const int ctas = std::max(1, std::min(unitCount, sms > 0 ? sms : 148));
        const long long share = std::max<long long>(tiles, (totalTiles + ctas - 1) / ctas);
        std::vector<Piece> pieces;
        for (int gi = 0; gi < groups; ++gi) {
            const int total = static_cast<int>(active) * groupColumnsHost_[gi];
            Piece cur;
            for (int col = 0; col < total; col += span) {
                const Unit u{gi, col, std::min(span, total - col)};
                const long long t = (u.count + 63) / 64;
                if (!cur.units.empty() && cur.work + t > share) {
                    cur.work += 1;
                    pieces.push_back(std::move(cur));
                    cur = Piece{};
                }
                cur.units.push_back(u);
                cur.work += t;
            }
            if (!cur.units.empty()) {
                cur.work += 1;
                pieces.push_back(std::move(cur));
            }
        }
        std::vector<int> order(pieces.size());
        for (size_t i = 0; i < order.size(); ++i) order[i] = static_cast<int>(i);
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return pieces[a].work > pieces[b].work; });
        std::vector<std::vector<int>> owned(ctas);
        // Least-loaded CTA by a min-heap of (load, cta).
        std::vector<std::pair<long long, int>> heap;
        for (int c = 0; c < ctas; ++c) heap.push_back({0, c});
        auto greater = [](const std::pair<long long, int>& a, const std::pair<long long, int>& b) { return a > b; };
        std::make_heap(heap.begin(), heap.end(), greater);
        for (const int pi : order) {
            std::pop_heap(heap.begin(), heap.end(), greater);
            auto& least = heap.back();
            owned[least.second].push_back(pi);
            least.first += pieces[pi].work;
            std::push_heap(heap.begin(), heap.end(), greater);
        }
        std::vector<int> ug, uc, un, first{0};
        for (int c = 0; c < ctas; ++c) {
            for (const int pi : owned[c])
                for (const Unit& u : pieces[pi].units) {
                    ug.push_back(u.g);
                    uc.push_back(u.col);
                    un.push_back(u.count);
                }
            first.push_back(static_cast<int>(ug.size()));
        }
        UnitTable table;
        table.units = static_cast<int>(ug.size());
        table.ctas = ctas;
        table.group = upload_vector(ug);
        table.column = upload_vector(uc);
        table.count = upload_vector(un);
        table.first = upload_vector(first);
        tables.push_back(std::move(table));
    }
    unitTables_ = std::move(tables);
    unitTiles_ = tiles;
}

void VerticalPlan::set_unit_tiles(int tiles) {
    if (!tensor_core()) throw Error(-3, "work-unit size applies to the tensor-core forms only");
    if (smallGroups_)
        unitTiles_ = tiles;  // no units: the choice has no effect
    else if (tiles != unitTiles_)
        build_units(tiles);
}

std::uint64_t VerticalPlan::persistentBytes() const {
    std::uint64_t units = 0;
    for (const auto& t : unitTables_) units += t.group.bytes() + t.column.bytes() + t.count.bytes() + t.first.bytes();
    for (const auto& t : tileTables_)
        units += t.group.bytes() + t.column.bytes() + t.count.bytes() + t.per.bytes() + t.first.bytes();
    return matrices_.bytes() + units +
           groupColumns_.bytes() + groupFirst_.bytes() + error_.bytes();
}

void VerticalPlan::execute(ComplexOperand in, ComplexOperand out, cudaStream_t s, std::uint64_t members,
                           const BinBoundary* inBins, const BinBoundary* outBins) const {
    if (members == 0) members = members_;
    if (members > members_) throw Error(-1, "more ensemble members than the plan was built for");
    if (tensor_core() && (in.im != nullptr || out.im != nullptr))
        throw Error(-3, "the tensor-core GEMM form takes interleaved complex operands");
    if (tensor_core() && !smallGroups_) {
        const UnitTable& table = unitTables_[members - 1];
        TcGemmArgs a{};
        a.B = matrices_.get<unsigned char>();
        a.imageStride = imageStride_;
        a.R = R_;
        a.S = S_;
        a.NP = (R_ + 15) / 16 * 16;
        a.KCH = (S_ + 31) / 32;
        a.unitGroup = table.group.get<int>();
        a.unitColumn = table.column.get<int>();
        a.unitCount = table.count.get<int>();
        a.units = table.units;
        a.ctaFirst = table.first.get<int>();
        a.ctas = table.ctas;
        a.groupColumns = groupColumns_.get<int>();
        a.groupFirst = groupFirst_.get<int>();
        a.memberColumns = memberColumns_;
        a.in = static_cast<const float2*>(in.re);
        a.out = static_cast<float2*>(out.re);
        a.error = error_.get<int>();
        a.expireWaitForTest = expireWaitForTest_ ? 1 : 0;
        a.kind = p_ == GemmPrecision::bf16x3 ? 1 : 0;
        if (inBins != nullptr) a.inBins = *inBins;
        if (outBins != nullptr) a.outBins = *outBins;
        check_cuda(launch_tc_gemm(a, s), "tensor-core grouped vertical GEMM kernel");
        return;
    }
    // SIMT tiles of the table for this member count; cell-addressed operands
    // decompose a tile column's global plan column into (member, mode, field)
    // with the plan's columns per member.
    const TileTable& table = tileTables_[virtualTiles_ ? members - 1 : 0];
    const GroupTiles t{table.group.get<int>(), table.column.get<int>(), table.count.get<int>(), table.per.get<int>(),
                       table.first.get<int>(), tilePrefix_[members - 1], memberColumns_, matrixStride_,
                       virtualTiles_};
    BinBoundary ib, ob;
    if (inBins != nullptr) {
        ib = *inBins;
        ib.memberColumns = memberColumns_;
    }
    if (outBins != nullptr) {
        ob = *outBins;
        ob.memberColumns = memberColumns_;
    }
    if (smallGroups_) {
        check_cuda(launch_grouped_gemm_tf32(R_, S_, matrices_.get<float>(), t, static_cast<const float2*>(in.re),
                                            static_cast<float2*>(out.re), ib, ob, s),
                   "split-TF32x3 grouped vertical GEMM kernel");
        return;
    }
    check_cuda(launch_grouped_gemm(p_, R_, S_, matrices_.get(), t, in, out, s, inBins ? &ib : nullptr,
                                   outBins ? &ob : nullptr),
               "grouped vertical GEMM kernel");
}

void VerticalPlan::check_device_error() const {
    if (error_.bytes() == 0) return;
    int flag = 0;
    check_cuda(cudaMemcpy(&flag, error_.get(), sizeof(int), cudaMemcpyDeviceToHost), "cudaMemcpy D2H");
    if (flag != 0) throw Error(-2, "tensor-core GEMM: a bounded device wait expired (MMA completion not observed)");
}

}  // namespace skb
