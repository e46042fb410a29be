#include "session.hpp"

#include "kernels/gemm_i8_tcgen05.hpp"

#include <algorithm>
#include <array>
#include <iterator>
#include <map>
#include <cstdlib>
#include <set>
#include <string>

namespace mlel {

namespace {
uint64_t roundUp(uint64_t v, uint64_t a) { return (v + a - 1) / a * a; }
} // namespace

Session::Session(GraphPipeline *pipeline) : pipeline_(pipeline) {
    pipeline_->finalize();
    plan();
    // Counters of the tile-level hand-over, if two tensor-core convolutions follow each other anywhere in the list.
    // Made here and not at the first dispatch, which may run inside a stream capture.  Without them (no
    // device, no memory) the dispatch simply does without the hand-over.
    const auto &exec = pipeline_->getExecList();
    // one counter per 128 output pixels (the narrowest tile) of every convolution whose output the next one reads, where both
    // are the channel-major kernel's: zeroing the counters is a node of its own at the head of a replayed graph, 2 to 5 us of
    // a pass that does not use them
    size_t words = 0;
    const auto pixelsOf = [&](const OpDesc &op) {
        const TensorDescriptor &out = pipeline_->tensor(op.out[0]);
        return out.dims.back() == 0 ? int64_t(0) : out.numel() / out.dims.back();
    };
    const auto channelMajor = [&](const OpDesc &op) {
        return op.tc != 0 && (op.kind == OP_CONV2D || op.kind == OP_FUSED_CONV2D) && !op.out.empty() && !op.in.empty() &&
               gemmI8OcMajorMayTake(pixelsOf(op), pipeline_->tensor(op.out[0]).dims.back());
    };
    for (size_t k = 0; k + 1 < exec.size(); ++k) {
        if (channelMajor(exec[k]) && channelMajor(exec[k + 1]) && exec[k + 1].in[0] == exec[k].out[0]) {
            words += size_t((pixelsOf(exec[k]) + 127) / 128);
        }
    }
    if (words != 0 && (cudaMalloc(&progressWords_, words * sizeof(uint32_t)) != cudaSuccess ||
                       cudaMemset(progressWords_, 0, words * sizeof(uint32_t)) != cudaSuccess)) {
        if (progressWords_ != nullptr) {
            cudaFree(progressWords_);
        }
        progressWords_ = nullptr;
        cudaGetLastError();
    }
    progressCapacity_ = progressWords_ != nullptr ? words : 0;
}

void Session::dropCaptureStream() {
    if (captureStream_ != nullptr) {
        cudaStreamDestroy(captureStream_);
        captureStream_ = nullptr;
    }
}

Session::~Session() {
    dropGraphs();
    dropCaptureStream();
    if (progressWords_ != nullptr) {
        cudaFree(progressWords_);
    }
}

void Session::dropGraphs() {
    for (auto &entry : graphs_) {
        if (entry.second.exec != nullptr) {
            cudaGraphExecDestroy(entry.second.exec);
        }
        if (entry.second.graph != nullptr) {
            cudaGraphDestroy(entry.second.graph);
        }
    }
    graphs_.clear();
}

std::vector<const void *> Session::bindingKey() const {
    std::vector<const void *> key{memory_};
    for (const auto &entry : external_) {
        key.push_back(entry.second);
    }
    return key;
}

// Live range of a session tensor = [first, last] execution index over {inputs node = 0,
// operators 1..n, outputs node = n + 1} that touch it (graph/interval_memory_planner.cpp:53-115).
// The operator list used is the one that is actually launched: with fusion on, an elided
// intermediate is touched by nothing and the fused node keeps its inputs alive until it runs.
void Session::plan() {
    const auto &exec = pipeline_->getExecList();
    const auto &sessionTensors = pipeline_->getTensors();
    std::map<int32_t, std::pair<uint32_t, uint32_t>> ranges;
    const auto touch = [&](int32_t t, uint32_t index) {
        if (t < 0 || pipeline_->tensor(t).cls != TensorClass::Session) {
            return;
        }
        auto it = ranges.find(t);
        if (it == ranges.end()) {
            ranges[t] = {index, index};
        } else {
            it->second.first = std::min(it->second.first, index);
            it->second.second = std::max(it->second.second, index);
        }
    };
    uint32_t index = 0;
    for (auto t : pipeline_->graphInputs()) {
        touch(t, index);
    }
    ++index;
    for (const auto &op : exec) {
        for (auto t : op.in) {
            touch(t, index);
        }
        for (auto t : op.out) {
            touch(t, index);
        }
        touch(op.epi.shortcutTensor, index);
        touch(op.scratch, index);
        ++index;
    }
    for (auto t : pipeline_->graphOutputs()) {
        touch(t, index);
    }

    // With fusion on, a RESHAPE between two packed session tensors of one size moves no bytes: its result shares
    // its input's storage (the launch skips the copy when both addresses are equal), and the shared storage
    // lives as long as either tensor.  Chains of such RESHAPEs resolve to the first tensor.
    std::map<int32_t, int32_t> aliasOf;
    if (!(pipeline_->flags() & MLEL_PIPELINE_NO_FUSION)) {
        for (const auto &op : exec) {
            if (op.kind != OP_RESHAPE || op.in.empty() || op.out.empty()) {
                continue;
            }
            const int32_t src = op.in[0], dst = op.out[0];
            if (src < 0 || dst < 0 || src == dst) {
                continue;
            }
            const TensorDescriptor &a = pipeline_->tensor(src), &b = pipeline_->tensor(dst);
            if (a.cls != TensorClass::Session || b.cls != TensorClass::Session || !a.packed() || !b.packed() ||
                a.dtype != b.dtype || a.sizeBytes() != b.sizeBytes()) {
                continue;
            }
            const auto rootIt = aliasOf.find(src);
            const int32_t root = rootIt != aliasOf.end() ? rootIt->second : src;
            if (!ranges.count(root) || !ranges.count(dst)) {
                continue;
            }
            aliasOf[dst] = root;
            auto &r = ranges[root];
            const auto d = ranges[dst];
            r.first = std::min(r.first, d.first);
            r.second = std::max(r.second, d.second);
            ranges.erase(dst);
        }
    }

    // One record per session tensor that needs storage, in session-tensor order.
    planned_.clear();
    for (size_t order = 0; order < sessionTensors.size(); ++order) {
        const int32_t t = sessionTensors[order];
        const uint64_t size = roundUp(pipeline_->tensor(t).sizeBytes(), kSessionAlignment);
        const auto it = ranges.find(t);
        if (it != ranges.end()) {
            planned_.push_back({t, 0, size, it->second.first, it->second.second, true});
        } else if (pipeline_->flags() & MLEL_PIPELINE_NO_FUSION) {
            planned_.push_back({t, 0, size, 0, 0, false});
        }
        // With fusion on, a tensor nothing touches was elided and needs no storage.
    }
    planner_ = plannerFromEnvironment();
    switch (planner_) {
    case PlannerKind::Linear:
        planLinear();
        break;
    case PlannerKind::BestFit:
        planBestFit();
        break;
    case PlannerKind::Interval:
        planInterval();
        break;
    }
    offsets_.clear();
    for (const auto &p : planned_) {
        offsets_[p.tensor] = p.offset;
    }
    for (const auto &alias : aliasOf) {
        const auto it = offsets_.find(alias.second);
        if (it != offsets_.end()) {
            offsets_[alias.first] = it->second;
        }
    }
}

// The session's planner is chosen by VMEL_MEMORY_PLANNER exactly as the reference chooses it
// (graph/graph_layer.cpp:282-297): "Linear", "BestFit", anything else (or unset) = interval.
PlannerKind plannerFromEnvironment() {
    const char *name = std::getenv("VMEL_MEMORY_PLANNER");
    if (name != nullptr && std::string(name) == "Linear") {
        return PlannerKind::Linear;
    }
    if (name != nullptr && std::string(name) == "BestFit") {
        return PlannerKind::BestFit;
    }
    return PlannerKind::Interval;
}

const char *plannerName(PlannerKind kind) {
    switch (kind) {
    case PlannerKind::Linear:
        return "Linear";
    case PlannerKind::BestFit:
        return "BestFit";
    case PlannerKind::Interval:
        break;
    }
    return "Interval";
}

void Session::planInterval() {
    std::vector<LiveInterval> intervals;
    std::vector<UnseenAllocation> unseen;
    for (size_t k = 0; k < planned_.size(); ++k) {
        const auto &p = planned_[k];
        if (p.seen) {
            intervals.push_back({uint64_t(k), p.first, p.last, p.size, uint64_t(k)});
        } else {
            unseen.push_back({uint64_t(k), p.size});
        }
    }
    const AllocationPlan plan = allocateIntervals(std::move(intervals), unseen, kSessionAlignment);
    memorySize_ = plan.memorySize;
    for (const auto &[k, offset] : plan.offsets) {
        planned_[size_t(k)].offset = offset;
    }
}

// Every tensor gets storage of its own, one after the other (LinearMemoryPlanner,
// graph/memory_planner.cpp:52-98).  Sizes are already multiples of the alignment.
void Session::planLinear() {
    uint64_t offset = 0;
    for (auto &p : planned_) {
        p.offset = offset;
        offset += p.size;
    }
    memorySize_ = offset;
}

// Best fit (BestFitMemoryPlanner, graph/memory_planner.cpp:239-263, 284-310, 352-381): tensors are
// taken largest first; each looks, among the already placed tensors that are at least as large and
// that it may share memory with, for the smallest one whose slot holds only tensors it may share
// with, and moves in at that slot's address; if there is none it opens a new slot at the end.
// Two tensors may share memory when their live ranges over the launched operator list do not
// intersect -- the relation the reference derives by passing tensor references along the graph's
// edges (memory_planner.cpp:154-237) stated on the linear execution order that a stream gives.
// A tensor no operator touches never shares.
void Session::planBestFit() {
    std::vector<size_t> order(planned_.size());
    for (size_t k = 0; k < order.size(); ++k) {
        order[k] = k;
    }
    std::stable_sort(order.begin(), order.end(),
                     [&](size_t a, size_t b) { return planned_[a].size > planned_[b].size; });
    const auto mayShare = [&](size_t a, size_t b) {
        const auto &x = planned_[a];
        const auto &y = planned_[b];
        return x.seen && y.seen && (x.last < y.first || y.last < x.first);
    };
    std::vector<int> slotOf(planned_.size(), -1);
    std::vector<std::vector<size_t>> slots; // occupants of each slot; all share the slot's address
    std::vector<size_t> placed;             // tensors placed so far, smallest first (stable)
    uint64_t end = 0;
    for (const size_t k : order) {
        int chosen = -1;
        for (const size_t alt : placed) {
            if (planned_[alt].size < planned_[k].size || !mayShare(k, alt)) {
                continue;
            }
            const auto &occupants = slots[size_t(slotOf[alt])];
            if (std::all_of(occupants.begin(), occupants.end(), [&](size_t o) { return mayShare(k, o); })) {
                chosen = slotOf[alt];
                planned_[k].offset = planned_[alt].offset;
                break;
            }
        }
        if (chosen < 0) {
            chosen = int(slots.size());
            slots.emplace_back();
            planned_[k].offset = end;
            end += planned_[k].size;
        }
        slotOf[k] = chosen;
        slots[size_t(chosen)].push_back(k);
        // keep `placed` sorted by size ascending; among equal sizes earlier placements come first
        const auto pos = std::upper_bound(placed.begin(), placed.end(), k, [&](size_t a, size_t b) {
            return planned_[a].size < planned_[b].size;
        });
        placed.insert(pos, k);
    }
    memorySize_ = end;
}

bool Session::tensorOffset(int32_t tensor, uint64_t *offset) const {
    const auto it = offsets_.find(tensor);
    if (it == offsets_.end()) {
        return false;
    }
    *offset = it->second;
    return true;
}

void Session::bindMemory(void *memory, uint64_t offset) {
    memory_ = static_cast<char *>(memory) + offset;
    resolved_ = false;
}

void Session::setExternal(uint32_t set, uint32_t binding, uint32_t arrayIndex, void *devicePtr) {
    (void)pipeline_->getTensor(set, binding, arrayIndex); // throws std::out_of_range when unknown
    char *&slot = external_[std::make_tuple(set, binding, arrayIndex)];
    if (slot != static_cast<char *>(devicePtr)) {
        slot = static_cast<char *>(devicePtr);
        resolved_ = false;
    }
}

int Session::resolve() {
    if (resolved_) {
        return MLEL_SUCCESS;
    }
    const int32_t n = pipeline_->tensorCount();
    views_.assign(size_t(n), TView{});
    char *constBase = pipeline_->constantBase();
    // Only tensors some launched operator touches must be bound.
    std::set<int32_t> used;
    for (const auto &op : pipeline_->getExecList()) {
        used.insert(op.in.begin(), op.in.end());
        used.insert(op.out.begin(), op.out.end());
        for (const FusedRescale *f : {&op.epi.main, &op.epi.a, &op.epi.b, &op.epi.out}) {
            used.insert(f->multTensor);
            used.insert(f->shiftTensor);
        }
        used.insert(op.epi.shortcutTensor);
        used.insert(op.epi.tableTensor);
        used.insert(std::begin(op.aux), std::end(op.aux));
        used.insert(op.scratch);
    }
    used.erase(-1);
    for (int32_t t = 0; t < n; ++t) {
        const TensorDescriptor &td = pipeline_->tensor(t);
        TView &v = views_[size_t(t)];
        v.dtype = td.dtype;
        v.rank = td.rank();
        for (int i = 0; i < td.rank(); ++i) {
            v.dims[i] = uint32_t(td.dims[size_t(i)]);
            v.strides[i] = td.strides[size_t(i)];
        }
        switch (td.cls) {
        case TensorClass::Constant:
            v.ptr = constBase + td.constOffset;
            break;
        case TensorClass::Session: {
            const auto it = offsets_.find(t);
            if (it != offsets_.end()) {
                if (memory_ == nullptr && used.count(t)) {
                    setLastError("session memory is not bound");
                    return MLEL_ERROR_UNKNOWN;
                }
                v.ptr = memory_ + it->second;
            }
            break;
        }
        case TensorClass::External: {
            const auto it = external_.find(std::make_tuple(td.set, td.binding, td.arrayIndex));
            if (it == external_.end() || it->second == nullptr) {
                if (used.count(t)) {
                    setLastError("external tensor (set " + std::to_string(td.set) + ", binding " +
                                 std::to_string(td.binding) + ", element " + std::to_string(td.arrayIndex) +
                                 ") is not bound");
                    return MLEL_ERROR_UNKNOWN;
                }
            } else {
                v.ptr = it->second;
            }
            break;
        }
        }
    }
    resolved_ = true;
    return MLEL_SUCCESS;
}

int Session::dispatch(cudaStream_t stream) {
    const int rc = resolve();
    if (rc != MLEL_SUCCESS) {
        return rc;
    }
    // Operators run in creation order on one stream: the stream order is the full
    // write-to-read barrier the reference records between consecutive dispatches
    // (graph/compute_graph_op.cpp:251-299).
    const auto &exec = pipeline_->getExecList();
    GraphProfiler *profiler = pipeline_->profiler();
    if (profiler != nullptr) {
        // The reference wraps every operator's dispatch in a pair of timestamp writes when profiling is on
        // (graph/graph_profiler.cpp:157-191); one event after each kernel closes it and opens the next.
        const size_t token = profiler->beginDispatch(stream, exec.size());
        for (size_t k = 0; k < exec.size(); ++k) {
            const int r = launchOp(exec[k], views_.data(), stream);
            if (r != MLEL_SUCCESS) {
                return r;
            }
            profiler->afterOperator(token, uint32_t(k), exec[k].name, stream);
        }
        return MLEL_SUCCESS;
    }
    // Consecutive convolutions hand their output over tile by tile where the kernels can (LaunchChain).  The
    // counters are the session's own (allocated with the session), zeroed in stream order before the first kernel.
    LaunchChain chain{};
    if (progressWords_ != nullptr) {
        if (cudaMemsetAsync(progressWords_, 0, progressCapacity_ * sizeof(uint32_t), stream) != cudaSuccess) {
            setLastError("cudaMemsetAsync of the progress counters failed");
            return MLEL_ERROR_DEVICE;
        }
        chain.words = progressWords_;
        chain.capacity = progressCapacity_;
    }
    for (size_t k = 0; k < exec.size(); ++k) {
        const int r = enqueueOp(k, chain.words != nullptr ? &chain : nullptr, stream);
        if (r != MLEL_SUCCESS) {
            return r;
        }
    }
    return MLEL_SUCCESS;
}

int Session::enqueueOp(size_t k, LaunchChain *chain, cudaStream_t stream) {
    const auto &exec = pipeline_->getExecList();
    const OpDesc &op = exec[k];
    if (chain != nullptr) {
        // does the next operator read this one's output as the pixel operand of a tensor-core convolution?
        chain->publishNext = k + 1 < exec.size() && exec[k + 1].tc != 0 &&
                             (exec[k + 1].kind == OP_CONV2D || exec[k + 1].kind == OP_FUSED_CONV2D) && !op.out.empty() &&
                             !exec[k + 1].in.empty() && exec[k + 1].in[0] == op.out[0];
    }
    return launchOp(op, views_.data(), stream, chain);
}

namespace {

// Bytes that a tensor's elements lie in; empty for an address that is not bound.
struct ByteRange {
    uintptr_t begin, end;
};
ByteRange bytesOf(const TView &v, uint64_t elementBytes) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(v.ptr);
    if (at == 0) {
        return {0, 0};
    }
    int64_t low = 0, high = 0;
    for (int i = 0; i < v.rank; ++i) {
        const int64_t reach = v.dims[i] > 0 ? int64_t(v.dims[i] - 1) * v.strides[i] : 0;
        (reach < 0 ? low : high) += reach;
    }
    return {at + uintptr_t(low), at + uintptr_t(high) + uintptr_t(elementBytes)};
}
// Who wrote bytes last and who has read them since, for operators taken in order.
class Hazards {
  public:
    // Calls f(piece) for the pieces that make up the range.
    struct Piece {
        uintptr_t end;
        size_t writer = SIZE_MAX;
        std::vector<size_t> readers;
    };
    template <class F> void over(const ByteRange &r, F &&f) {
        cut(r.begin);
        cut(r.end);
        uintptr_t at = r.begin;
        for (auto it = pieces_.lower_bound(r.begin); at < r.end; ++it) {
            if (it == pieces_.end() || it->first > at) { // bytes that no operator has touched
                const uintptr_t end = it == pieces_.end() ? r.end : std::min(r.end, it->first);
                it = pieces_.emplace_hint(it, at, Piece{end, SIZE_MAX, {}});
            }
            f(it->second);
            at = it->second.end;
        }
    }

  private:
    void cut(uintptr_t at) {
        auto it = pieces_.lower_bound(at);
        if (it == pieces_.begin() || (it != pieces_.end() && it->first == at)) {
            return;
        }
        Piece &piece = std::prev(it)->second;
        if (piece.end > at) {
            pieces_.emplace_hint(it, at, piece); // (a copy that ends where the piece did)
            piece.end = at;
        }
    }
    std::map<uintptr_t, Piece> pieces_; // by first byte, disjoint
};
// Kernels that pace themselves by dependent launches, or that chains of those run through.
bool isPaced(const OpDesc &op) {
    return op.tc != 0 || op.kind == OP_FUSED_ATTENTION || op.kind == OP_FUSED_ROWS;
}

} // namespace

// For every one of these operators the earlier ones (as positions in the list, ascending) that it has to follow: who wrote last what
// it reads or overwrites, and who has read since what it overwrites; what these follow themselves is not named again.  By address,
// so that tensors which the session or the application placed over one another count.
std::vector<std::vector<size_t>> Session::branches(const std::vector<size_t> &ops) const {
    const auto &exec = pipeline_->getExecList();
    std::vector<std::vector<size_t>> before(ops.size());
    std::vector<ByteRange> reads, writes;
    Hazards hazards;
    for (size_t k = 0; k < ops.size(); ++k) {
        const OpDesc &op = exec[ops[k]];
        const auto add = [&](std::vector<ByteRange> &list, int32_t t) {
            if (t >= 0 && pipeline_->tensor(t).cls != TensorClass::Constant) {
                const ByteRange r = bytesOf(views_[size_t(t)], elemSize(views_[size_t(t)].dtype));
                if (r.begin < r.end) {
                    list.push_back(r);
                }
            }
        };
        reads.clear(), writes.clear();
        for (const int32_t t : op.in) {
            add(reads, t);
        }
        add(reads, op.epi.shortcutTensor);
        for (const int32_t t : op.out) {
            add(writes, t);
        }
        add(writes, op.scratch);
        std::vector<size_t> &list = before[k];
        const auto follow = [&](size_t earlier) {
            if (earlier != SIZE_MAX && earlier != k) {
                list.push_back(earlier);
            }
        };
        for (const ByteRange &r : reads) {
            hazards.over(r, [&](Hazards::Piece &piece) {
                follow(piece.writer);
                if (piece.readers.empty() || piece.readers.back() != k) {
                    piece.readers.push_back(k);
                }
            });
        }
        for (const ByteRange &r : writes) {
            hazards.over(r, [&](Hazards::Piece &piece) {
                follow(piece.writer);
                std::for_each(piece.readers.begin(), piece.readers.end(), follow);
                piece.writer = k;
                piece.readers.clear();
            });
        }
        std::sort(list.begin(), list.end());
        list.erase(std::unique(list.begin(), list.end()), list.end());
    }
    return before;
}

// Four lanes for a stretch of operators: which earlier ones each follows by an edge, and whether that is quicker than one after the
// other by enough.
//
// Times are counted in bytes, a launch as 12 MB (2 us).  In a row they add up; on lanes the longest path through the edges counts, but
// no less than all bytes take together.  Lanes are taken from a sixteenth less on: of 56 stretches of 2 to 12 operators with that much
// (tensors of 4 KB to 17 MB, 2 to 4 chains) none was slower on lanes, most took 0.45 to 0.85 of the time; but they add 0.04 (two
// lanes) to 0.14 ms (four) to the capture, once per set of addresses, which 50 operators that mostly follow one another (57.4 us
// in a row, 56.6 on lanes) would not earn.
Session::LanePlan Session::planLanes(const std::vector<size_t> &ops) const {
    constexpr uint64_t kLaunch = uint64_t(12) << 20;
    const auto &exec = pipeline_->getExecList();
    const std::vector<std::vector<size_t>> before = branches(ops);
    LanePlan plan;
    plan.after.resize(ops.size());
    std::vector<size_t> laneOf(ops.size());
    std::array<size_t, kLanes> tail;
    std::array<uint64_t, kLanes> load{};
    tail.fill(SIZE_MAX);
    // of every operator the last one of each lane that precedes it (or is it), plus one: an edge is laid only from operators
    // that no other edge implies (with all of them 400 operators on four chains replayed in 1730 us instead of 430)
    std::vector<std::array<size_t, kLanes>> known(ops.size());
    std::vector<uint64_t> finish(ops.size());
    uint64_t inARow = 0, bytes = 0, longest = 0;
    for (size_t j = 0; j < ops.size(); ++j) {
        // An operator goes on where the last one that it follows ended, or else on the lane with the least to do.
        size_t lane = size_t(std::min_element(load.begin(), load.end()) - load.begin());
        for (size_t l = 0; l < kLanes; ++l) {
            if (!before[j].empty() && tail[l] == before[j].back()) {
                lane = l;
            }
        }
        std::array<size_t, kLanes> &mine = known[j];
        mine.fill(0);
        uint64_t start = 0;
        const auto edgeFrom = [&](size_t b) {
            if (mine[laneOf[b]] <= b) {
                plan.after[j].push_back(b);
                start = std::max(start, finish[b]);
                for (size_t l = 0; l < kLanes; ++l) {
                    mine[l] = std::max(mine[l], known[b][l]);
                }
            }
        };
        if (tail[lane] != SIZE_MAX) {
            edgeFrom(tail[lane]);
        }
        std::for_each(before[j].rbegin(), before[j].rend(), edgeFrom); // (the last ones imply most)
        tail[lane] = j, laneOf[j] = lane, mine[lane] = j + 1;
        uint64_t moved = 0;
        for (const auto *list : {&exec[ops[j]].in, &exec[ops[j]].out}) {
            for (const int32_t t : *list) {
                moved += t >= 0 ? pipeline_->tensor(t).sizeBytes() : 0;
            }
        }
        bytes += moved, inARow += kLaunch + moved, load[lane] += kLaunch + moved;
        finish[j] = start + kLaunch + moved;
        longest = std::max(longest, finish[j]);
    }
    plan.pays = 16 * std::max(longest, bytes) <= 15 * inARow;
    return plan;
}

int Session::capture(cudaStream_t stream) {
    // Operators that neither run on the tensor cores nor belong to the row kernels -- element-wise ones, pools, reductions,
    // movement -- are short or bound by memory, and one after the other each waits for the last block of the one before it
    // and starts anew.  Where it pays (planLanes) a stretch of them is laid on four lanes, and an operator follows those
    // whose bytes it touches and the one before it on its lane (stream order is a full barrier like the one that the
    // reference records, graph/compute_graph_op.cpp:251-299; what it guarantees to the results are the former edges).
    // Twelve operators without dependencies, small and large tensors, on 1, 2, 3, 4, 6 and 12 lanes: 30.7, 19.9, 18.4, 17.2,
    // 17.8, 34.4 and 228, 203, 205, 202, 207, 216 us: a replayed graph pays for every root and every join.
    // Elsewhere consecutive launches overlap by dependent launches, which beat edges of this kind.
    const auto &exec = pipeline_->getExecList();
    LaunchChain chain{};
    if (progressWords_ != nullptr) {
        if (cudaMemsetAsync(progressWords_, 0, progressCapacity_ * sizeof(uint32_t), stream) != cudaSuccess) {
            setLastError("cudaMemsetAsync of the progress counters failed");
            return MLEL_ERROR_DEVICE;
        }
        chain.words = progressWords_;
        chain.capacity = progressCapacity_;
    }
    LaunchChain *const chainOrNull = chain.words != nullptr ? &chain : nullptr;
    const auto leaves = [&](std::vector<cudaGraphNode_t> *out) {
        cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
        const cudaGraphNode_t *nodes = nullptr;
        size_t count = 0;
        if (cudaStreamGetCaptureInfo_v2(stream, &status, nullptr, nullptr, &nodes, &count) != cudaSuccess) {
            return false;
        }
        out->assign(nodes, nodes + count);
        return true;
    };
    const auto follow = [&](std::vector<cudaGraphNode_t> &nodes) {
        return cudaStreamUpdateCaptureDependencies(stream, nodes.data(), nodes.size(), cudaStreamSetCaptureDependencies) == cudaSuccess;
    };
    // (a RESHAPE within one storage launches nothing)
    const auto launches = [&](const OpDesc &op) {
        return op.kind != OP_RESHAPE || views_[size_t(op.in[0])].ptr != views_[size_t(op.out[0])].ptr;
    };
    bool joined = false; // several nodes precede the next launch
    for (size_t k = 0; k < exec.size();) {
        size_t end = k;
        std::vector<size_t> ops;
        for (; end < exec.size() && !isPaced(exec[end]); ++end) {
            if (launches(exec[end])) {
                ops.push_back(end);
            }
        }
        const LanePlan plan = ops.size() < 2 ? LanePlan{} : planLanes(ops);
        if (!plan.pays) {
            for (const size_t last = std::max(end, k + 1); k < last; ++k) {
                const PlainLaunches plain(joined);
                const int r = enqueueOp(k, chainOrNull, stream);
                if (r != MLEL_SUCCESS) {
                    return r;
                }
                joined = joined && !launches(exec[k]);
            }
            continue;
        }
        std::vector<cudaGraphNode_t> entry;
        std::vector<std::vector<cudaGraphNode_t>> exits(ops.size());
        std::vector<bool> followed(ops.size(), false);
        const auto failed = [&] {
            setLastError("CUDA graph capture: dependencies refused");
            return MLEL_ERROR_DEVICE;
        };
        if (!leaves(&entry)) {
            return failed();
        }
        const PlainLaunches plain(true);
        for (size_t j = 0; j < ops.size(); ++j) {
            const std::vector<size_t> &after = plan.after[j];
            std::vector<cudaGraphNode_t> from = after.empty() ? entry : std::vector<cudaGraphNode_t>{};
            for (const size_t b : after) {
                from.insert(from.end(), exits[b].begin(), exits[b].end());
                followed[b] = true;
            }
            std::sort(from.begin(), from.end());
            from.erase(std::unique(from.begin(), from.end()), from.end());
            if (!follow(from)) {
                return failed();
            }
            const int r = enqueueOp(ops[j], chainOrNull, stream);
            if (r != MLEL_SUCCESS) {
                return r;
            }
            if (!leaves(&exits[j])) {
                return failed();
            }
        }
        std::vector<cudaGraphNode_t> last;
        for (size_t j = 0; j < ops.size(); ++j) {
            if (!followed[j]) {
                last.insert(last.end(), exits[j].begin(), exits[j].end());
            }
        }
        std::sort(last.begin(), last.end());
        last.erase(std::unique(last.begin(), last.end()), last.end());
        if (!follow(last)) {
            return failed();
        }
        joined = true;
        k = end;
    }
    return MLEL_SUCCESS;
}

int Session::dispatchProfiled(cudaStream_t stream, float *msOut, uint32_t capacity) {
    const int rc = resolve();
    if (rc != MLEL_SUCCESS) {
        return rc;
    }
    const auto &exec = pipeline_->getExecList();
    if (capacity < exec.size()) {
        setLastError("dispatch_profiled: output array too short");
        return MLEL_INCOMPLETE;
    }
    std::vector<cudaEvent_t> events(exec.size() + 1);
    for (auto &e : events) {
        cudaEventCreate(&e);
    }
    int result = MLEL_SUCCESS;
    cudaEventRecord(events[0], stream);
    for (size_t k = 0; k < exec.size() && result == MLEL_SUCCESS; ++k) {
        result = launchOp(exec[k], views_.data(), stream);
        cudaEventRecord(events[k + 1], stream);
    }
    if (cudaStreamSynchronize(stream) != cudaSuccess && result == MLEL_SUCCESS) {
        setLastError("dispatch_profiled: stream synchronisation failed");
        result = MLEL_ERROR_DEVICE;
    }
    for (size_t k = 0; k < exec.size() && result == MLEL_SUCCESS; ++k) {
        cudaEventElapsedTime(&msOut[k], events[k], events[k + 1]);
    }
    for (auto &e : events) {
        cudaEventDestroy(e);
    }
    return result;
}

int Session::dispatchGraph(cudaStream_t stream) {
    if (pipeline_->profiler() != nullptr) {
        return dispatch(stream); // timestamps go between the kernels, which a replayed graph has no place for
    }
    int rc = resolve();
    if (rc != MLEL_SUCCESS) {
        return rc;
    }
    // One or two kernels are enqueued quicker than a graph of them is launched: back to back 5.4 against 8.2 us for a small
    // convolution, 6.4 against 8.2 for one with a padded copy, 5.6 against 8.2 and 10.3 against 12.3 for products of two
    // activations -- a replay begins on a whole number of 2.048 us (see launch_overlapped.cuh), launches behind one another do not.
    // Three (copied rows besides) keep the host 8 us, and a replay takes 6.2, 8.2 or 10.3: enqueued where all three depend on one
    // another, 15 of 15 products 1.03 to 1.3 times as fast (4 x 17 x 55 x 384 7.95 and 9.3, 4 x 43 x 18 x 224 8.0 and 8.2, 5 x 189 x 99 x 640
    // 8.6 and 10.3); replayed where the second operand is transposed first (2 x 40 x 30 x 64 7.7 and 6.2, 3 x 138 x 253 x 438 12.3 and
    // 10.4; of 42 products 21 the one way, 21 the other) or a TABLE follows.
    const auto &exec = pipeline_->getExecList();
    if (exec.size() == 1) {
        const OpDesc &op = exec[0];
        const int launches = op.scratch < 0 ? 1 : contractionLaunches(op, views_.data());
        if (launches <= 2 || (launches == 3 && launchesAllDepend(op, views_.data()))) {
            return dispatch(stream);
        }
        // (a stream that is being captured takes kernels, not the launch of a graph)
        cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(stream, &status) == cudaSuccess && status == cudaStreamCaptureStatusActive) {
            return dispatch(stream);
        }
    }
    // A captured graph holds the addresses that were bound when it was taken: one graph per set of bindings.
    constexpr size_t kMaxCapturedGraphs = 64;
    const std::vector<const void *> key = bindingKey();
    auto found = graphs_.find(key);
    if (found == graphs_.end()) {
        if (graphs_.size() >= kMaxCapturedGraphs) {
            // Make room for one: the entry that was launched longest ago goes.  Its last launch may still be running
            // on the caller's stream, so wait for that stream before the executable graph is destroyed.
            auto oldest = graphs_.begin();
            for (auto it = graphs_.begin(); it != graphs_.end(); ++it) {
                if (it->second.lastUse < oldest->second.lastUse) {
                    oldest = it;
                }
            }
            cudaStreamSynchronize(stream);
            if (oldest->second.exec != nullptr) {
                cudaGraphExecDestroy(oldest->second.exec);
            }
            if (oldest->second.graph != nullptr) {
                cudaGraphDestroy(oldest->second.graph);
            }
            graphs_.erase(oldest);
        }
        // The stream that takes the capture stays with the session: to make and to destroy one costs 0.11 ms, as much as a third of
        // a first dispatch.
        int device = 0;
        if (cudaGetDevice(&device) != cudaSuccess || (captureStream_ != nullptr && device != captureDevice_)) {
            dropCaptureStream();
        }
        if (captureStream_ == nullptr) {
            if (cudaStreamCreateWithFlags(&captureStream_, cudaStreamNonBlocking) != cudaSuccess) {
                captureStream_ = nullptr;
                setLastError("cudaStreamCreate failed");
                return MLEL_ERROR_DEVICE;
            }
            captureDevice_ = device;
        }
        CapturedGraph captured;
        cudaError_t err = cudaStreamBeginCapture(captureStream_, cudaStreamCaptureModeThreadLocal);
        if (err == cudaSuccess) {
            rc = capture(captureStream_);
            err = cudaStreamEndCapture(captureStream_, &captured.graph);
        }
        if (err == cudaSuccess && rc == MLEL_SUCCESS) {
            err = cudaGraphInstantiate(&captured.exec, captured.graph, 0);
        }
        if (rc != MLEL_SUCCESS || err != cudaSuccess) {
            if (captured.exec != nullptr) {
                cudaGraphExecDestroy(captured.exec);
            }
            if (captured.graph != nullptr) {
                cudaGraphDestroy(captured.graph);
            }
            if (rc != MLEL_SUCCESS) {
                return rc;
            }
            setLastError(std::string("CUDA graph capture failed: ") + cudaGetErrorString(err));
            return MLEL_ERROR_DEVICE;
        }
        found = graphs_.emplace(key, captured).first;
    }
    found->second.lastUse = ++useCounter_;
    if (cudaGraphLaunch(found->second.exec, stream) != cudaSuccess) {
        setLastError("cudaGraphLaunch failed");
        return MLEL_ERROR_DEVICE;
    }
    return MLEL_SUCCESS;
}

int Session::runHost(const mlel_host_io *inputs, uint32_t nIn, const mlel_host_io *outputs, uint32_t nOut,
                     cudaStream_t stream) {
    int rc = resolve();
    if (rc != MLEL_SUCCESS) {
        return rc;
    }
    const auto devPtr = [&](const mlel_host_io &io, uint64_t *bytes) -> char * {
        const int32_t t = pipeline_->getTensor(io.set, io.binding, io.array_index);
        *bytes = pipeline_->tensor(t).sizeBytes();
        return views_[size_t(t)].ptr;
    };
    for (uint32_t k = 0; k < nIn; ++k) {
        uint64_t bytes = 0;
        char *d = devPtr(inputs[k], &bytes);
        if (d == nullptr || inputs[k].bytes != bytes) {
            setLastError("run_host: input size does not match the bound tensor");
            return MLEL_ERROR_UNKNOWN;
        }
        if (cudaMemcpyAsync(d, inputs[k].host_ptr, bytes, cudaMemcpyHostToDevice, stream) != cudaSuccess) {
            setLastError("run_host: host-to-device copy failed");
            return MLEL_ERROR_DEVICE;
        }
    }
    rc = dispatchGraph(stream);
    if (rc != MLEL_SUCCESS) {
        return rc;
    }
    for (uint32_t k = 0; k < nOut; ++k) {
        uint64_t bytes = 0;
        char *d = devPtr(outputs[k], &bytes);
        if (d == nullptr || outputs[k].bytes != bytes) {
            setLastError("run_host: output size does not match the bound tensor");
            return MLEL_ERROR_UNKNOWN;
        }
        if (cudaMemcpyAsync(outputs[k].host_ptr, d, bytes, cudaMemcpyDeviceToHost, stream) != cudaSuccess) {
            setLastError("run_host: device-to-host copy failed");
            return MLEL_ERROR_DEVICE;
        }
    }
    if (cudaStreamSynchronize(stream) != cudaSuccess) {
        setLastError(std::string("run_host: ") + cudaGetErrorString(cudaGetLastError()));
        return MLEL_ERROR_DEVICE;
    }
    return MLEL_SUCCESS;
}

} // namespace mlel
