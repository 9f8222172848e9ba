// Serving loop: requests (NTT, BGV encryption, ciphertext x ciphertext) are
// submitted from any host thread and return a ticket; a scheduler thread
// batches compatible pending requests as device lanes (streams) and memory
// free up, so work of requests that arrive while others run overlaps on the
// device (continuous batching).
//
// Admission is by device memory: the server reserves one pool at creation and
// every dispatch takes its scratch from it; a dispatch waits until its
// scratch fits, and a request whose scratch can never fit is rejected.  Keys
// and twiddle tables stay resident.  Every request's result is the result it
// would have alone: transforms and products have no state, and an encryption
// draws its randomness from its own nonce with coefficient indices local to
// the request (per-polynomial descriptors), whatever batch it lands in.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <map>
#include <memory>
#include <mutex>
#include <thread>
#include <tuple>
#include <unordered_map>
#include <vector>

#include "internal.hpp"

using namespace hmpc_gb300;
using namespace hmpc_gb300::detail;

namespace
{
    using clock_type = std::chrono::steady_clock;

    enum state : int
    {
        state_queued = 0,
        state_running = 1,
        state_done = 2,
        state_failed = -2,
    };

    struct Request
    {
        hmpc_request r{};
        uint64_t ticket = 0;
        clock_type::time_point submitted, finished;
        std::atomic<int> st{state_queued};
    };

    struct ResidentKey
    {
        hmpc_modulus* q = nullptr;
        hmpc_modulus* p = nullptr;
        uint64_t n = 0;
        uint32_t* a = nullptr;
        uint32_t* b = nullptr;
    };

    // first-fit allocator over the reserved device pool
    class Pool
    {
    public:
        void reset(uint64_t bytes)
        {
            free_.clear();
            free_[0] = bytes;
            total_ = bytes;
        }
        bool allocate(uint64_t bytes, uint64_t& offset)
        {
            bytes = (bytes + 255) & ~uint64_t{255};
            for (auto it = free_.begin(); it != free_.end(); ++it)
            {
                if (it->second >= bytes)
                {
                    offset = it->first;
                    const uint64_t rest = it->second - bytes;
                    const uint64_t at = it->first + bytes;
                    free_.erase(it);
                    if (rest)
                    {
                        free_[at] = rest;
                    }
                    return true;
                }
            }
            return false;
        }
        void release(uint64_t offset, uint64_t bytes)
        {
            bytes = (bytes + 255) & ~uint64_t{255};
            auto it = free_.emplace(offset, bytes).first;
            auto next = std::next(it);
            if (next != free_.end() && it->first + it->second == next->first)
            {
                it->second += next->second;
                free_.erase(next);
            }
            if (it != free_.begin())
            {
                auto prev = std::prev(it);
                if (prev->first + prev->second == it->first)
                {
                    prev->second += it->second;
                    free_.erase(it);
                }
            }
        }
        uint64_t total() const
        {
            return total_;
        }

    private:
        std::map<uint64_t, uint64_t> free_;
        uint64_t total_ = 0;
    };

    // Device words held as disjoint ascending ranges.
    class Ranges
    {
    public:
        void clear()
        {
            ranges_.clear();
        }
        bool overlaps(const uint32_t* words, uint64_t count)
        {
            const auto it = ending_after(words);
            return it != ranges_.end() && it->first < words + count;
        }
        void add(const uint32_t* words, uint64_t count)
        {
            const uint32_t* end = words + count;
            const auto first = ending_after(words);
            auto last = first;
            for (; last != ranges_.end() && last->first < end; ++last)
            {
                words = std::min(words, last->first);
                end = std::max(end, last->second);
            }
            ranges_.insert(ranges_.erase(first, last), {words, end});
        }

    private:
        using Range = std::pair<const uint32_t*, const uint32_t*>;
        std::vector<Range>::iterator ending_after(const uint32_t* words)
        {
            return std::upper_bound(ranges_.begin(), ranges_.end(), words,
                                    [](const uint32_t* w, const Range& r) { return w < r.second; });
        }
        std::vector<Range> ranges_;
    };

    struct Dispatch
    {
        std::vector<Request*> reqs;
        int lane = -1;
        uint64_t offset = 0, bytes = 0;
        uint64_t own_words = 0, tc_words = 0;  // of the scratch: buffers of its own, tensor-core digits after them
        bool direct = false;                   // runs in the requests' own buffers
        // No request writes what another one reads or writes, so they may run side
        // by side in their own buffers.  Otherwise (a transform submitted twice into
        // one buffer, a result over another request's input) a pass of one would
        // meet half-made results of another: every input is gathered before the
        // first result is written, and the results follow in the requests' order.
        bool apart = true;
    };

    using GroupKey = std::tuple<int, const void*, uint64_t, uint32_t>;  // kind, modulus, n, key
}

struct hmpc_server
{
    hmpc_context* ctx = nullptr;
    uint32_t max_batch = 16;
    std::vector<std::unique_ptr<hmpc_context>> lanes;
    std::vector<cudaEvent_t> lane_done;
    std::vector<PolyRequest*> lane_desc;     // pinned descriptors per lane
    uint32_t* lane_error = nullptr;          // pinned, one per lane: its tensor-core error word after a dispatch
    std::vector<Dispatch> lane_work;
    std::vector<bool> lane_busy;
    uint32_t desc_capacity = 0;              // polynomials per lane descriptor buffer
    uint32_t batch_window_us = 0;            // hold a group that is not full for compatible arrivals
    PolyRequest* d_desc = nullptr;           // device descriptors, one region per lane
    uint8_t* pool_base = nullptr;
    Pool pool;
    std::vector<ResidentKey> keys;
    Ranges read_words, written_words;        // of the dispatch being put together (worker thread)

    std::mutex mu;
    std::condition_variable cv;
    std::deque<Request*> incoming;
    std::map<GroupKey, std::deque<Request*>> pending;
    std::unordered_map<uint64_t, std::unique_ptr<Request>> requests;
    uint64_t next_ticket = 1;
    std::thread worker;
    std::atomic<bool> stop{false};
    std::atomic<uint64_t> in_system{0};

    // statistics (worker thread; read under mu)
    uint64_t submitted = 0, completed = 0, rejected = 0, failed = 0, dispatches = 0, batched_requests = 0;
    std::vector<double> latencies_us;

    static uint64_t words_of(const hmpc_modulus* m, uint64_t n, uint64_t count)
    {
        return n * count * static_cast<uint64_t>(m->c.limbs);
    }

    // words of tensor-core digit buffers (two buffers of ceil((4L + 2) / 4)
    // words per element) that a forward transform of `polys` polynomials
    // takes when q's plan for that shape is the tensor-core engine, else 0
    static uint64_t tc_words(hmpc_modulus* q, uint64_t n, uint64_t polys)
    {
        if (n < 16 || !tc_applicable(q, __builtin_ctzll(n), producer_tensor, nullptr) ||
            !tc_plan_splits(q, n, polys))
        {
            return 0;
        }
        return 2 * ((4ull * static_cast<uint64_t>(q->c.limbs) + 5) / 4) * n * polys;
    }

    // What a dispatch of the given requests takes, and which way it then runs:
    // a plan that changes before it is issued does not change the dispatch.
    struct Need
    {
        uint64_t own = 0, tc = 0;  // words
        bool direct = false;
        uint64_t bytes() const
        {
            return (own + tc) * 4;
        }
    };

    Need need_of(const std::vector<Request*>& rs, bool apart) const
    {
        const hmpc_request& r0 = rs.front()->r;
        uint64_t polys = 0;
        for (auto* x : rs)
        {
            polys += x->r.count;
        }
        const bool single = rs.size() == 1;
        Need need;
        if (r0.kind == HMPC_REQUEST_NTT)
        {
            need.direct = !single && apart && r0.q->choice(r0.n, false, polys).radix_bits >= 2;
            need.own = single || need.direct ? 0 : words_of(r0.q, r0.n, polys);
            need.tc = need.direct ? 0 : tc_words(r0.q, r0.n, polys);
        }
        else if (r0.kind == HMPC_REQUEST_ENCRYPT)
        {
            const ResidentKey& k = keys[r0.key_id];
            const bool parts = parts_applicable(k.q, k.p);
            need.direct = parts && apart;
            need.own = 3 * words_of(k.q, k.n, polys);  // u, v/w, msg
            if (!single && !need.direct)
            {
                need.own += words_of(k.p, k.n, polys) + 2 * words_of(k.q, k.n, polys);  // plaintext, c0, c1
            }
            need.tc = parts ? 0 : tc_words(k.q, k.n, polys);
        }
        return need;
    }

    // whether the dispatch's requests stay apart with one more
    bool stays_apart(const Dispatch& d, const hmpc_request& r)
    {
        if (!d.apart || r.kind == HMPC_REQUEST_CT_MUL)
        {
            return d.apart;  // products are one launch each, in order
        }
        const uint64_t out_words = words_of(r.q, r.n, r.count);
        const bool encrypt = r.kind == HMPC_REQUEST_ENCRYPT;
        const uint64_t in_words = encrypt ? words_of(keys[r.key_id].p, r.n, r.count) : out_words;
        bool apart = !written_words.overlaps(r.in0, in_words);
        for (const uint32_t* out : {r.out0, encrypt ? r.out1 : nullptr})
        {
            apart = apart && !(out && (written_words.overlaps(out, out_words) || read_words.overlaps(out, out_words)));
        }
        // a transform may run in place, but not over a part of its own input
        return apart && (encrypt || r.out0 == r.in0 || !overlap(r.out0, out_words, r.in0, in_words));
    }

    void joined(const hmpc_request& r)
    {
        if (r.kind == HMPC_REQUEST_CT_MUL)
        {
            return;
        }
        const uint64_t out_words = words_of(r.q, r.n, r.count);
        const bool encrypt = r.kind == HMPC_REQUEST_ENCRYPT;
        read_words.add(r.in0, encrypt ? words_of(keys[r.key_id].p, r.n, r.count) : out_words);
        written_words.add(r.out0, out_words);
        if (encrypt)
        {
            written_words.add(r.out1, out_words);
        }
    }

    GroupKey group_of(const hmpc_request& r) const
    {
        return GroupKey{r.kind, r.q, r.n, r.kind == HMPC_REQUEST_ENCRYPT ? r.key_id : 0u};
    }

    // gather / scatter request blocks of a limb-planar batch buffer
    static cudaError_t copy_block(uint32_t* dst, uint64_t dst_pitch_words, const uint32_t* src,
                                  uint64_t src_pitch_words, uint64_t width_words, int limbs, cudaStream_t s)
    {
        return cudaMemcpy2DAsync(dst, dst_pitch_words * 4, src, src_pitch_words * 4, width_words * 4,
                                 static_cast<size_t>(limbs), cudaMemcpyDeviceToDevice, s);
    }

    // the descriptors of a dispatch's polynomials, on their way to the lane's
    // region of device memory
    int describe(Dispatch& d, uint64_t n, uint64_t polys, const PolyRequest** out)
    {
        PolyRequest* host_desc = lane_desc[static_cast<size_t>(d.lane)];
        PolyRequest* dev_desc = d_desc + static_cast<uint64_t>(d.lane) * desc_capacity;
        uint64_t poly = 0;
        for (auto* x : d.reqs)
        {
            for (uint64_t j = 0; j < x->r.count; ++j, ++poly)
            {
                PolyRequest& desc = host_desc[poly];
                std::copy(x->r.nonce, x->r.nonce + 3, desc.nonce);
                desc.index = static_cast<uint32_t>(j);
                desc.count = static_cast<uint32_t>(x->r.count);
                desc.in = x->r.in0 + j * n;
                desc.out[0] = x->r.out0 + j * n;
                desc.out[1] = x->r.out1 ? x->r.out1 + j * n : nullptr;
                desc.stride = n * x->r.count;
            }
        }
        HMPC_CUDA(cudaMemcpyAsync(dev_desc, host_desc, polys * sizeof(PolyRequest), cudaMemcpyHostToDevice,
                                  lanes[static_cast<size_t>(d.lane)]->stream),
                  "uploading request descriptors");
        *out = dev_desc;
        return HMPC_OK;
    }

    int issue(Dispatch& d)
    {
        hmpc_context* lane = lanes[static_cast<size_t>(d.lane)].get();
        cudaStream_t s = lane->stream;
        const hmpc_request& r0 = d.reqs.front()->r;
        const bool single = d.reqs.size() == 1;
        uint64_t polys = 0;
        for (auto* x : d.reqs)
        {
            polys += x->r.count;
        }
        uint32_t* scratch = reinterpret_cast<uint32_t*>(pool_base + d.offset);
        lane->tc_spin_limit = ctx->tc_spin_limit;
        lane->tc_test_stall = ctx->tc_test_stall;
        // the lane's tensor-core digit buffers come from the dispatch's share
        // of the pool, after its own buffers
        struct Lend
        {
            hmpc_context* ctx;
            ~Lend()
            {
                ctx->tc_lent = nullptr;
                ctx->tc_lent_words = 0;
            }
        } lend{lane};
        if (d.tc_words)
        {
            lane->tc_lent = scratch + d.own_words;
            lane->tc_lent_words = d.tc_words;
        }
        if (r0.kind == HMPC_REQUEST_NTT)
        {
            hmpc_modulus* q = r0.q;
            const int L = q->c.limbs;
            if (single)
            {
                return run_transform(lane, q, r0.n, r0.count, false, producer_tensor, 0, 0, r0.in0, r0.out0);
            }
            // between the requests' own buffers, unless these are not apart or
            // the plan is an engine that works on one buffer
            if (d.direct)
            {
                const PolyRequest* dev_desc = nullptr;
                if (int rc = describe(d, r0.n, polys, &dev_desc))
                {
                    return rc;
                }
                return run_requests(lane, q, r0.n, polys, dev_desc);
            }
            const uint64_t total = r0.n * polys;
            uint64_t at = 0;
            for (auto* x : d.reqs)
            {
                const uint64_t w = x->r.n * x->r.count;
                HMPC_CUDA(copy_block(scratch + at, total, x->r.in0, w, w, L, s), "gathering transform inputs");
                at += w;
            }
            if (int rc = run_transform(lane, q, r0.n, polys, false, producer_tensor, 0, 0, scratch, scratch))
            {
                return rc;
            }
            at = 0;
            for (auto* x : d.reqs)
            {
                const uint64_t w = x->r.n * x->r.count;
                HMPC_CUDA(copy_block(x->r.out0, w, scratch + at, total, w, L, s), "scattering transform outputs");
                at += w;
            }
            return HMPC_OK;
        }
        if (r0.kind == HMPC_REQUEST_CT_MUL)
        {
            for (auto* x : d.reqs)
            {
                const hmpc_request& r = x->r;
                cudaError_t e = r.q->kt->ct_mul(r.out0, r.out1, r.out2, r.in0, r.in1, r.in2, r.in3, r.n * r.count,
                                                r.q->h, s);
                if (e != cudaSuccess)
                {
                    return cuda_fail(e, "launching ciphertext product");
                }
                ++lane->launches;
            }
            return HMPC_OK;
        }
        // encryption: the batch of requests shares the key; polynomial i of
        // the batch draws with its request's nonce and local index
        const ResidentKey& k = keys[r0.key_id];
        const uint64_t n = k.n;
        const int lq = k.q->c.limbs;
        const int lp = k.p->c.limbs;
        const uint64_t total = n * polys;
        const uint64_t qw = total * static_cast<uint64_t>(lq);
        uint32_t* pt = scratch + 3 * qw;
        uint32_t* c0 = pt + total * static_cast<uint64_t>(lp);
        uint32_t* c1 = c0 + qw;
        const PolyRequest* dev_desc = nullptr;
        if (int rc = describe(d, n, polys, &dev_desc))
        {
            return rc;
        }
        if (d.direct)
        {
            return encrypt_cuda_cores(lane, k.q, k.p, n, polys, k.a, k.b, nullptr, nullptr, nullptr, scratch, dev_desc,
                                      false);
        }
        const uint32_t* plaintext = r0.in0;
        if (!single)
        {
            plaintext = pt;
            uint64_t at = 0;
            for (auto* x : d.reqs)
            {
                const uint64_t w = n * x->r.count;
                HMPC_CUDA(copy_block(pt + at, total, x->r.in0, w, w, lp, s), "gathering plaintexts");
                at += w;
            }
        }
        uint32_t* out0 = single ? r0.out0 : c0;
        uint32_t* out1 = single ? r0.out1 : c1;
        if (int rc = encrypt_cuda_cores(lane, k.q, k.p, n, polys, k.a, k.b, plaintext, out0, out1, scratch, dev_desc,
                                        false))
        {
            return rc;
        }
        if (!single)
        {
            uint64_t at = 0;
            for (auto* x : d.reqs)
            {
                const uint64_t w = n * x->r.count;
                HMPC_CUDA(copy_block(x->r.out0, w, c0 + at, total, w, lq, s), "scattering c0");
                HMPC_CUDA(copy_block(x->r.out1, w, c1 + at, total, w, lq, s), "scattering c1");
                at += w;
            }
        }
        return HMPC_OK;
    }

    // the lane's error word, on its way to the host behind the dispatch's work
    cudaError_t report(int lane_index)
    {
        hmpc_context* lane = lanes[static_cast<size_t>(lane_index)].get();
        return lane->tc_error ? cudaMemcpyAsync(lane_error + lane_index, lane->tc_error, sizeof(uint32_t),
                                                cudaMemcpyDeviceToHost, lane->stream)
                              : cudaSuccess;
    }

    void finish(int lane_index, bool ok)
    {
        Dispatch& d = lane_work[static_cast<size_t>(lane_index)];
        if (lane_error[lane_index])
        {
            // a bounded wait ran out: the requests failed, the next dispatch starts clean
            ok = false;
            lane_error[lane_index] = 0;
            hmpc_context* lane = lanes[static_cast<size_t>(lane_index)].get();
            cudaMemsetAsync(lane->tc_error, 0, sizeof(uint32_t), lane->stream);
        }
        const auto now = clock_type::now();
        {
            std::lock_guard<std::mutex> lock(mu);
            for (auto* x : d.reqs)
            {
                x->finished = now;
                x->st.store(ok ? state_done : state_failed);
                if (ok)
                {
                    ++completed;
                    latencies_us.push_back(std::chrono::duration<double, std::micro>(now - x->submitted).count());
                }
                else
                {
                    ++failed;
                }
            }
            // under the lock: between a drain's look at the count and its wait, a
            // change and its notification would be missed, and the drain sleep
            // until its timeout
            in_system.fetch_sub(d.reqs.size());
        }
        if (d.bytes)
        {
            pool.release(d.offset, d.bytes);
        }
        d = Dispatch{};
        lane_busy[static_cast<size_t>(lane_index)] = false;
        cv.notify_all();
    }

    void run()
    {
        cudaSetDevice(ctx->device);
        while (!stop.load())
        {
            bool progress = false;
            {
                std::unique_lock<std::mutex> lock(mu);
                while (!incoming.empty())
                {
                    Request* x = incoming.front();
                    incoming.pop_front();
                    pending[group_of(x->r)].push_back(x);
                    progress = true;
                }
            }
            // completions
            for (size_t i = 0; i < lanes.size(); ++i)
            {
                if (lane_busy[i])
                {
                    const cudaError_t e = cudaEventQuery(lane_done[i]);
                    if (e != cudaErrorNotReady)
                    {
                        finish(static_cast<int>(i), e == cudaSuccess);
                        progress = true;
                    }
                }
            }
            // dispatch: oldest group first, one batch per free lane
            for (;;)
            {
                int lane = -1;
                for (size_t i = 0; i < lanes.size(); ++i)
                {
                    if (!lane_busy[i])
                    {
                        lane = static_cast<int>(i);
                        break;
                    }
                }
                if (lane < 0)
                {
                    break;
                }
                std::deque<Request*>* best = nullptr;
                const auto now = std::chrono::steady_clock::now();
                for (auto& kv : pending)
                {
                    if (kv.second.empty() || (best && kv.second.front()->submitted >= best->front()->submitted))
                    {
                        continue;
                    }
                    // a group that could still grow waits for the window to pass
                    // since its oldest request arrived
                    if (batch_window_us && kv.second.size() < max_batch &&
                        now - kv.second.front()->submitted < std::chrono::microseconds(batch_window_us))
                    {
                        continue;
                    }
                    best = &kv.second;
                }
                if (!best)
                {
                    break;
                }
                Dispatch d;
                d.lane = lane;
                read_words.clear();
                written_words.clear();
                uint64_t polys = 0;
                while (!best->empty() && d.reqs.size() < max_batch &&
                       polys + best->front()->r.count <= desc_capacity)
                {
                    d.reqs.push_back(best->front());
                    const bool apart = stays_apart(d, best->front()->r);
                    const Need need = need_of(d.reqs, apart);
                    if (need.bytes() > pool.total())
                    {
                        d.reqs.pop_back();
                        break;
                    }
                    // grow the dispatch's block: give the old one back first
                    if (d.bytes)
                    {
                        pool.release(d.offset, d.bytes);
                    }
                    uint64_t offset = 0;
                    if (need.bytes() && !pool.allocate(need.bytes(), offset))
                    {
                        if (d.bytes)
                        {
                            pool.allocate(d.bytes, d.offset);  // the block just released fits again
                        }
                        d.reqs.pop_back();
                        break;
                    }
                    d.offset = offset;
                    d.bytes = need.bytes();
                    d.own_words = need.own;
                    d.tc_words = need.tc;
                    d.direct = need.direct;
                    d.apart = apart;
                    joined(best->front()->r);
                    polys += best->front()->r.count;
                    best->pop_front();
                }
                if (d.reqs.empty())
                {
                    break;  // the oldest group waits for memory
                }
                for (auto* x : d.reqs)
                {
                    x->st.store(state_running);
                }
                lane_work[static_cast<size_t>(lane)] = d;
                lane_busy[static_cast<size_t>(lane)] = true;
                ++dispatches;
                batched_requests += d.reqs.size();
                const int rc = issue(lane_work[static_cast<size_t>(lane)]);
                cudaError_t e = report(lane);
                if (e == cudaSuccess)
                {
                    e = cudaEventRecord(lane_done[static_cast<size_t>(lane)],
                                        lanes[static_cast<size_t>(lane)]->stream);
                }
                if (rc != HMPC_OK || e != cudaSuccess)
                {
                    cudaStreamSynchronize(lanes[static_cast<size_t>(lane)]->stream);
                    finish(lane, false);
                }
                progress = true;
            }
            if (!progress)
            {
                std::unique_lock<std::mutex> lock(mu);
                cv.wait_for(lock, std::chrono::microseconds(20), [&] { return !incoming.empty() || stop.load(); });
            }
        }
    }
};

extern "C" {

int hmpc_server_create(hmpc_context* ctx, const hmpc_server_config* config, hmpc_server** out)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    if (!config || !out || config->lanes == 0 || config->max_batch == 0)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "bad server configuration");
    }
    auto srv = std::make_unique<hmpc_server>();
    srv->ctx = ctx;
    srv->max_batch = config->max_batch;
    srv->desc_capacity = config->max_batch_polynomials ? config->max_batch_polynomials : 4096;
    srv->batch_window_us = config->batch_window_us;
    for (uint32_t i = 0; i < config->lanes; ++i)
    {
        auto lane = std::make_unique<hmpc_context>();
        lane->device = ctx->device;
        std::memcpy(lane->key, ctx->key, sizeof lane->key);
        HMPC_CUDA(cudaStreamCreateWithFlags(&lane->stream, cudaStreamNonBlocking), "creating a lane stream");
        cudaEvent_t ev;
        HMPC_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), "creating a lane event");
        PolyRequest* desc = nullptr;
        HMPC_CUDA(cudaMallocHost(&desc, srv->desc_capacity * sizeof(PolyRequest)), "allocating descriptors");
        srv->lanes.push_back(std::move(lane));
        srv->lane_done.push_back(ev);
        srv->lane_desc.push_back(desc);
    }
    HMPC_CUDA(cudaMallocHost(&srv->lane_error, config->lanes * sizeof(uint32_t)), "allocating the lanes' error words");
    std::fill(srv->lane_error, srv->lane_error + config->lanes, 0u);
    srv->lane_work.resize(config->lanes);
    srv->lane_busy.assign(config->lanes, false);
    HMPC_CUDA(cudaMalloc(&srv->d_desc, srv->desc_capacity * static_cast<uint64_t>(config->lanes) * sizeof(PolyRequest)),
              "allocating descriptors");
    if (config->memory_budget_bytes)
    {
        if (cudaMalloc(&srv->pool_base, config->memory_budget_bytes) != cudaSuccess)
        {
            return fail(HMPC_ERROR_OUT_OF_MEMORY, "reserving the server's memory pool");
        }
    }
    srv->pool.reset(config->memory_budget_bytes);
    hmpc_server* raw = srv.get();
    srv->worker = std::thread([raw] { raw->run(); });
    *out = srv.release();
    return HMPC_OK;
}

int hmpc_server_add_key(hmpc_server* srv, hmpc_modulus* q, hmpc_modulus* p, uint64_t n, const uint32_t* a,
                        const uint32_t* b, uint32_t* key_id)
{
    if (!srv || !q || !p || !a || !b || !key_id)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    if (int rc = enter(srv->ctx))
    {
        return rc;
    }
    if (int rc = check_degree(n))
    {
        return rc;
    }
    if (int rc = q->prepare(n, nullptr))
    {
        return rc;
    }
    ResidentKey k;
    k.q = q;
    k.p = p;
    k.n = n;
    const uint64_t bytes = n * static_cast<uint64_t>(q->c.limbs) * sizeof(uint32_t);
    HMPC_CUDA(cudaMalloc(&k.a, bytes), "allocating a resident key");
    HMPC_CUDA(cudaMalloc(&k.b, bytes), "allocating a resident key");
    HMPC_CUDA(cudaMemcpy(k.a, a, bytes, cudaMemcpyDeviceToDevice), "copying a resident key");
    HMPC_CUDA(cudaMemcpy(k.b, b, bytes, cudaMemcpyDeviceToDevice), "copying a resident key");
    std::lock_guard<std::mutex> lock(srv->mu);
    *key_id = static_cast<uint32_t>(srv->keys.size());
    srv->keys.push_back(k);
    return HMPC_OK;
}

int hmpc_server_submit(hmpc_server* srv, const hmpc_request* request, uint64_t* ticket)
{
    if (!srv || !request || !ticket)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    const hmpc_request& r = *request;
    if (r.count == 0 || r.count > srv->desc_capacity)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "request polynomial count out of range");
    }
    switch (r.kind)
    {
    case HMPC_REQUEST_NTT:
        if (!r.q || !r.in0 || !r.out0)
        {
            return fail(HMPC_ERROR_INVALID_ARGUMENT, "transform request needs q, in0, out0");
        }
        if (int rc = check_degree(r.n))
        {
            return rc;
        }
        if (int rc = r.q->prepare(r.n, nullptr))
        {
            return rc;
        }
        break;
    case HMPC_REQUEST_ENCRYPT:
    {
        std::lock_guard<std::mutex> lock(srv->mu);
        if (r.key_id >= srv->keys.size() || !r.in0 || !r.out0 || !r.out1 || srv->keys[r.key_id].n != r.n)
        {
            return fail(HMPC_ERROR_INVALID_ARGUMENT, "encryption request needs a resident key of its degree");
        }
        break;
    }
    case HMPC_REQUEST_CT_MUL:
        if (!r.q || !r.in0 || !r.in1 || !r.in2 || !r.in3 || !r.out0 || !r.out1 || !r.out2)
        {
            return fail(HMPC_ERROR_INVALID_ARGUMENT, "product request needs two ciphertexts and three outputs");
        }
        break;
    default:
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "unknown request kind");
    }
    auto x = std::make_unique<Request>();
    x->r = r;
    if (r.kind == HMPC_REQUEST_ENCRYPT)
    {
        x->r.q = srv->keys[r.key_id].q;
    }
    x->submitted = clock_type::now();
    {
        std::lock_guard<std::mutex> lock(srv->mu);
        // a request that cannot run even alone is rejected
        std::vector<Request*> alone{x.get()};
        if (srv->need_of(alone, true).bytes() > srv->pool.total())
        {
            ++srv->rejected;
            return fail(HMPC_ERROR_REJECTED, "request needs more scratch than the server's memory budget");
        }
        x->ticket = srv->next_ticket++;
        *ticket = x->ticket;
        ++srv->submitted;
        srv->in_system.fetch_add(1);  // before the worker can see, and finish, the request
        srv->incoming.push_back(x.get());
        srv->requests.emplace(x->ticket, std::move(x));
    }
    srv->cv.notify_all();
    return HMPC_OK;
}

int hmpc_server_poll(hmpc_server* srv, uint64_t ticket, int* state, double* latency_us)
{
    if (!srv || !state)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    std::lock_guard<std::mutex> lock(srv->mu);
    auto it = srv->requests.find(ticket);
    if (it == srv->requests.end())
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "unknown ticket");
    }
    *state = it->second->st.load();
    if (latency_us)
    {
        *latency_us = *state == state_done
                          ? std::chrono::duration<double, std::micro>(it->second->finished - it->second->submitted).count()
                          : 0.0;
    }
    return HMPC_OK;
}

int hmpc_server_drain(hmpc_server* srv, uint32_t timeout_ms)
{
    if (!srv)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null server");
    }
    std::unique_lock<std::mutex> lock(srv->mu);
    const bool ok = srv->cv.wait_for(lock, std::chrono::milliseconds(timeout_ms),
                                     [&] { return srv->in_system.load() == 0; });
    return ok ? HMPC_OK : fail(HMPC_ERROR_TIMEOUT, "requests still in flight");
}

int hmpc_server_get_stats(hmpc_server* srv, hmpc_server_stats* out)
{
    if (!srv || !out)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    std::lock_guard<std::mutex> lock(srv->mu);
    *out = hmpc_server_stats{};
    out->submitted = srv->submitted;
    out->completed = srv->completed;
    out->rejected = srv->rejected;
    out->failed = srv->failed;
    out->dispatches = srv->dispatches;
    out->mean_batch = srv->dispatches ? static_cast<double>(srv->batched_requests) / srv->dispatches : 0.0;
    uint64_t launches = 0;
    for (auto& lane : srv->lanes)
    {
        launches += lane->launches;
    }
    out->launches = launches;
    std::vector<double> lat = srv->latencies_us;
    if (!lat.empty())
    {
        std::sort(lat.begin(), lat.end());
        auto at = [&](double f) { return lat[std::min(lat.size() - 1, static_cast<size_t>(f * (lat.size() - 1) + 0.5))]; };
        out->p50_us = at(0.50);
        out->p99_us = at(0.99);
        double sum = 0;
        for (double v : lat)
        {
            sum += v;
        }
        out->mean_us = sum / lat.size();
    }
    return HMPC_OK;
}

int hmpc_server_destroy(hmpc_server* srv)
{
    if (!srv)
    {
        return HMPC_OK;
    }
    srv->stop.store(true);
    srv->cv.notify_all();
    if (srv->worker.joinable())
    {
        srv->worker.join();
    }
    cudaSetDevice(srv->ctx->device);
    for (size_t i = 0; i < srv->lanes.size(); ++i)
    {
        cudaStreamSynchronize(srv->lanes[i]->stream);
        cudaStreamDestroy(srv->lanes[i]->stream);
        cudaEventDestroy(srv->lane_done[i]);
        cudaFreeHost(srv->lane_desc[i]);
        srv->lanes[i]->stream = nullptr;
    }
    for (auto& k : srv->keys)
    {
        cudaFree(k.a);
        cudaFree(k.b);
    }
    cudaFreeHost(srv->lane_error);
    cudaFree(srv->d_desc);
    cudaFree(srv->pool_base);
    delete srv;
    return HMPC_OK;
}

}  // extern "C"
