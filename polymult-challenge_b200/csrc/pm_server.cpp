// pm_server.cpp -- serving: a request loop with continuous batching, admission by an HBM
// budget, and operands kept resident on the device in NTT form.
//
// No reference counterpart: the reference serves one fherma_run call at a time
// (main.cpp:181-186 times each call alone).  Here a server holds one point and R fixed
// operands b_0 .. b_{R-1}, each already through decomposition, column pass and row pass (the
// forward transform a multiply otherwise recomputes per call: k_row_fwd's output,
// solve.cu:341-355).  A request multiplies a fresh operand a by one of them, so it costs one
// decomposition, one forward column pass, the fused row pass (forward a, pointwise with the
// resident b_k, inverse), the inverse column pass and the CRT -- five kernels, or three where the
// GEMM kernels run the column passes -- plus its own H2D and D2H copy.
//
// Admission: every in-flight request holds its input, residue and output buffers
// (8NL + 4KN bytes, K rounded up to an even number in the form of three kernels); the budget minus the resident transforms and the tables bounds the
// requests in flight (max_inflight).  Device memory is carved at start-up into `streams`
// slots of cap = min(max_batch, max_inflight / streams) requests each.
//
// Continuous batching: the caller's thread runs the loop.  Requests join a FIFO queue at
// their arrival time; whenever a slot is free and the in-flight count allows, the slot takes
// every queued request up to its capacity -- whatever their resident operand (the fused row
// kernel reads resident transform sel[z] for batch entry z) -- and launches the batch: H2D copies,
// the kernels (three, or five in the separate form), D2H copies, an event.  Batches of different slots
// overlap on the device and on the copy engines; a slot's requests complete when its event
// has fired, and the slot takes the next batch at once.  Latency = completion seen by the
// loop - arrival time.
#include "pm_server.h"

#include "pm_kernels.cuh"

#include <algorithm>
#include <chrono>
#include <deque>
#include <thread>

namespace pm {

// A piece's input at least: its copies must outlast what starting them behind an event costs.  Wall
// time of a run, us, with pieces of one request / of 4 MB / of 8 MB / of whole batches:
//   24 requests of 16384 x 1747 bits (3.6 MB each) 2842 / 2739 / 2455 / 2803; 17 of 32768 x 868 bits
//   (3.7 MB) 1960 / 1793 / 1850 / 2145; 10 of 8192 x 3000 bits (3.1 MB) 993 / 965 / 1026 / 1414;
//   4 of 65536 x 1747 bits (14.4 MB) 1673 / 1693 / 1705 / 2452.
constexpr size_t PIECE_BYTES = 8u << 20;

Server::Server(uint32_t N, uint32_t W, uint32_t L, const uint32_t* q, const uint32_t* resident, uint32_t nresident,
               uint64_t hbm_budget, uint32_t max_batch, uint32_t streams, int gemm_request, int device)
    : device_(device), nres_(nresident), max_batch_(std::max(1u, max_batch)) {
    if (!resident || nresident == 0) throw InvalidPoint("a server needs at least one resident operand");
    if (streams == 0) throw InvalidPoint("streams must be >= 1");
    EngineOptions opt;
    opt.host_pipeline = false;
    eng_.reset(new Engine(N, W, L, q, gemm_request, device, opt));
    auto fixed_bytes = [&] { return (uint64_t)nres_ * eng_->residue_words() * 4 + eng_->table_bytes(); };
    auto request_bytes = [&] { return (uint64_t)(2 * eng_->plan().coeff_words() + eng_->residue_words()) * 4; };
    // the fused form's constant images and its even number of primes take a little more than the separate
    // form, which serves a budget that ends between the two
    if (eng_->fused() && hbm_budget <= fixed_bytes() + request_bytes()) {
        opt.w1 = eng_->split_w1();
        eng_.reset();
        eng_.reset(new Engine(N, W, L, q, gemm_request, device, opt));
    }
    try {
        const Plan& P = eng_->plan();
        const size_t cw = P.coeff_words(), rw = eng_->residue_words();
        const uint64_t fixed = fixed_bytes(), per_req = request_bytes();
        if (hbm_budget <= fixed + per_req)
            throw InvalidPoint("HBM budget too small: resident operands and tables need " + std::to_string(fixed) +
                               " bytes and one request " + std::to_string(per_req));
        max_inflight_ = (uint32_t)std::min<uint64_t>((hbm_budget - fixed) / per_req, 1u << 30);
        const uint32_t ns = std::min(streams, max_inflight_);
        cap_ = std::max(1u, std::min(max_batch_, max_inflight_ / ns));
        auto dalloc = [&](size_t words) {
            void* p = nullptr;
            cuda_check(cudaMalloc(&p, std::max<size_t>(words, 1) * 4), "cudaMalloc server");
            dev_.push_back(p);
            return static_cast<uint32_t*>(p);
        };
        resident_ = dalloc((size_t)nres_ * rw);
        eng_->reserve((size_t)ns * cap_ * P.N);  // a blocked CRT's partials: one region per slot
        piece_ = (uint32_t)std::max<size_t>(1, (PIECE_BYTES + cw * 4 - 1) / (cw * 4));
        slots_.resize(ns);
        for (Slot& s : slots_) {
            cuda_check(cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking), "stream");
            cuda_check(cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming), "event");
            s.in = dalloc((size_t)cap_ * cw);
            s.res = dalloc((size_t)cap_ * rw);
            s.out = dalloc((size_t)cap_ * cw);
            s.sel_d = dalloc(cap_);
            s.dig_d = reinterpret_cast<uint64_t*>(dalloc(2 * (size_t)cap_));
            if (cap_ > piece_) {
                cuda_check(cudaStreamCreateWithFlags(&s.in_stream, cudaStreamNonBlocking), "stream");
                cuda_check(cudaStreamCreateWithFlags(&s.out_stream, cudaStreamNonBlocking), "stream");
            }
            s.ev_in.resize((cap_ + piece_ - 1) / piece_);
            s.ev_c.resize(s.ev_in.size());
            for (cudaEvent_t& e : s.ev_in) cuda_check(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "event");
            for (cudaEvent_t& e : s.ev_c) cuda_check(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "event");
            cuda_check(cudaHostAlloc(&s.sel_h, cap_ * 4, cudaHostAllocDefault), "cudaHostAlloc");
            cuda_check(cudaHostAlloc(&s.dig_h, cap_ * 8, cudaHostAllocDefault), "cudaHostAlloc");
        }
        // resident operands -> forward transforms, through slot 0's input buffer
        const Chunk all{0, P.ncols};
        Slot& s0 = slots_[0];
        for (uint32_t k = 0; k < nres_; ++k) {
            cuda_check(cudaMemcpyAsync(s0.in, resident + (size_t)k * cw, cw * 4, cudaMemcpyHostToDevice, s0.stream),
                       "resident upload");
            uint32_t* rk = resident_ + (size_t)k * rw;
            eng_->launch_fwd(s0.in, all, 1, rk, s0.stream, /*ra=*/true, false, eng_->fused());  // the fused pass's RA operand
            eng_->launch_rows(false, rk, nullptr, 1, s0.stream, nullptr, false, eng_->fused());
            cuda_check(cudaStreamSynchronize(s0.stream), "resident transform");
        }
        eng_->throw_if_status();
    } catch (...) {
        release();
        throw;
    }
}

Server::~Server() { release(); }

void Server::release() {
    cudaSetDevice(device_);
    cudaDeviceSynchronize();
    for (Slot& s : slots_) {
        for (cudaStream_t st : {s.stream, s.in_stream, s.out_stream})
            if (st) cudaStreamDestroy(st);
        if (s.done) cudaEventDestroy(s.done);
        for (cudaEvent_t e : s.ev_in)
            if (e) cudaEventDestroy(e);
        for (cudaEvent_t e : s.ev_c)
            if (e) cudaEventDestroy(e);
        if (s.sel_h) cudaFreeHost(s.sel_h);
        if (s.dig_h) cudaFreeHost(s.dig_h);
    }
    slots_.clear();
    for (void* p : dev_) cudaFree(p);
    dev_.clear();
    for (void* p : host_) cudaFreeHost(p);
    host_.clear();
    eng_.reset();
}

void* Server::host_alloc(size_t bytes) {
    void* p = nullptr;
    cuda_check(cudaSetDevice(device_), "cudaSetDevice");
    cuda_check(cudaHostAlloc(&p, std::max<size_t>(bytes, 1), cudaHostAllocPortable), "cudaHostAlloc");
    host_.push_back(p);
    return p;
}

void Server::host_free(void* p) {
    auto it = std::find(host_.begin(), host_.end(), p);
    if (it == host_.end()) throw InvalidPoint("pointer was not allocated by this server");
    cudaFreeHost(p);
    host_.erase(it);
}

// the products of batch entries i0 .. i0 + n - 1, on the slot's stream
void Server::compute(Slot& s, uint32_t i0, uint32_t n, bool digest) {
    const Plan& P = eng_->plan();
    const size_t cw = P.coeff_words();
    const Chunk all{0, P.ncols};
    // after the copies the launches follow one another (each may overlap the previous one's tail)
    const bool f = eng_->fused();
    uint32_t* res = s.res + i0 * eng_->residue_words();
    eng_->launch_fwd(s.in + i0 * cw, all, n, res, s.stream, false, false, f);
    eng_->launch_rows(true, res, resident_, n, s.stream, s.sel_d + i0, true, f);
    eng_->launch_inv(res, all, n, s.out + i0 * cw, s.stream, ((size_t)(&s - slots_.data()) * cap_ + i0) * P.N, true, f);
    if (digest) launch_digest(s.out + i0 * cw, cw, n, s.dig_d + i0, s.stream);
}

void Server::copy_out(Slot& s, uint32_t i0, uint32_t n, uint32_t* const* c, bool digest, cudaStream_t st) {
    const size_t cw = eng_->plan().coeff_words();
    if (digest)
        cuda_check(cudaMemcpyAsync(s.dig_h + i0, s.dig_d + i0, n * 8, cudaMemcpyDeviceToHost, st), "digest D2H");
    for (uint32_t i = i0; i < i0 + n; ++i)
        cuda_check(cudaMemcpyAsync(c[s.reqs[i]], s.out + i * cw, cw * 4, cudaMemcpyDeviceToHost, st), "result D2H");
}

void Server::launch(Slot& s, const uint32_t* sel, const uint32_t* const* a, uint32_t* const* c, bool digest) {
    const size_t cw = eng_->plan().coeff_words();
    const uint32_t nb = (uint32_t)s.reqs.size();
    for (uint32_t i = 0; i < nb; ++i) {
        const uint32_t r = s.reqs[i];
        if (sel[r] >= nres_) throw InvalidPoint("request " + std::to_string(r) + ": resident index out of range");
        s.sel_h[i] = sel[r];
    }
    // A large batch with at most half of the slots in flight runs as a pipeline of pieces: piece
    // k + 1 is copied in while piece k is computed and piece k - 1 copied out (in one stream, its results
    // waited for all of its inputs).  Behind more batches it runs whole: their copies overlap its own,
    // and copies behind events are slower to start (65536 x 1747 bits, a queue that never empties: 2970
    // requests a second always in pieces, 3300 whole).
    size_t busy = 0;
    for (const Slot& o : slots_) busy += o.busy;
    const uint32_t np = 2 * busy <= slots_.size() ? (nb + piece_ - 1) / piece_ : 1, n = (nb + np - 1) / np;
    cudaStream_t in = np > 1 ? s.in_stream : s.stream, out = np > 1 ? s.out_stream : s.stream;
    for (uint32_t k = 0, i0 = 0; i0 < nb; ++k, i0 += n) {
        const uint32_t m = std::min(n, nb - i0);
        for (uint32_t i = i0; i < i0 + m; ++i)
            cuda_check(cudaMemcpyAsync(s.in + i * cw, a[s.reqs[i]], cw * 4, cudaMemcpyHostToDevice, in), "request H2D");
        if (k == 0) cuda_check(cudaMemcpyAsync(s.sel_d, s.sel_h, nb * 4, cudaMemcpyHostToDevice, in), "selector H2D");
        if (np > 1) {
            cuda_check(cudaEventRecord(s.ev_in[k], in), "record");
            cuda_check(cudaStreamWaitEvent(s.stream, s.ev_in[k], 0), "wait");
        }
        compute(s, i0, m, digest);
        if (np > 1) cuda_check(cudaEventRecord(s.ev_c[k], s.stream), "record");
    }
    // (after every launch: a copy into pageable memory holds the host until it is done)
    for (uint32_t k = 0, i0 = 0; i0 < nb; ++k, i0 += n) {
        if (np > 1) cuda_check(cudaStreamWaitEvent(out, s.ev_c[k], 0), "wait");
        copy_out(s, i0, std::min(n, nb - i0), c, digest, out);
    }
    cuda_check(cudaEventRecord(s.done, out), "record");
    s.busy = true;
}

void Server::run(uint32_t n, const double* t_arrive, const uint32_t* sel, const uint32_t* const* a,
                 uint32_t* const* c, double* latency, pm_serve_stats* stats, uint64_t* digest) {
    cuda_check(cudaSetDevice(device_), "cudaSetDevice");
    for (uint32_t i = 0; i < n; ++i) {
        if (!a[i] || !c[i]) throw InvalidPoint("request " + std::to_string(i) + ": null operand");
        if (i && t_arrive[i] < t_arrive[i - 1]) throw InvalidPoint("arrival times must not decrease");
    }
    using clk = std::chrono::steady_clock;
    const auto t0 = clk::now();
    auto now = [&] { return std::chrono::duration<double>(clk::now() - t0).count(); };
    std::deque<uint32_t> queue;
    uint32_t next = 0, done = 0, inflight = 0, peak = 0;
    uint64_t batches = 0, batched = 0;
    double t_last = 0.0;
    try {
        while (done < n) {
            bool progressed = false;
            const double t = now();
            while (next < n && t_arrive[next] <= t) queue.push_back(next++);
            for (Slot& s : slots_) {
                if (!s.busy) continue;
                const cudaError_t q = cudaEventQuery(s.done);
                if (q == cudaErrorNotReady) continue;
                cuda_check(q, "batch");
                const double tc = now();
                for (uint32_t r : s.reqs) latency[r] = tc - t_arrive[r];
                if (digest)
                    for (size_t i = 0; i < s.reqs.size(); ++i) digest[s.reqs[i]] = s.dig_h[i];
                done += (uint32_t)s.reqs.size();
                inflight -= (uint32_t)s.reqs.size();
                t_last = tc;
                s.reqs.clear();
                s.busy = false;
                progressed = true;
            }
            for (Slot& s : slots_) {
                if (s.busy || queue.empty() || inflight >= max_inflight_) continue;
                const uint32_t nb = std::min<uint32_t>({cap_, (uint32_t)queue.size(), max_inflight_ - inflight});
                for (uint32_t i = 0; i < nb; ++i) {
                    s.reqs.push_back(queue.front());
                    queue.pop_front();
                }
                launch(s, sel, a, c, digest != nullptr);
                inflight += nb;
                peak = std::max(peak, inflight);
                ++batches;
                batched += nb;
                progressed = true;
            }
            if (!progressed) {
                // nothing to do before the next arrival or completion: yield briefly
                if (next < n && queue.empty() && inflight == 0 && t_arrive[next] - now() > 200e-6)
                    std::this_thread::sleep_for(std::chrono::microseconds(50));
#if defined(__x86_64__)
                else
                    __builtin_ia32_pause();
#endif
            }
        }
    } catch (...) {
        cudaDeviceSynchronize();
        for (Slot& s : slots_) {
            s.reqs.clear();
            s.busy = false;
        }
        throw;
    }
    eng_->throw_if_status();
    if (stats) {
        stats->requests = n;
        stats->batches = batches;
        stats->mean_batch = batches ? (double)batched / batches : 0.0;
        stats->peak_inflight = peak;
        stats->max_inflight = max_inflight_;
        stats->seconds = n ? t_last - t_arrive[0] : 0.0;
    }
}

}  // namespace pm
