// The reference's bridge class (include/mpcd/api/simulation_handle.hpp:14-45):
// owns one Backend chosen by name.
#pragma once

#include <memory>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "backend.hpp"

namespace mpcd {

// Backend factory (reference: src/libmpcd/common/backend_factory.hpp:15-27).
// "cuda" selects the GB300 backend; any other name throws "Unsupported backend type".
std::unique_ptr<Backend> create_backend(SimulationParameters const& params, std::string const& backend_type);

namespace api {

// Result vectors of one simulation, given back by the arrays that held them: a read of
// the size of an earlier one finds its memory mapped already, without page faults and a zero
// fill (69 MB of fields: 3.3 -> 0.9 ms).  Holds at most four vectors of up to 80 MiB, 128 MiB
// in all: copies into longer-lived memory of 350 MB took 2 to 54 ms here, into fresh memory
// a steady 17.5.
// Once its simulation is gone, what comes back is freed.
class ResultPool {
public:
    std::vector<float> take(size_t n)
    {
        std::lock_guard<std::mutex> lock(mutex_);
        for (auto& v : free_)
            if (v.size() == n) {
                std::vector<float> out = std::move(v);
                std::swap(v, free_.back());
                free_.pop_back();
                return out;
            }
        return {};
    }

    void give(std::vector<float>&& v)
    {
        std::lock_guard<std::mutex> lock(mutex_);
        size_t bytes = v.size() * sizeof(float);
        for (auto const& f : free_) bytes += f.size() * sizeof(float);
        if (!closed_ && free_.size() < 4 && v.size() * sizeof(float) <= (size_t(80) << 20) && bytes <= (size_t(1) << 27)) free_.push_back(std::move(v));
        else std::vector<float>().swap(v);
    }

    void close()
    {
        std::lock_guard<std::mutex> lock(mutex_);
        closed_ = true;
        free_.clear();
    }

private:
    std::mutex mutex_;
    std::vector<std::vector<float>> free_;
    bool closed_ = false;
};

class SimulationHandle {
public:
    SimulationHandle(SimulationParameters const&, std::string backend_type);
    ~SimulationHandle();

    SimulationHandle(SimulationHandle&&) noexcept;
    SimulationHandle& operator=(SimulationHandle&&) noexcept;
    SimulationHandle(const SimulationHandle&) = delete;
    SimulationHandle& operator=(const SimulationHandle&) = delete;

    SimulationParameters const& getParameters() const;

    void step(int n_steps);
    void stepAndAccumulateSample(int n_steps);
    void getSampleMean(std::vector<float>& mean_density, std::vector<float>& mean_velocity);

    void getParticlePositions(std::vector<float>& positions) const;
    void getParticleVelocities(std::vector<float>& velocities) const;
    void setParticlePositions(std::vector<float> const& positions);
    void setParticleVelocities(std::vector<float> const& velocities);
    void setParticles(std::vector<float> const& positions, std::vector<float> const& velocities);

    size_t getNParticles() const;

    std::shared_ptr<ResultPool> const& results() const { return results_; }

private:
    std::shared_ptr<ResultPool> results_ = std::make_shared<ResultPool>();
    std::unique_ptr<Backend> backend_;
};

}  // namespace api
}  // namespace mpcd
