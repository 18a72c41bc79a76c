// tile_program.h -- host side of the tile driver (tile_device.cuh): the bodies'
// parameters in joint frames and the order in which a tile of instances takes
// them.
//
// A tile is up to 32 instances, one per lane, swept by W warps in lockstep
// steps: at a step each warp takes one body of each instance, and all of them
// are of one class (mobilizer), so lanes never diverge over mobilizers. Which
// bodies depends on the tile: a list schedule over its instances' trees, base
// to tip (run backwards it is the tip-to-base order). A body follows its
// parent, and follows the sibling before it, by at least one step: children
// add to their parent's record, and two of them at one step would race. The
// order among siblings is fixed by the topology alone, so an instance's sums,
// and with them its results, do not depend on which tile it is in.
#pragma once
#include <algorithm>
#include <array>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <exception>
#include <functional>
#include <map>
#include <mutex>
#include <queue>
#include <thread>
#include <vector>

#include "tile_core.cuh"
#include "topology_internal.h"

namespace sbg {

// f(0) ... f(n - 1), in any order, on up to eight host threads, one for every
// 3,000 of the `rows` schedule rows that the calls make, so that a small batch
// starts none (30 us each). What a call throws is thrown here.
template <class F> inline void tileParallel(int n, int64_t rows, F f) {
    const int64_t most = std::min<int64_t>({8, (int64_t)std::thread::hardware_concurrency(), rows / 3000, n});
    std::atomic<int> next{0};
    std::mutex m;
    std::exception_ptr thrown;
    auto work = [&] {
        try {
            for (int k = next++; k < n; k = next++) f(k);
        } catch (...) {
            std::lock_guard<std::mutex> lock(m);
            if (!thrown) thrown = std::current_exception();
            next = n;
        }
    };
    std::vector<std::thread> pool;
    if (most > 1) {
        pool.reserve(most - 1);
        try {
            while ((int64_t)pool.size() < most - 1) pool.emplace_back(work);
        } catch (...) {  // no more threads to be had: those there are do the work
        }
    }
    work();
    for (std::thread& t : pool) t.join();
    if (thrown) std::rethrow_exception(thrown);
}

// A body's FP64 instructions per RHS by class: what a step costs its sub-partition.
inline int tileCost(int cls, int n) {
    static const int c[tile::CL_COUNT] = {300, 205, 500, 390, 600, 400};
    return c[cls] + (cls == tile::CL_GEN ? 150 * n : 0);
}
// In FP64 instructions: what a step waits for its barrier, and what a body waits
// for its loads; another warp of the sub-partition fills the latter.
constexpr int kTileStepCost = 60, kTileBodyWait = 150;

inline int tileClassOf(int info) {
    using namespace tile;
    const int type = info & 15;
    const bool quat = (info & F_QUAT) != 0;
    return type == SBG_PIN ? CL_PIN : type == SBG_SLIDER ? CL_SLIDER : type == SBG_UNIVERSAL ? CL_UNIV
           : type == SBG_BALL && quat ? CL_BALL : type == SBG_FREE && quat ? CL_FREE : CL_GEN;
}

// Orders the instances of a batch so that a tile's trees have their mobilizers
// in like numbers: at a step all lanes take one class, so a tile takes as many
// steps of a class as its richest tree. Halves the set at the median of the
// class whose work spreads most, down to tiles of 32 (and of 8 within them);
// the tiles with the most work come first. work: per instance and class. 8,192
// random trees: lanes busy 57 % in the order of size alone, 65 % in this one.
inline void tileOrder(std::vector<int>& pos, const std::vector<std::array<float, tile::CL_COUNT>>& work) {
    using namespace tile;
    struct Rec {
        static void split(int* a, int n, const std::vector<std::array<float, CL_COUNT>>& work) {
            const int unit = n > 32 ? 32 : 8;
            if (n <= 8) return;
            int best = 0;
            float spread = -1;
            for (int c = 0; c < CL_COUNT; ++c) {
                float lo = work[a[0]][c], hi = lo, sum = 0, sq = 0;
                for (int k = 0; k < n; ++k) {
                    const float v = work[a[k]][c];
                    lo = std::min(lo, v);
                    hi = std::max(hi, v);
                    sum += v;
                    sq += v * v;
                }
                const float s = hi > lo ? sq - sum * sum / n : -1;
                if (s > spread) { spread = s; best = c; }
            }
            if (spread < 0) return;  // all alike
            const int m = ((n + 2 * unit - 1) / (2 * unit)) * unit;
            if (m >= n) return;
            std::nth_element(a, a + m, a + n, [&](int x, int y) {
                return work[x][best] != work[y][best] ? work[x][best] > work[y][best] : x < y;
            });
            split(a, m, work);
            split(a + m, n - m, work);
        }
    };
    const int n = (int)pos.size();
    if (n == 0) return;
    Rec::split(pos.data(), n, work);
    std::vector<std::pair<float, int>> tiles;  // work of the richest instance, first position
    for (int p = 0; p + 32 <= n; p += 32) {
        float most = 0;
        for (int k = p; k < p + 32; ++k) {
            float t = 0;
            for (float v : work[pos[k]]) t += v;
            most = std::max(most, t);
        }
        tiles.push_back({-most, p});
    }
    std::sort(tiles.begin(), tiles.end());
    std::vector<int> out;
    for (const auto& t : tiles) out.insert(out.end(), pos.begin() + t.second, pos.begin() + t.second + 32);
    out.insert(out.end(), pos.begin() + n / 32 * 32, pos.end());
    pos.swap(out);
}

// The rows of one topology for the tile driver. The FP32 routines have two
// widths, and the chain driver's order in which children add to their parent
// (falling rows, tip to base); the FP64 ones a class per mobilizer, and
// siblings in the order of falling height.
struct TileRows {
    int nb = 0;
    bool pose = false, gen = false;
    const sbg_topology_s* t = nullptr;
    std::vector<int16_t> cls;
    std::vector<int> height, cost;
    std::vector<int32_t> info;          // info words with the tile driver's flags
    std::vector<int> waits;             // parent and sibling that come before, per row
    std::vector<int> next0, next;       // rows that wait for row r: next[next0[r]] ...

    TileRows() {}
    TileRows(const sbg_topology_s& topo, bool fp32) : nb(topo.nb), t(&topo) {
        using namespace tile;
        cls.resize(nb); height.assign(nb, 0); cost.resize(nb); info.resize(nb); waits.assign(nb, 0);
        for (int r = 0; r < nb; ++r) {
            const int n = (t->info[r] >> 4) & 15, p = t->parent[r];
            info[r] = t->info[r];
            if (fp32) {
                cls[r] = n == 6 ? CL_FREE : CL_BALL;
                gen |= n == 6;
                cost[r] = n == 6 ? 900 : 300;
                continue;
            }
            cls[r] = (int16_t)tileClassOf(t->info[r]);
            gen |= cls[r] == CL_GEN;
            cost[r] = tileCost(cls[r], n);
            pose |= t->kcnt[r] > 0;
            // C = R_MB of the parent times R_PF
            bool ci = (t->info[r] & F_RPF_I) && (p < 0 || (t->info[p] & F_RMB_I));
            if (!ci && p >= 0) {
                const double *PR = &t->par[(size_t)p * kParamStride + 22], *RPF = &t->par[(size_t)r * kParamStride + 10];
                ci = true;
                for (int i = 0; i < 3; ++i)
                    for (int j = 0; j < 3; ++j)
                        ci &= PR[3 * i] * RPF[j] + PR[3 * i + 1] * RPF[3 + j] + PR[3 * i + 2] * RPF[6 + j] == (i == j);
            }
            unsigned springs = 0, dampers = 0;
            for (int f = t->fbeg[r]; f < t->fbeg[r] + t->fcnt[r]; ++f)
                if (t->fcoef[f] != 0) ((t->fkw[f] >> 8) ? dampers : springs) |= 1u << (t->fkw[f] & 255);
            const bool all = (springs & dampers) == (1u << n) - 1;  // each mobility has both
            info[r] |= (ci ? F_CI : 0) | (t->fcnt[r] == 0 ? F_FREELY : 0) | (all ? F_FORCES : 0);
        }
        for (int r = nb - 1; r >= 0; --r) {
            height[r] += cost[r] + (fp32 ? 0 : kTileStepCost);
            if (t->parent[r] >= 0) height[t->parent[r]] = std::max(height[t->parent[r]], height[r]);
        }
        // a body waits for its parent and for the sibling before it
        std::vector<int> sib(nb, -1), kids;
        for (int r = 0; r < nb; ++r) {
            kids.assign(t->clist.begin() + t->cbeg[r], t->clist.begin() + t->cbeg[r] + t->ccnt[r]);
            if (!fp32) std::stable_sort(kids.begin(), kids.end(), [&](int x, int y) { return height[x] > height[y]; });
            for (size_t k = 1; k < kids.size(); ++k) sib[kids[k - 1]] = kids[k];
        }
        next0.reserve(nb + 1);
        next.reserve(2 * nb);
        for (int r = 0; r < nb; ++r) {
            next0.push_back((int)next.size());
            next.insert(next.end(), t->clist.begin() + t->cbeg[r], t->clist.begin() + t->cbeg[r] + t->ccnt[r]);
            if (sib[r] >= 0) next.push_back(sib[r]);
        }
        next0.push_back((int)next.size());
        for (int k : next) ++waits[k];
    }
};

// Schedule of one tile: classes of (step, warp), and the row each lane takes
// there (-1: none).
struct TileSchedule {
    int nsteps = 0, lanes = 0;
    std::vector<int32_t> cls;              // nsteps * W
    std::vector<int> row;                  // per slot and lane
    // FP64 instructions: length, step by step of the busiest sub-partition (a
    // block's warps take the SM's four in turn); load, of the busiest one in all
    int64_t length = 0, load = 0;
    static constexpr double kCritical = 1.0;

    TileSchedule() {}
    TileSchedule(const std::vector<const TileRows*>& rows, int W) : lanes((int)rows.size()) {
        using namespace tile;
        const int nl = lanes;
        std::vector<std::vector<int>> ready(nl), waits(nl), done(nl);
        int remaining = 0;
        for (int l = 0; l < nl; ++l) {
            waits[l] = rows[l]->waits;
            remaining += rows[l]->nb;
            for (int r = 0; r < rows[l]->nb; ++r)
                if (!waits[l][r]) ready[l].push_back(r);
        }
        std::vector<int> turn(W);  // warps, the one with the least work so far first
        std::vector<int64_t> sum(W, 0), sub(std::min(W, 4), 0), stepSub, stepBody;
        for (int w = 0; w < W; ++w) turn[w] = w;
        while (remaining > 0) {
            stepSub.assign(sub.size(), 0);
            stepBody.assign(sub.size(), 0);
            for (auto& d : done) d.clear();
            std::stable_sort(turn.begin(), turn.end(), [&](int a, int b) { return sum[a] < sum[b]; });
            cls.resize(cls.size() + W, -1);
            row.resize(row.size() + (size_t)W * nl, -1);
            for (int w : turn) {
                const size_t slot = (size_t)nsteps * W + w;
                // the class with the most work ready, weighted by how critical it is
                double score[CL_COUNT] = {};
                for (int l = 0; l < nl; ++l) {
                    if (ready[l].empty()) continue;
                    const TileRows& t = *rows[l];
                    int most[CL_COUNT] = {}, top = 0;
                    for (int r : ready[l]) {
                        most[t.cls[r]] = std::max(most[t.cls[r]], t.height[r]);
                        top = std::max(top, t.height[r]);
                    }
                    for (int c = 0; c < CL_COUNT; ++c)
                        if (most[c]) score[c] += 1.0 + kCritical * most[c] / top;
                }
                int best = -1;
                for (int c = 0; c < CL_COUNT; ++c)
                    if (score[c] > 0 && (best < 0 || score[c] > score[best])) best = c;
                if (best < 0) break;
                cls[slot] = best;
                int stepCost = 0;
                for (int l = 0; l < nl; ++l) {
                    const TileRows& t = *rows[l];
                    auto& rd = ready[l];
                    int at = -1;
                    for (int k = 0; k < (int)rd.size(); ++k)
                        if (t.cls[rd[k]] == best && (at < 0 || t.height[rd[k]] > t.height[rd[at]])) at = k;
                    if (at < 0) continue;
                    const int r = rd[at];
                    rd.erase(rd.begin() + at);
                    row[slot * nl + l] = r;
                    done[l].push_back(r);
                    --remaining;
                    stepCost = std::max(stepCost, t.cost[r]);
                }
                sum[w] += stepCost;
                sub[w % 4] += stepCost;
                stepSub[w % 4] += stepCost;
                stepBody[w % 4] = std::max<int64_t>(stepBody[w % 4], stepCost + kTileBodyWait);
            }
            for (int l = 0; l < nl; ++l) {
                const TileRows& t = *rows[l];
                for (int r : done[l])
                    for (int k = t.next0[r]; k < t.next0[r + 1]; ++k)
                        if (--waits[l][t.next[k]] == 0) ready[l].push_back(t.next[k]);
            }
            length += std::max(*std::max_element(stepSub.begin(), stepSub.end()),
                               *std::max_element(stepBody.begin(), stepBody.end())) + kTileStepCost;
            ++nsteps;
        }
        load = *std::max_element(sub.begin(), sub.end()) + (int64_t)nsteps * kTileStepCost / 4;
    }
};

// The tables of a batch's tiles on the host. Parameters are formed on the
// device from the body table (parRow: its row and kParIdentity per slot and
// lane, -1: none).
struct TileProgram {
    int W = 1, rs = 0, rsTotal = 0;
    int ls = 32;           // lanes per tile
    bool shared = false;   // every tile has one topology: tables without lanes
    bool pose = false;
    std::vector<TileDesc> desc;
    std::vector<int32_t> cls, slots, parRow;
    int64_t recElems = 0, maxTile = 0;  // record doubles of all tiles, of the largest

    // A tile: the order position of its first instance, its lanes' topologies.
    struct Lanes {
        int pos0;
        std::vector<int> topo;
    };
    // The tables of the tiles. rows: per topology, rowBase: its first row in the
    // body table. Tiles are scheduled and written side by side (8,192 trees of 30
    // bodies: 85 ms one after another, 17 ms on eight threads).
    void build(const std::vector<Lanes>& tiles, const std::vector<const TileRows*>& rows,
               const std::vector<int32_t>& rowBase) {
        using namespace tile;
        std::vector<int> first(tiles.size()), own;  // the tile whose tables a tile has; those with their own
        std::map<int, int> known;
        int64_t work = 0;
        for (int k = 0; k < (int)tiles.size(); ++k) {
            first[k] = shared ? known.emplace(tiles[k].topo[0], k).first->second : k;
            if (first[k] != k) continue;
            own.push_back(k);
            for (int l = 0; l < (shared ? 1 : (int)tiles[k].topo.size()); ++l) work += rows[tiles[k].topo[l]]->nb;
        }
        std::vector<TileSchedule> plans(own.size());
        tileParallel((int)own.size(), work, [&](int i) {
            const std::vector<int>& topo = tiles[own[i]].topo;
            std::vector<const TileRows*> lanes;
            for (size_t l = 0; l < (shared ? 1 : topo.size()); ++l) lanes.push_back(rows[topo[l]]);
            plans[i] = TileSchedule(lanes, W);
        });
        const int st = shared ? 1 : ls;
        int64_t nCls = 0, nSlots = 0;
        desc.resize(tiles.size());
        for (int k = 0, i = 0; k < (int)tiles.size(); ++k) {
            TileDesc& d = desc[k];
            if (first[k] == k) {
                d.nsteps = plans[i++].nsteps;
                d.cls0 = (int32_t)nCls;
                d.slot0 = nSlots * SI_COUNT;
                d.par0 = nSlots * PR_COUNT;
                nCls += (int64_t)d.nsteps * W;
                nSlots += (int64_t)d.nsteps * W * st;
            } else {
                d = desc[first[k]];
            }
            d.pos0 = tiles[k].pos0;
            d.lanes = (int)tiles[k].topo.size();
            d.rec0 = recElems;
            const int64_t n = (int64_t)d.nsteps * W * rsTotal * ls;
            recElems += n;
            maxTile = std::max(maxTile, n);
        }
        cls.resize(nCls);
        slots.resize(nSlots * SI_COUNT);
        parRow.resize(nSlots);
        tileParallel((int)own.size(), work, [&](int i) {
            const TileDesc& d = desc[own[i]];
            const TileSchedule& s = plans[i];
            const std::vector<int>& topo = tiles[own[i]].topo;
            const int nl = s.lanes;
            const int64_t nslots = (int64_t)s.nsteps * W;
            std::copy(s.cls.begin(), s.cls.end(), cls.begin() + d.cls0);
            int32_t* const table = slots.data() + d.slot0;
            int32_t* const bodies = parRow.data() + d.par0 / PR_COUNT;
            std::fill(table, table + nslots * SI_COUNT * st, -1);
            std::fill(bodies, bodies + nslots * st, -1);
            std::vector<int> slotOf;
            for (int l = 0; l < nl; ++l) {
                const TileRows& t = *rows[topo[l]];
                slotOf.assign(t.nb, -1);
                for (int64_t k = 0; k < nslots; ++k) {
                    const int r = s.row[k * nl + l];
                    if (r < 0) continue;
                    slotOf[r] = (int)k;  // a parent's slot comes before
                    int32_t* o = table + (k * st + l) * SI_COUNT;
                    o[SI_Q] = t.t->qoff[r]; o[SI_U] = t.t->uoff[r];
                    o[SI_PARENT] = t.t->parent[r] < 0 ? -1 : slotOf[t.t->parent[r]];
                    o[SI_INFO] = t.info[r]; o[SI_ROW] = r;
                    o[SI_KBEG] = t.t->kbeg[r]; o[SI_KCNT] = t.t->kcnt[r];
                    bodies[k * st + l] = (rowBase[topo[l]] + r) | ((t.info[r] & F_CI) ? kParIdentity : 0);
                }
            }
            // the lanes of a step agree on these flags
            for (int64_t k = 0; k < nslots; ++k) {
                int32_t* o = table + k * st * SI_COUNT + SI_INFO;
                int all = F_CI | F_FREELY | F_FORCES;
                for (int l = 0; l < nl; ++l)
                    if (s.row[k * nl + l] >= 0) all &= o[l * SI_COUNT];
                for (int l = 0; l < nl; ++l)
                    if (s.row[k * nl + l] >= 0) o[l * SI_COUNT] &= ~(F_CI | F_FREELY | F_FORCES) | all;
            }
        });
    }

    // Instances per tile and warps per tile for a batch on `sms` SMs, topoAt[p]
    // the topology at order position p: the shape with the least time by the
    // schedule's FP64 instructions. Fewer lanes per tile follow a lane's own
    // tree better and more warps shorten the steps; both take sub-partitions
    // from other tiles. The lengths and loads of a sample of the tiles stand
    // for all, dealt out in order to the SMs (or, of fewer than four warps, to
    // the SM's shares): a share is done no sooner than its longest tile, the
    // sum of its loads, or its tiles one after another on the warps that
    // registers leave room for (eight an SM). Measured, ms, 8/32 lanes x 4/8
    // warps: 8,192 random trees 35.3 36.0 12.6 13.7; 3,000 with contacts 26.9
    // 26.6 13.3 12.6; 1,500 trees of 4 to 256 bodies 24.1 17.9 24.6 19.2.
    static void shape(const std::vector<int>& topoAt, const std::vector<const TileRows*>& rows, int sms, int& TW, int& W) {
        const int n = (int)topoAt.size();
        double best = 0;
        TW = 32; W = 1;
        const bool same = std::all_of(topoAt.begin(), topoAt.end(), [&](int k) { return k == topoAt[0]; });
        struct Candidate {
            int tw, w, tiles, samples;
            double len[6], load[6];
        };
        std::vector<Candidate> cand;
        std::vector<std::pair<int, int>> jobs;  // candidate, sample
        int64_t work = 0;
        for (int tw : {32, 8, 1}) {
            if (same && tw < 32) break;  // alignment is perfect at any width
            const int tiles = (n + tw - 1) / tw;
            if (tw < 32 && tiles > 16 * sms) break;
            for (int w : {1, 2, 4, 8}) {
                cand.push_back({tw, w, tiles, std::min(tiles, same ? 1 : 6), {}, {}});
                for (int s = 0; s < cand.back().samples; ++s) {
                    jobs.push_back({(int)cand.size() - 1, s});
                    work += (int64_t)tw * rows[topoAt[0]]->nb;
                }
            }
        }
        tileParallel((int)jobs.size(), work, [&](int j) {
            Candidate& c = cand[jobs[j].first];
            const int s = jobs[j].second;
            const int at = c.samples == 1 ? 0 : (int)((int64_t)(c.tiles - 1) * s / (c.samples - 1)), p0 = at * c.tw;
            std::vector<const TileRows*> lanes;
            for (int p = p0; p < std::min(n, p0 + (same ? 1 : c.tw)); ++p) lanes.push_back(rows[topoAt[p]]);
            const TileSchedule sc(lanes, c.w);
            c.len[s] = (double)sc.length;
            c.load[s] = (double)sc.load;
        });
        for (const Candidate& c : cand) {
            const int tw = c.tw, w = c.w, tiles = c.tiles, samples = c.samples;
            const double *len = c.len, *load = c.load;
            const int shares = sms * std::max(1, 4 / w);
            const double resident = w == 8 ? 1 : 2;
            std::vector<double> sum(shares, 0), row(shares, 0);
            std::priority_queue<std::pair<double, int>, std::vector<std::pair<double, int>>, std::greater<>> q;
            for (int k = 0; k < shares; ++k) q.push({0, k});
            double t = 0;
            for (int k = 0; k < tiles; ++k) {
                const double x = samples == 1 ? 0 : double(k) * (samples - 1) / std::max(1, tiles - 1);
                const int i = std::min((int)x, std::max(0, samples - 2)), j = std::min(i + 1, samples - 1);
                const double ln = len[i] + (x - i) * (len[j] - len[i]), ld = load[i] + (x - i) * (load[j] - load[i]);
                const int sh = q.top().second;
                q.pop();
                sum[sh] += ld;
                row[sh] += ln / resident;
                const double d = std::max(sum[sh], row[sh]);
                t = std::max({t, d, ln});
                q.push({d, sh});
            }
            if (best == 0 || t < 0.97 * best) { best = t; TW = tw; W = w; }
        }
    }

    // Warps per tile of the FP32 forms, whose tiles are bound by latency: the
    // fewest steps, while the GPU holds the warps at once (8 an SM; at 128
    // registers, 16 an SM, the spills cost more than the warps gave). Realize of
    // random trees, us, 2 / 4 / 8 warps: 512 trees 355 / 259 / 258, 4,096 633 /
    // 553 / 569, 16,384 935 / 1007 / 1582.
    static int warps32(const std::vector<int>& topoAt, const std::vector<const TileRows*>& rows, int sms) {
        const int n = (int)topoAt.size(), tiles = (n + 31) / 32;
        int W = 1;
        double best = 0;
        for (int w : {1, 2, 4}) {
            double steps = 0;
            const int samples = std::min(tiles, 4);
            for (int s = 0; s < samples; ++s) {
                std::vector<const TileRows*> lanes;
                const int p0 = (int)((int64_t)tiles * s / samples) * 32;
                for (int p = p0; p < std::min(n, p0 + 32); ++p) lanes.push_back(rows[topoAt[p]]);
                steps += double(TileSchedule(lanes, w).nsteps) / samples;
            }
            const double t = steps * std::max(1.0, double(tiles) * w / (8 * sms));
            if (best == 0 || t < 0.95 * best) { best = t; W = w; }
        }
        return W;
    }
};

}  // namespace sbg
