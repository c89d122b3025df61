// plan.h -- topology-only setup of the batched polar Newton solver (host side).
//
// Counterpart of the reference's one-off setup: nr_klu.cpp:732-759 (build_topology,
// build_J_pattern), p3s/cuda/polar_topology.py:100-194 (Jacobian pattern + inverse map)
// and p3s/cuda/lean_lu_plan.py:205-321 (fill-reducing order, symbolic factorization,
// level schedule). Re-designed for the GB300 kernel:
//
//  * The Jacobian is factored in 2x2 BUS BLOCKS. Every non-slack bus owns the variable
//    pair (angle, magnitude) and the equation pair (P, Q); a PV bus's magnitude column
//    and Q row are carried as an identity dummy. A block pivot is a whole bus, so one
//    block multiply-subtract does 8 FMAs on 8 loaded values (the scalar form needs 16
//    loads for the same 8 FMAs), and the elimination tree is the bus graph's -- half the
//    height of the scalar one, i.e. half the barriers per factorization.
//  * The fill-reducing order is a minimum-degree order of the bus graph.
//  * Factor entries are computed in Crout form, one task per block; a pivot's diagonal block
//    and its column of L form one chain on one worker (the inverse diagonal stays in
//    registers and scales each L block as it is computed: no separate scaling pass, one
//    barrier per level). The inverse diagonal is stored apart, at block nblk + row, and no task
//    writes a diagonal block in its own level: a chain heavier than its level's share of a
//    worker is cut into segments, each later segment led by a copy of the diagonal task that
//    recomputes the inverse from it without storing anything. Tasks and chain segments are
//    grouped by elimination-tree height (level), bundled with others of like length into steps
//    of a warp, and the bundles dealt to the CTA's warps longest-first onto the least-loaded one
//    (Schedule below). Pairs of a long task whose operands are final earlier are summed in an
//    earlier level, also into a diagonal block: after a pass it may hold a part of its sum, so
//    that every factorization needs a Jacobian evaluated anew. The forward substitution rides
//    along in the same levels.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

namespace gbpf {

enum TaskKind { TK_DIAG = 0, TK_U = 1, TK_L = 2, TK_FWD = 3 };
constexpr int TASK_SCALE = 1 << 3;  // L block: multiply by the inverse diagonal block computed just before
constexpr int TASK_FILL = 1 << 4;   // block not in the Jacobian: accumulate from zero
// (bit 5: the diagonal block has two real pivots -- a PQ row; set when a schedule is uploaded)
constexpr int TASK_NOSTORE = 1 << 6;  // diagonal recomputed for a chain segment: keep the inverse in registers
constexpr int TASK_CONT = 1 << 7;     // forward row whose leading pairs are already summed in its y
constexpr int TASK_ROW_SHIFT = 8;     // diagonal tasks: block row in code >> 8 (inverse at block nblk + row)

// One unit of factorization work before it is dealt to a worker: its level, destination
// block (or row), code, pair range and weight (the dealing key).
struct PlanTask {
    int level, dst, code, p0, p1;
    long long w;
    int next = -1;     // the next task of its chain (dealt to the same worker, laid out right after)
    bool head = true;  // first task of a chain (or a task on its own)
};

// The worker-dependent part of a plan: the level tasks dealt to `nwarps` warps of `wpw` workers
// each. A warp's program is its steps of level 0, 1, ...; step s holds the tasks of its workers
// at [s * wpw, (s + 1) * wpw) (4 ints each, destination -1: none), and warp u's steps of level h
// are [ptr[u * (levels + 1) + h], ptr[u * (levels + 1) + h + 1]). One spare step and one spare
// pointer at the end are read ahead by the kernel.
struct Schedule {
    int nwarps = 0, wpw = 0;
    std::vector<int> taskA, ptrA;   // factor levels with the forward substitution
    std::vector<int> taskF, ptrF;   // the forward substitution alone (chord passes)
    std::vector<int> taskC, ptrC;   // backward substitution
    std::vector<int> level_work;    // per level: max worker load
    std::vector<int> tasks_at, rows_at;  // tasks of every factor level, rows of every backward level
};

struct Plan {
    int n = 0;    // buses
    int nnzY = 0;
    int nv = 0;   // variable (non-slack) buses = block rows
    std::vector<int> vbus;          // v -> bus (pv then pq)
    std::vector<int> vidx;          // bus -> v, -1 for slack
    std::vector<uint8_t> bus_pq;    // bus is PQ
    std::vector<int> perm, pinv;    // pivot order over v
    std::vector<int> row_of_bus;    // bus -> block row (pivot index) or -1
    std::vector<int> bus_of_row;    // block row -> bus
    std::vector<uint8_t> row_pq;    // block row is a PQ bus
    std::vector<int> eval_order;    // buses in reverse Cuthill-McKee order (the evaluation's sweep:
                                    // buses evaluated together share their neighbours' state)
    // symbolic (block level, pivot numbering)
    std::vector<int> Lp, Li;        // strict lower structure of each pivot column, ascending
    std::vector<int> parent, height, depth;
    std::vector<int> base;          // first block of each pivot (its diagonal), size nv+1
    int nblk = 0;                   // blocks of the pattern; factor arrays hold nblk + nv (the
                                    // inverse diagonal of row r at block nblk + r)
    std::vector<int> posmap;        // Ybus nnz -> block position, -1 if a slack is involved
    std::vector<int> ydiag;         // bus -> CSR index of its diagonal, -1 if none
    // schedule for W workers
    int W = 0, warp = 1;            // workers, workers per warp
    int nlev = 0, nblev = 0;
    std::vector<int> taskA;         // 4 ints per task: dst, kind|flags, p0, p1 (see Schedule)
    std::vector<int> ptrA;
    std::vector<int> taskF, ptrF;   // forward rows alone
    std::vector<int> taskC;         // backward: 4 ints: row, inverse-diagonal block, p0, p1
    std::vector<int> ptrC;
    std::vector<int> pairs;         // 2 ints per pair
    std::vector<int> pair_level;    // level that makes a factor / forward pair's operands final
    // undealt tasks (factor levels, backward), kept so other worker counts can be scheduled
    std::vector<PlanTask> tasksA, tasksC;
    // statistics
    long long n_factor_pairs = 0, n_fwd_pairs = 0, n_bwd_pairs = 0;
    double rcond0 = 0.0;            // pivot ratio of the flat-start factorization
    double jinv_est = 0.0;          // |J^-1| (infinity norm) estimate at the flat start
    double y_rowsum = 0.0;          // largest row sum of |Ybus|
    std::vector<int> level_work;    // per level: max worker load (critical path estimate)
};

// Build everything topology-only, with a schedule for `workers` workers in the plan itself (0: none).
// Returns an empty string on success, else the error.
std::string build_plan(Plan& p, int n, const int* Yp, const int* Yj, int nnz, const int* pv, int npv,
                       const int* pq, int npq, int workers, double chain_cap = 1.0);

// Deal the plan's tasks to `nwarps` warps of `wpw` workers (longest first onto the least-loaded
// warp); a level's diagonal-and-L chain heavier than chain_cap x the level's mean work per
// worker is cut into segments on different workers, each later one recomputing the diagonal
// inverse (0: chains are never cut). `quad`: the same tasks dealt once more for four lanes a
// task (wpw / 4 tasks a step), or null.
void make_schedule(const Plan& p, int nwarps, int wpw, Schedule& out, double chain_cap = 1.0, Schedule* quad = nullptr);

// Host replica of the device algorithm (double precision): Jacobian blocks at (Vm, Va)
// written to `blocks` (nblk*4, zero where not in the Jacobian) and residual R (nv*2).
// host_factor / host_solve take arrays of (nblk + nv) * 4 (the inverse diagonals after them).
void host_eval(const Plan& p, const int* Yp, const int* Yj, const double* Yx, const double* Vm, const double* Va,
               const double* S, const uint8_t* pin, double* blocks, double* R);
// Serial block LU with the plan (in place); returns min/max real pivot in pmin/pmax and
// false on a zero / non-finite pivot.
bool host_factor(const Plan& p, double* blocks, double* pmin, double* pmax);
// Solve with factored blocks: b (nv*2, block-row order) -> x in place.
void host_solve(const Plan& p, const double* blocks, double* b);

}  // namespace gbpf
