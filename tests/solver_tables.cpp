// The solver's tables for the host (built by test_cpu_policy_tables.py).
#include "qz_solver.h"

extern "C" {
int table_window(int n) { return qz::nw_table(n); }
int table_shifts(int nh) { return qz::ns_table(nh); }
}
