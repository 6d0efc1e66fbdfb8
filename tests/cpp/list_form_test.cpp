// list_form_test.cpp -- host checks of the rule that picks the list step's form
// (pe_b200/csrc/list_form.h): its lines, and that a scene whose list entries hover around one of them
// keeps its form.  Prints "ok" on success.
#include <stdio.h>

#include <initializer_list>

#include "list_form.h"

static int failures = 0;
#define CHECK(c)                                                 \
    do {                                                         \
        if (!(c)) {                                              \
            printf("FAIL line %d: %s\n", __LINE__, #c);          \
            ++failures;                                          \
        }                                                        \
    } while (0)

// changes of form over 100 read-backs of lo and hi entries in turn
static int changes(int64_t n, bool fp64, int64_t lo, int64_t hi) {
    bool dense = false;
    int form = 0, count = 0;
    for (int k = 0; k < 100; ++k) {
        dense = peb::list_dense(dense, n, (k & 1) ? hi : lo);
        const int f = peb::list_form_rule(true, fp64, n, dense);
        if (f != form) ++count;
        form = f;
    }
    return count;
}

int main() {
    for (int fp64 = 0; fp64 < 2; ++fp64)
        for (int64_t n : {int64_t(30000), int64_t(99999), int64_t(1) << 31}) {
            CHECK(changes(n, fp64, 2 * n - 1, 2 * n) <= 1);
            CHECK(changes(n, fp64, 2 * n - 2 * n / 10, 2 * n + n / 10) <= 1);
        }
    CHECK(peb::list_dense(false, 100, 200) && !peb::list_dense(false, 100, 199));
    CHECK(peb::list_dense(true, 100, 175) && !peb::list_dense(true, 100, 174));
    CHECK(peb::list_form_rule(true, true, 1, true) == 2);
    CHECK(peb::list_form_rule(true, false, 24999, true) == 0);
    CHECK(peb::list_form_rule(true, false, 25000, true) == 2);
    CHECK(peb::list_form_rule(true, true, 99999, false) == 0);
    CHECK(peb::list_form_rule(true, true, 100000, false) == 2);
    CHECK(peb::list_form_rule(true, false, 399999, false) == 0);
    CHECK(peb::list_form_rule(true, false, 400000, false) == 2);
    CHECK(peb::list_form_rule(false, true, 1 << 20, true) == 0);
    if (failures == 0) printf("ok\n");
    return failures != 0;
}
