/*
 * Orders in which the persistent launches of a batch take their tasks (host
 * only).  A CTA takes the next task of the list and waits in it for the blocks
 * that it reads, so every list must hold a block's operands before the block:
 * then the earliest unfinished task can always run, however few CTAs there are.
 */
#ifndef EXAGEOSTAT_B200_BATCH_ORDER_H
#define EXAGEOSTAT_B200_BATCH_ORDER_H

#include <algorithm>
#include <vector>

struct XgBatchColumn {
    double key;
    int f, J;
};

/* Block columns of the fields f0 .. f1 - 1 (nb(f) each).  The fields advance
 * together, each by the same share of its columns (J / nb): neighbouring
 * columns of one field then lie far apart in the list, so a task rarely waits
 * for the one before it, and the fields end together, so the last columns of
 * the largest one do not run alone. */
template <class Nb> std::vector<XgBatchColumn> xg_batch_columns(int f0, int f1, Nb nb)
{
    std::vector<XgBatchColumn> cols;
    for (int f = f0; f < f1; ++f)
        for (int J = 0; J < nb(f); ++J) cols.push_back(XgBatchColumn{(double)J / nb(f), f, J});
    std::sort(cols.begin(), cols.end(), [](const XgBatchColumn &a, const XgBatchColumn &b) {
        return a.key != b.key ? a.key < b.key : a.f != b.f ? a.f < b.f : a.J < b.J;
    });
    return cols;
}

/* emit(f, I, J): the factorisation's blocks (tile_dag.cu) */
template <class Nb, class Emit> void xg_batch_factor_order(const std::vector<XgBatchColumn> &cols, Nb nb, Emit emit)
{
    for (const XgBatchColumn &c : cols)
        for (int I = c.J; I < nb(c.f); ++I) emit(c.f, I, c.J);
}

/* emit(f, J): the backward solve's block columns (solve.cu), every field's descending */
template <class Emit> void xg_batch_backward_order(const std::vector<XgBatchColumn> &cols, Emit emit)
{
    for (size_t q = cols.size(); q-- > 0;) emit(cols[q].f, cols[q].J);
}

/* emit(f, I, J, product): the inverse factors' blocks (rows_dag.cu), then
 * their products, the longest sums first */
template <class Nb, class Emit> void xg_batch_inverse_order(std::vector<XgBatchColumn> cols, Nb nb, Emit emit)
{
    for (const XgBatchColumn &c : cols)
        for (int I = 0; I <= c.J; ++I) emit(c.f, I, c.J, 0);
    std::sort(cols.begin(), cols.end(), [&](const XgBatchColumn &a, const XgBatchColumn &b) {
        const int la = nb(a.f) - a.J, lb = nb(b.f) - b.J;
        return la != lb ? la > lb : a.f < b.f;
    });
    for (const XgBatchColumn &c : cols)
        for (int J = 0; J <= c.J; ++J) emit(c.f, c.J, J, 1);
}

#endif
