// copy_table (hd_edit_batch.cu) between direct-mapped tables: pool, page lines,
// page table, page numbers and bucket sizes word for word, whatever the
// target held before.  Exits 0 when all agree.
#include "../hashdag_gb300/csrc/hd_edit_batch.cu"

#include <cstdio>

static std::vector<uint32_t> words(const void* d, size_t n)
{
    std::vector<uint32_t> h(n);
    cudaMemcpy(h.data(), d, n * 4, cudaMemcpyDeviceToHost);
    return h;
}

static bool same(hd_ctx* a, hd_ctx* b)
{
    const size_t pages = a->g.pool_pages, nv = a->g.total_vpages;
    return words(a->t.pool, pages * HD_PAGE_SIZE) == words(b->t.pool, pages * HD_PAGE_SIZE) &&
           words(a->t.meta, pages * kPageMeta) == words(b->t.meta, pages * kPageMeta) &&
           words(a->t.page_ids, nv) == words(b->t.page_ids, nv) &&
           words(a->t.page_table, nv) == words(b->t.page_table, nv) &&
           words(a->t.bucket_sizes, a->g.total_buckets) == words(b->t.bucket_sizes, a->g.total_buckets);
}

static bool edit(hd_ctx* c, uint32_t tool, float x, float radius)
{
    hd_edit e{};
    e.tool = tool;
    e.center[0] = x;
    e.center[1] = e.center[2] = 512;
    e.radius = radius;
    hd_edit_stats s;
    return hd_edit_apply(c, &e, &s) == HD_OK;
}

int main()
{
    hd_config cfg;
    hd_default_config(10, &cfg);
    hd_ctx *a, *k;
    bool ok = hd_create(&cfg, &a) == HD_OK && hd_create(&cfg, &k) == HD_OK && hd_generate_scene(a, 1) == HD_OK &&
              hd_set_stream(k, a->stream) == HD_OK && a->t.direct;
    auto copied = [&](const char* what) {
        copy_table(k, a);
        const bool s = same(a, k);
        std::printf("%s: %s\n", what, s ? "same" : "different");
        ok = ok && s;
    };
    if (ok) {
        copied("into an empty table");
        ok = ok && edit(k, HD_TOOL_SPHERE_REMOVE, 500, 120) && edit(k, HD_TOOL_SPHERE_ADD, 400, 60) && !same(a, k);
        copied("into one with pages of its own");
        ok = ok && edit(a, HD_TOOL_SPHERE_ADD, 520, 150) && edit(a, HD_TOOL_SPHERE_REMOVE, 520, 150) &&
             hd_gc_ex(a, nullptr, 0, HD_GC_RELEASE_PAGES) == HD_OK && edit(k, HD_TOOL_BOX_ADD, 300, 200);
        copied("after a page-releasing GC");
        ok = ok && edit(k, HD_TOOL_SPHERE_ADD, 600, 90) && edit(a, HD_TOOL_SPHERE_ADD, 600, 90) && a->root == k->root;
    }
    return ok ? 0 : 1;
}
