/* An NVTX tool that writes the names of pushed ranges to the file named by NVTX_NAMES. */
#include <nvtx3/nvToolsExt.h>
#include <stdio.h>
#include <stdlib.h>

static FILE *out;
static int depth;

static int push(const char *name) {
    fprintf(out, "%d %s\n", depth++, name);
    fflush(out);
    return depth - 1;
}
static int pop(void) { return --depth; }

int InitializeInjectionNvtx2(NvtxGetExportTableFunc_t get) {
    const NvtxExportTableCallbacks *callbacks = (const NvtxExportTableCallbacks *)get(NVTX_ETID_CALLBACKS);
    NvtxFunctionTable table;
    unsigned int size = 0;
    const char *path = getenv("NVTX_NAMES");
    if (!path || !(out = fopen(path, "a"))) return 0;
    if (!callbacks || !callbacks->GetModuleFunctionTable(NVTX_CB_MODULE_CORE, &table, &size)) return 0;
    *table[NVTX_CBID_CORE_RangePushA] = (NvtxFunctionPointer)push;
    *table[NVTX_CBID_CORE_RangePop] = (NvtxFunctionPointer)pop;
    return 1;
}
